"""The steppers' rule for steady attempts against the full step-size law.

An attempt at h = max_step whose error is at most kSteadyErr of its scale in
every component skips the error norm, its root and the clamp
(gg_device.cuh).  Here the law it stands for (geodesic.rs:310-321, the RMS
norms over four and eight components and the plain norm) is evaluated on
errors inside the rule's bound, its edge included: the attempt has to be
accepted and the next step has to be max_step."""
from __future__ import annotations

import re
from pathlib import Path

import numpy as np
import pytest

CSRC = Path(__file__).resolve().parents[1] / "gargantua_b200" / "csrc"
BOUND = float(re.search(r"kSteadyErr = ([0-9.]+);", (CSRC / "gg_device.cuh").read_text()).group(1))


def full_law(err, tol, h, h_min, h_max):
    """(accepted, next h) of an attempt with error norm err."""
    if not (err < tol or h <= h_min):
        return False, None
    if not err > 0.0:
        return True, h
    with np.errstate(over="ignore", divide="ignore"):
        hn = h * 0.9 * (np.float64(tol) / err) ** 0.2
    return True, min(max(hn, h_min), h_max)


def errors(n, scale, rng):
    """Error vectors inside the bound: spread over magnitudes, zero, one component
    at the edge, all of them at the edge."""
    edge = BOUND * scale
    out = [rng.uniform(-1, 1, n) * edge * 10.0 ** rng.uniform(-250, 0) for _ in range(500)]
    out += [np.zeros(n), np.eye(n)[0] * edge, np.full(n, edge), -np.full(n, edge),
            np.full(n, 5e-324)]
    return out


@pytest.mark.parametrize("n", [4, 8])
@pytest.mark.parametrize("h_max", [1e-3, 0.37, 1.0, 60.0])
def test_steady_attempt_keeps_max_step_rms(n, h_max):
    rng = np.random.default_rng(n)
    for scale in (1e-10, 1e-8, 1e-2, 3.0):
        for d in errors(n, scale, rng):
            q = d / scale
            err = np.sqrt((q * q).sum() / n)
            assert full_law(err, 1.0, h_max, 1e-8, h_max) == (True, h_max)


@pytest.mark.parametrize("tol", [1e-12, 1e-6, 1e-2])
def test_steady_attempt_keeps_max_step_norm(tol):
    rng = np.random.default_rng(1)
    limit = BOUND * BOUND * 0.98 * tol * tol
    for d in errors(4, tol, rng):
        s = float((d * d).sum())
        if s < limit:
            assert full_law(np.sqrt(s), tol, 1.0, 1e-8, 1.0) == (True, 1.0)
    assert full_law(np.sqrt(limit), tol, 1.0, 1e-8, 1.0) == (True, 1.0)
