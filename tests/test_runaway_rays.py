"""Rays whose velocity runs away to infinity.

A ray followed through the horizon (a negative horizon buffer) gains speed until
its products overflow in FP64.  Where they do, and so how the ray's last attempts
go and what its state ends as, depends on the size of every product of the
right-hand side.  The outcomes of such renders are held to recorded ones, with
infinities and NaN as they come, to the bit."""
from __future__ import annotations

import hashlib
import math

import numpy as np
import pytest

from gargantua_b200 import abi
from gargantua_b200.curved import Camera, RenderOptions, Scene
from gargantua_b200.gr_core import Kerr, RK45Integrator, Schwarzschild

pytestmark = pytest.mark.gpu

# spin (None: Schwarzschild), camera radius, inclination, side, max_step, rtol, buffer, full DP
CASES = [
    ((0.998, 6.0, 36.0, 280, 16.0, 1e-8, -0.05, False), "737266a093911684492e5091a04611f3cb5e1457"),
    ((0.9, 4.7, 90.0, 200, 1.0, 0.0, -0.05, False), "818b0d247b2658e2c36e903528950394bbab8816"),
    ((0.9, 7.0, 137.0, 250, 1.0, 9e-6, -0.2, False), "4adf1935d51c54fe2a564b12660aaf37e7784e81"),
    ((-0.9, 6.0, 60.0, 250, 4.0, 6e-8, -0.05, False), "e1f71f1d20da39f58ea767d3dc8801a28e01c045"),
    ((0.3, 8.0, 90.0, 250, 1.0, 1e-8, -1.0, True), "4c1bd70e85af3a6431459d6c03da766185b98e44"),
    ((None, 6.0, 80.0, 200, 4.0, 1e-8, -0.05, False), "1c23ade471ebb5add112b2e72ab6cb2c9f70976e"),
]


def outcomes(renderer, case):
    spin, r_cam, incl, side, h_max, rtol, buffer, full = case
    stepper = abi.GG_STEPPER_DP45 if full else abi.GG_STEPPER_REFERENCE
    integ = RK45Integrator(max_radius=200.0, max_step=h_max, rtol=rtol, atol=1e-10, stepper=stepper,
                           horizon_buffer=buffer)
    scene = Scene(Schwarzschild(1.0) if spin is None else Kerr(1.0, spin),
                  Camera.inclined(r_cam, math.radians(incl), math.radians(60.0), 1.0), side, side,
                  None, RenderOptions(max_steps=1200, integrator=integ))
    img, o = renderer.render(scene, rays=True)
    h = hashlib.sha1(img.tobytes())
    for a in (o.cls, o.attempts, o.accepted, o.x, o.v):
        h.update(np.ascontiguousarray(a).tobytes())
    return h.hexdigest()


@pytest.mark.parametrize("case,want", CASES)
def test_recorded_outcomes(renderer, case, want):
    assert outcomes(renderer, case) == want
