"""The mixed form where the first step is far too large.

An attempt that leaps across the hole forms FP32 stages far outside any ray's
range, up to overflow, and is taken again with a smaller step.  How often, and
so every output, depends on which of its products overflow: the FP32 right-hand
side's operations and their scale are part of the results.  The outcomes of such
renders are held to recorded ones (attempts, classes and states to the bit)."""
from __future__ import annotations

import hashlib
import math

import numpy as np
import pytest

from gargantua_b200 import abi
from gargantua_b200.curved import Camera, CheckerSky, RenderOptions, Scene, ThinDisk
from gargantua_b200.gr_core import Kerr, RK45Integrator

pytestmark = pytest.mark.gpu

# spin, camera radius, inclination, side, initial step, max_step, rtol, tolerance, disk: sha1
CASES = [
    ((0.998, 13.8, 90.0, 200, 19.8, 1.0, 0.0, 7e-5, False), "6b4983e5b9c3fd173a88704023906d17cfe30009"),
    ((0.9, 8.3, 70.0, 160, 36.0, 0.9, 0.0, 1e-6, True), "369d84a1fd6db0b53f1c20f47d0fa50994345866"),
    ((0.3, 6.3, 169.0, 220, 31.5, 4.1, 0.0, 7e-6, True), "1bff2f94aa323f82ac7c3d318c76a6e06f35eb2e"),
    ((-0.7, 10.0, 75.0, 170, 47.6, 1.7, 3.6e-4, 1e-6, True), "33452a33dd9134e80489902d644db53ca6cf16ae"),
    ((0.9, 12.0, 75.0, 200, 60.0, 50.0, 1e-2, 1e-6, True), "2664cc04693f154b9d04b293fb1ca3f6102fc99c"),
    ((0.95, 15.0, 85.0, 180, 120.0, 1.0, 1e-8, 1e-6, True), "76cbb9abe83930329f4f621755a784d453e9085a"),
]


def outcomes(renderer, case):
    spin, r_cam, incl, side, first, h_max, rtol, tol, disk = case
    integ = RK45Integrator(max_radius=200.0, initial_step=first, max_step=h_max, rtol=rtol,
                           atol=1e-10, tolerance=tol, stepper=abi.GG_STEPPER_DP45)
    scene = Scene(Kerr(1.0, spin), Camera.inclined(r_cam, math.radians(incl), math.radians(60.0), 1.0),
                  side, side, ThinDisk(4.0, 30.0, 3.0) if disk else None,
                  RenderOptions(sky=CheckerSky(18, 36, 5), max_steps=2000, integrator=integ,
                                precision=abi.GG_PREC_MIXED))
    img, o = renderer.render(scene, rays=True)
    h = hashlib.sha1(img.tobytes())
    for a in (o.cls, o.attempts, o.accepted, o.x, o.v):
        h.update(np.ascontiguousarray(a).tobytes())
    return h.hexdigest()


@pytest.mark.parametrize("case,want", CASES)
def test_recorded_outcomes(renderer, case, want):
    assert outcomes(renderer, case) == want
