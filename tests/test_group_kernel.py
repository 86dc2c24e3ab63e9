"""The group kernel (several lanes per ray) against the lane-per-ray kernels.

Renders of the reference's step with few samples run on the group kernel, and
larger ones, by their size on a kernel with its stages unrolled or in a loop,
hand their last rays to it; renders with an attempt budget never do.  Both carry out the same operations in the same order per ray, so every
output has to agree bit for bit: one sample, sizes that leave a group or a
warp part empty, both sides of the size rule, and images large enough to
drain into the second pass, over the metrics, disks, scenes, error norms and
supersampling."""
from __future__ import annotations

import copy
import math

import numpy as np
import pytest

from gargantua_b200 import workloads
from gargantua_b200.curved import (AccretionDisk, Camera, CheckerSky, ProceduralSky, RenderOptions,
                                   Scene, ThinDisk)
from gargantua_b200.gr_core import Kerr, RK45Integrator, Schwarzschild

pytestmark = pytest.mark.gpu

DISKS = {"none": None, "volumetric": AccretionDisk(), "thin": ThinDisk(6.0, 20.0, 3.0)}
CASES = [
    # width, height, samples per axis, Kerr, disk, objects, rtol
    (1, 1, 1, True, "none", False, 0.0),
    (5, 3, 1, False, "thin", False, 1e-8),
    (33, 7, 1, True, "thin", False, 1e-8),
    (31, 17, 2, True, "volumetric", False, 0.0),
    (29, 23, 1, False, "volumetric", True, 0.0),
    (47, 31, 1, True, "none", True, 0.0),
    (128, 128, 1, False, "none", False, 0.0),   # the size rule's last group render
    (129, 128, 1, True, "none", False, 0.0),    # and the first that drains into it
    (256, 128, 1, False, "none", False, 0.0),
    (257, 128, 1, True, "none", False, 0.0),
    (512, 512, 1, False, "thin", False, 1e-8),  # the last unrolled render
    (513, 512, 1, True, "none", False, 1e-8),   # and the first rolled one
    (512, 256, 1, True, "volumetric", False, 0.0),
    (513, 256, 1, False, "volumetric", True, 0.0),
    (301, 200, 1, False, "volumetric", False, 0.0),
    (301, 200, 1, True, "thin", False, 1e-8),
    (201, 100, 2, True, "volumetric", True, 0.0),
    (1201, 900, 1, True, "none", False, 1e-6),  # 2^20 samples and more
]


@pytest.mark.parametrize("w,h,spa,kerr,disk,objects,rtol", CASES)
def test_group_route_keeps_every_bit(renderer, w, h, spa, kerr, disk, objects, rtol):
    integ = RK45Integrator(max_radius=200.0, rtol=rtol, atol=1e-10)
    opts = RenderOptions(samples_per_axis=spa, max_steps=3000, integrator=integ,
                         sky=CheckerSky(18, 36, 0) if disk == "thin" else ProceduralSky())
    scene = Scene(Kerr(1.0, 0.9) if kerr else Schwarzschild(1.0),
                  Camera.inclined(30.0, math.radians(88.0), math.radians(60.0), w / h), w, h,
                  DISKS[disk], opts, workloads.lensed_spheres() if objects else None)
    general = copy.copy(scene)
    general.options = copy.copy(opts)
    general.options.attempt_budget = 1 << 50
    img, a = renderer.render(scene, rays=True)
    s = renderer.stats()
    want, b = renderer.render(general, rays=True)
    t = renderer.stats()
    assert (img == want).all()
    for name in ("cls", "x", "v", "lam", "attempts", "accepted", "intensity", "color_temp", "rgb",
                 "cross"):
        x, y = getattr(a, name), getattr(b, name)
        assert np.array_equal(x, y, equal_nan=x.dtype.kind == "f"), name
    assert (s.rays, s.attempts, s.accepted) == (t.rays, t.attempts, t.accepted)
    assert list(s.class_count) == list(t.class_count)
