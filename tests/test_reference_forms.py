"""The reference's step in its four kernel forms, on the same samples.

A frame whose size puts it on one form (stages in a loop) is rendered whole and
as interleaved row shards whose sizes put them on the others (unrolled, eight
lanes per ray, the smaller register budget): every output has to agree bit for
bit, over both metrics, the disks and objects."""
from __future__ import annotations

import math

import numpy as np
import pytest

from gargantua_b200 import shard, workloads
from gargantua_b200.curved import (AccretionDisk, Camera, CheckerSky, ProceduralSky, RenderOptions,
                                   Scene, ThinDisk)
from gargantua_b200.gr_core import Kerr, RK45Integrator, Schwarzschild

pytestmark = pytest.mark.gpu

LARGE, SMALL, UNROLLED, GROUP = range(4)
DISKS = {"none": None, "volumetric": AccretionDisk(), "thin": ThinDisk(6.0, 20.0, 3.0)}
NAMES = ("cls", "x", "v", "lam", "attempts", "accepted", "intensity", "color_temp", "rgb", "cross")
CASES = [
    # Kerr, disk, objects, width, height, its form, (shards, their form) ...
    (True, "none", False, 513, 512, SMALL, ((2, UNROLLED), (64, GROUP))),
    (False, "none", False, 513, 512, LARGE, ((2, UNROLLED), (64, GROUP))),
    (True, "thin", False, 513, 512, SMALL, ((2, UNROLLED), (32, GROUP))),
    (False, "thin", False, 513, 512, LARGE, ((3, UNROLLED), (32, GROUP))),
    (True, "volumetric", False, 513, 256, SMALL, ((2, UNROLLED), (32, GROUP))),
    (False, "volumetric", False, 513, 256, LARGE, ((2, UNROLLED), (32, GROUP))),
    (True, "volumetric", True, 513, 256, SMALL, ((2, UNROLLED), (32, GROUP))),
    (False, "none", True, 513, 512, LARGE, ((2, UNROLLED), (64, GROUP))),
    (True, "none", False, 1025, 1024, LARGE, ((2, SMALL), (8, UNROLLED))),
]


@pytest.mark.parametrize("kerr,disk,objects,w,h,form,shards", CASES)
def test_forms_give_the_same_bits(renderer, gglib, kerr, disk, objects, w, h, form, shards):
    integ = RK45Integrator(max_radius=200.0, rtol=1e-8 if disk == "thin" else 0.0, atol=1e-10)
    scene = Scene(Kerr(1.0, 0.9) if kerr else Schwarzschild(1.0),
                  Camera.inclined(30.0, math.radians(86.0), math.radians(60.0), w / h), w, h,
                  DISKS[disk],
                  RenderOptions(max_steps=3000, integrator=integ,
                                sky=CheckerSky(18, 36, 0) if disk == "thin" else ProceduralSky()),
                  workloads.lensed_spheres() if objects else None)
    assert gglib.gg_check_trace_form(*scene.c_args()) == form
    img, whole = renderer.render(scene, rays=True)
    for world, part_form in shards:
        for k in sorted({0, world // 2, world - 1}):  # rows at the middle are the shadow's
            part = shard.shard_scene(scene, k, world)
            assert gglib.gg_check_trace_form(*part.c_args()) == part_form
            im, got = renderer.render(part, rays=True)
            assert np.array_equal(im, img[k::world])
            for name in NAMES:
                a, b = getattr(got, name), getattr(whole, name)
                if name == "rgb":
                    b = b.reshape(h, w, 3)[k::world].reshape(a.shape)
                else:
                    b = b.reshape(b.shape[:-1] + (h, w))[..., k::world, :].reshape(a.shape)
                assert np.array_equal(a, b, equal_nan=a.dtype.kind == "f"), (world, k, name)
