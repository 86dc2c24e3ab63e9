"""The unrolled full Dormand-Prince kernels against the rolled ones.

Small FP64 renders, and the mixed form's band passes over few rays, run a
form of the kernel with its stages unrolled; larger ones the rolled form.  A
frame whose samples (or band rays) are too many for the unrolled form is
rendered whole and as interleaved row shards that are not: every output has to
agree bit for bit.  The shards' sizes straddle the rules' lines, and the
smallest leave warps part empty."""
from __future__ import annotations

import copy
import math

import numpy as np
import pytest

from gargantua_b200 import abi, shard
from gargantua_b200.curved import AccretionDisk, Camera, CheckerSky, RenderOptions, Scene, ThinDisk
from gargantua_b200.gr_core import Kerr, RK45Integrator, Schwarzschild

pytestmark = pytest.mark.gpu

NAMES = ("cls", "x", "v", "lam", "attempts", "accepted", "intensity", "color_temp", "rgb", "cross")


def check(renderer, scene, world):
    img, whole = renderer.render(scene, rays=True)
    w = scene.width * scene.spp
    for k in range(world):
        part = shard.shard_scene(scene, k, world)
        im, g = renderer.render(part, rays=True)
        assert np.array_equal(im, img[k::world])
        for name in NAMES:
            a, b = getattr(g, name), getattr(whole, name)
            if name == "rgb":
                b = b.reshape(scene.height, w, 3)[k::world].reshape(-1, 3)
            else:
                b = b.reshape(b.shape[:-1] + (scene.height, w))[..., k::world, :]
                b = b.reshape(a.shape)
            assert np.array_equal(a, b, equal_nan=a.dtype.kind == "f"), (name, k)


@pytest.mark.parametrize("kerr,disk,w,h,world", [
    (True, "thin", 256, 193, 2),        # 49,408 samples: rolled; its halves unrolled
    (False, "thin", 301, 200, 7),
    (True, "none", 223, 221, 3),
    (False, "none", 320, 160, 160),     # shards of one row
    (True, "volumetric", 310, 160, 2),
])
def test_fp64_whole_and_shards(renderer, kerr, disk, w, h, world):
    d = {"none": None, "thin": ThinDisk(6.0, 20.0, 3.0), "volumetric": AccretionDisk()}[disk]
    scene = Scene(Kerr(1.0, 0.9) if kerr else Schwarzschild(1.0),
                  Camera.inclined(30.0, math.radians(80.0), math.radians(60.0), w / h), w, h, d,
                  RenderOptions(sky=CheckerSky(18, 36, 0), max_steps=5000,
                                integrator=RK45Integrator(max_radius=200.0, rtol=1e-8, atol=1e-10,
                                                          stepper=abi.GG_STEPPER_DP45)))
    check(renderer, scene, world)


def test_mixed_band_whole_and_shards(renderer):
    """The near, near-extremal view: about 100,000 of its samples pass the band."""
    k = Kerr(1.0, 0.998)
    scene = Scene(k, Camera.inclined(15.0, math.radians(85.0), math.radians(60.0), 1.0), 1000, 1000,
                  ThinDisk(k.isco(), 25.0, 3.0),
                  RenderOptions(sky=CheckerSky(18, 36, 0), max_steps=20000,
                                precision=abi.GG_PREC_MIXED,
                                integrator=RK45Integrator(max_radius=200.0, rtol=1e-8, atol=1e-10,
                                                          stepper=abi.GG_STEPPER_DP45)))
    renderer.render(copy.copy(scene))
    assert renderer.stats().fp64_rays > 1 << 16
    part = shard.shard_scene(scene, 0, 4)
    renderer.render(part)
    assert 0 < renderer.stats().fp64_rays < 1 << 16
    check(renderer, scene, 4)
