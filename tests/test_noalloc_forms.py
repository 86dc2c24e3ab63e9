"""The no-allocation render on each form of the trace kernel.

No group pass follows it, and its small renders take the group form up to
another size than the context's: every output has to equal the context's, on
both sides of either line, supersampled too."""
from __future__ import annotations

import ctypes as C
import math

import numpy as np
import pytest

from gargantua_b200 import abi
from gargantua_b200.curved import AccretionDisk, Camera, RenderOptions, Scene, ThinDisk
from gargantua_b200.gr_core import Kerr, RK45Integrator, Schwarzschild

pytestmark = pytest.mark.gpu

DISKS = {"none": None, "volumetric": AccretionDisk(), "thin": ThinDisk(6.0, 20.0, 3.0)}


@pytest.mark.parametrize("kerr,disk,w,h,spa", [
    (True, "none", 90, 90, 1),
    (True, "none", 110, 110, 1),
    (True, "volumetric", 301, 200, 1),
    (False, "thin", 513, 512, 1),
    (True, "none", 1031, 1021, 1),
    (True, "none", 211, 150, 2),
    (False, "none", 680, 257, 2),   # the colours end at the array's end
])
def test_equals_the_contexts_render(renderer, gglib, kerr, disk, w, h, spa):
    import torch
    integ = RK45Integrator(max_radius=200.0, rtol=0.0 if disk != "thin" else 1e-8, atol=1e-10)
    scene = Scene(Kerr(1.0, 0.9) if kerr else Schwarzschild(1.0),
                  Camera.inclined(30.0, math.radians(89.0), math.radians(60.0), w / h), w, h,
                  DISKS[disk], RenderOptions(samples_per_axis=spa, integrator=integ))
    want, rays = renderer.render(scene, rays=True)
    n = scene.n_samples
    rgb = torch.zeros(w * h * 3, dtype=torch.uint8, device="cuda")
    x = torch.zeros(4 * n, dtype=torch.float64, device="cuda")
    attempts = torch.zeros(n, dtype=torch.int32, device="cuda")
    out = abi.gg_ray_out_t()
    out.x = C.cast(C.c_void_p(x.data_ptr()), C.POINTER(C.c_double))
    out.attempts = C.cast(C.c_void_p(attempts.data_ptr()), C.POINTER(C.c_uint32))
    s = torch.cuda.current_stream()
    for _ in range(2):
        assert gglib.gg_render_device_noalloc(*scene.c_args(), C.c_void_p(rgb.data_ptr()),
                                              C.byref(out), C.c_void_p(s.cuda_stream)) == abi.GG_OK
        s.synchronize()
        assert np.array_equal(rgb.cpu().numpy().reshape(h, w, 3), want)
        assert np.array_equal(x.cpu().numpy().reshape(4, n), rays.x)
        assert np.array_equal(attempts.cpu().numpy().view(np.uint32), rays.attempts)
        rgb.zero_()
        x.zero_()
        attempts.zero_()
