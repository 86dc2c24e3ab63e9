"""Which form of the FP64 trace kernel a render takes, on the CPU.

The reference's step: eight lanes per ray up to 2^13 samples (2^14 with the thin
disk), stages unrolled up to 2^18 (2^17 with the volumetric disk), in a loop above.
Full Dormand-Prince: unrolled up to 3 * 2^14.  Kerr renders below 2^20 samples have
their own register budget."""
from __future__ import annotations

import math

import pytest

from gargantua_b200 import abi
from gargantua_b200.curved import AccretionDisk, Camera, RenderOptions, Scene, ThinDisk
from gargantua_b200.gr_core import Kerr, RK45Integrator, Schwarzschild

LARGE, SMALL, UNROLLED, GROUP = range(4)
DISKS = {"none": None, "volumetric": AccretionDisk(), "thin": ThinDisk(6.0, 20.0, 3.0)}


def form(gglib, kerr, disk, w, h, dp45=False, **options):
    integ = RK45Integrator(max_radius=200.0, rtol=1e-8, atol=1e-10,
                           stepper=abi.GG_STEPPER_DP45 if dp45 else abi.GG_STEPPER_REFERENCE)
    scene = Scene(Kerr(1.0, 0.9) if kerr else Schwarzschild(1.0),
                  Camera.inclined(30.0, math.radians(80.0), math.radians(60.0), w / h), w, h,
                  DISKS[disk], RenderOptions(integrator=integ, **options))
    return gglib.gg_check_trace_form(*scene.c_args())


@pytest.mark.parametrize("kerr", [False, True])
@pytest.mark.parametrize("disk,group", [("none", 1 << 13), ("volumetric", 1 << 13),
                                        ("thin", 1 << 14)])
def test_few_samples(gglib, kerr, disk, group):
    assert form(gglib, kerr, disk, 1, 1) == GROUP
    assert form(gglib, kerr, disk, group // 64, 64) == GROUP
    assert form(gglib, kerr, disk, group // 64 + 1, 64) == UNROLLED
    assert form(gglib, kerr, disk, group // 256, 64, samples_per_axis=2) == GROUP
    assert form(gglib, kerr, disk, group // 256 + 1, 64, samples_per_axis=2) == UNROLLED
    assert form(gglib, kerr, disk, 1, 1, attempt_budget=1 << 40) != GROUP
    assert form(gglib, kerr, disk, 1, 1, dp45=True) == UNROLLED


@pytest.mark.parametrize("kerr,rolled", [(False, LARGE), (True, SMALL)])
@pytest.mark.parametrize("disk,dp45,last", [("none", False, 1 << 18), ("thin", False, 1 << 18),
                                            ("volumetric", False, 1 << 17), ("none", True, 3 << 14),
                                            ("thin", True, 3 << 14), ("volumetric", True, 3 << 14)])
def test_more_samples(gglib, kerr, rolled, disk, dp45, last):
    assert form(gglib, kerr, disk, last // 256, 256, dp45) == UNROLLED
    assert form(gglib, kerr, disk, last // 256 + 1, 256, dp45) == rolled
    assert form(gglib, kerr, disk, (1 << 12) - 1, 256, dp45) == rolled
    assert form(gglib, kerr, disk, 1 << 12, 256, dp45) == LARGE


def test_refused(gglib):
    assert form(gglib, True, "thin", 8, 8, dp45=True,
                precision=abi.GG_PREC_MIXED) == abi.GG_ERR_UNSUPPORTED
    assert form(gglib, True, "none", 8, 8, max_steps=0) == abi.GG_ERR_INVALID_ARG
