"""The steppers' rule for steady attempts, in the kernels' own code.

An attempt at max_step whose errors are well inside their scales skips the
step-size law (kSteadyErr, gg_device.cuh); each of the three steppers has its
form of the rule.  gg_check_steps runs a stepper over a frame's rays with the rule
and with the full law in its place: state, next step and counts have to be the
same bits after every number of attempts, with the relative and the absolute
error norm, and steps from far inside the tolerance to far outside."""
from __future__ import annotations

import ctypes as C
import math

import numpy as np
import pytest

from gargantua_b200 import abi
from gargantua_b200.curved import Camera
from gargantua_b200.gr_core import Kerr, RK45Integrator, Schwarzschild

pytestmark = pytest.mark.gpu

W, H = 97, 61
FORMS = {"reference": (0, abi.GG_STEPPER_REFERENCE, abi.GG_PREC_FP64),
         "dp45": (1, abi.GG_STEPPER_DP45, abi.GG_PREC_FP64),
         "mixed": (2, abi.GG_STEPPER_DP45, abi.GG_PREC_MIXED)}


def steps(gglib, metric, camera, integ, form, steady, attempts):
    import torch
    n = W * H
    state = torch.full((n, 10), float("nan"), dtype=torch.float64, device="cuda")
    counts = torch.full((n, 3), -1, dtype=torch.int32, device="cuda")
    m, c = metric.to_c(), camera.to_c()
    st = gglib.gg_check_steps(C.byref(m), C.byref(c), C.byref(integ), W, H, form, steady, attempts,
                              C.c_void_p(state.data_ptr()), C.c_void_p(counts.data_ptr()), None)
    assert st == abi.GG_OK
    return state.cpu().numpy().view(np.uint64), counts.cpu().numpy()


@pytest.mark.parametrize("form", FORMS)
@pytest.mark.parametrize("kerr", [False, True])
@pytest.mark.parametrize("rtol,max_step", [(1e-8, 0.05), (1e-8, 1.0), (1e-6, 0.37), (1e-10, 7.3),
                                           (0.0, 0.05), (0.0, 1.0)])
def test_rule_gives_the_full_laws_bits(gglib, form, kerr, rtol, max_step):
    number, stepper, precision = FORMS[form]
    metric = Kerr(1.0, 0.9) if kerr else Schwarzschild(1.0)
    camera = Camera.inclined(20.0, math.radians(75.0), math.radians(60.0), W / H)
    integ = RK45Integrator(max_radius=200.0, rtol=rtol, atol=1e-10, max_step=max_step,
                           stepper=stepper).to_c(10000, precision)
    for attempts in (1, 7, 40, 400):
        s, c = steps(gglib, metric, camera, integ, number, 1, attempts)
        t, d = steps(gglib, metric, camera, integ, number, 0, attempts)
        assert np.array_equal(c, d)
        assert np.array_equal(s, t)
    made, at_max = c[:, 0].sum(), c[:, 2].sum()
    assert made > W * H
    if max_step == 0.05:
        assert at_max > made / 2


def test_bad_arguments(gglib):
    m, c = Kerr(1.0, 0.5).to_c(), Camera.inclined(20.0, 1.0, 1.0, 1.0).to_c()
    i = RK45Integrator().to_c(100, abi.GG_PREC_FP64)
    p = C.c_void_p(256)
    call = gglib.gg_check_steps
    assert call(C.byref(m), C.byref(c), C.byref(i), 4, 4, 3, 1, 1, p, p, None) == abi.GG_ERR_INVALID_ARG
    assert call(C.byref(m), C.byref(c), C.byref(i), 4, 4, 0, 1, 1, None, p, None) == abi.GG_ERR_INVALID_ARG
    assert call(C.byref(m), C.byref(c), C.byref(i), 2048, 2048, 0, 1, 1, p, p, None) == abi.GG_ERR_INVALID_ARG
