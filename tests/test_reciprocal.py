"""The mixed form's FP32 reciprocal against 1/x in FP64.

The PTX ISA gives rcp.approx.ftz.f32 an error of at most 1 ulp, and takes
subnormal arguments and results as zero.  Every float mantissa is tried at
exponents spread over the normal numbers whose reciprocal is normal too (r^4 of
a stage from r = 1e-9 to 1e9 M, r^2 and the error scales from FLT_MIN up lie among
them), both signs, and the ends of the range."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

from gargantua_b200 import abi

pytestmark = pytest.mark.gpu

FLT_MIN = np.float32(2.0 ** -126)


@pytest.fixture(scope="module")
def device_rcp(gglib):
    import torch

    def call(x):
        d = torch.from_numpy(np.ascontiguousarray(x, np.float32)).cuda()
        out = torch.empty_like(d)
        st = gglib.gg_check_rcp(C.c_void_p(d.data_ptr()), C.c_void_p(out.data_ptr()), d.numel(),
                                None)
        assert st == abi.GG_OK
        return out.cpu().numpy()

    return call


@pytest.mark.parametrize("exponent", [-126, -120, -63, -10, -1, 0, 1, 23, 100, 124])
def test_within_one_ulp_of_every_mantissa(device_rcp, exponent):
    x = np.ldexp(np.arange(1 << 23, 1 << 24, dtype=np.float32), exponent - 23).astype(np.float32)
    want = 1.0 / x.astype(np.float64)
    ulp = np.spacing(want.astype(np.float32)).astype(np.float64)
    got = device_rcp(x).astype(np.float64)
    assert (np.abs(got - want) <= ulp).all()
    assert np.array_equal(device_rcp(-x[:4096]).astype(np.float64), -got[:4096])


def test_ends_of_the_range(device_rcp):
    inf = np.float32(np.inf)
    x = np.array([FLT_MIN, 2.0 ** 125, FLT_MIN / 2, 1e-45, 0.0, 3e38, inf], np.float32)
    got = device_rcp(x)
    want = 1.0 / x[:2].astype(np.float64)
    assert (np.abs(got[:2] - want) <= np.spacing(want.astype(np.float32))).all()
    # subnormal arguments count as 0 and subnormal reciprocals are 0
    assert (got[2:5] == inf).all() and (got[5:] == 0.0).all()
    assert np.isnan(device_rcp(np.array([np.nan], np.float32))).all()


def test_null_pointers(gglib):
    assert gglib.gg_check_rcp(None, None, 0, None) == abi.GG_OK
    assert gglib.gg_check_rcp(None, None, 4, None) == abi.GG_ERR_INVALID_ARG
