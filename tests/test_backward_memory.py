"""The adjoint's backward where the device has little memory left.

Its step records take 2.1 GB at most, and no more than a quarter of what the
device has left: with less, the image is taken back in more and smaller windows,
with the same gradient (the same per-pixel terms summed in another order, so to
1e-9).  A second call reuses the first one's buffers.  An allocation that
fails (made to fail on the host) is tried at half the size, and remembered."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

from gargantua_b200 import abi, diff
from gargantua_b200.curved import Renderer

pytestmark = pytest.mark.gpu

FULL = (1 << 18) * 32 * 31 * 8  # records of the largest window
NO_LIMIT = 2 ** 64 - 1


class Fit:
    def __init__(self, gglib, side):
        self.lib = gglib
        self.r = Renderer(0)
        self.dr = diff.DiffRenderer(diff.DiffScene(width=side, height=side), self.r)
        target = self.dr.render(diff.target_params()).clone()
        self.dl = (2.0 * (self.dr.render(diff.perturbed_params()) - target)).contiguous()

    def memory(self, memory=NO_LIMIT, largest=NO_LIMIT):
        w, b = C.c_uint64(), C.c_uint64()
        assert self.lib.gg_check_backward_memory(self.r.handle, memory, largest, C.byref(w),
                                                 C.byref(b)) == abi.GG_OK
        return w.value, b.value

    def gradient(self):
        import torch
        self.dr.render(diff.perturbed_params())
        return self.dr.backward(self.dl.data_ptr(), torch.cuda.current_stream().cuda_stream)


@pytest.fixture
def fit(gglib, request):
    f = Fit(gglib, request.param)
    yield f
    f.r.close()


def close_to(a, b):
    return np.allclose(a, b, rtol=1e-9, atol=1e-12 * np.abs(b).max())


@pytest.mark.parametrize("fit", [640], indirect=True)
def test_records_do_not_exceed_the_largest_window(fit):
    fit.gradient()
    windows, held = fit.memory()
    assert windows > 1
    # the per-ray results: at most 42 doubles a segment, 11 a ray, and a quarter more
    assert FULL <= held <= FULL + 1.25 * 8 * (42 + 11) * (1 << 18)


@pytest.mark.parametrize("fit", [200], indirect=True)
@pytest.mark.parametrize("memory", [1 << 30, 200 << 20, 1 << 20, 0])
def test_little_memory_left(fit, memory):
    want = fit.gradient()
    one, held = fit.memory()
    assert one == 1
    fresh = Fit(fit.lib, 200)
    fresh.memory(memory)
    got = fresh.gradient()
    windows, small = fresh.memory(memory)
    assert close_to(got, want)
    assert (windows > 1) == (small < held)
    assert small <= max(1.25 * memory / 4, 30 << 20)
    assert windows > 1 or memory == 1 << 30
    again = fresh.gradient()
    assert fresh.memory(memory) == (windows, small) and close_to(again, want)
    fresh.r.close()


@pytest.mark.parametrize("fit", [200], indirect=True)
def test_allocations_that_fail(fit):
    want = fit.gradient()
    held = fit.memory()[1]
    fresh = Fit(fit.lib, 200)
    fresh.memory(largest=40 << 20)
    for _ in range(2):
        got = fresh.gradient()
        windows, small = fresh.memory(largest=40 << 20)
        assert close_to(got, want) and windows > 1 and small < held / 4
    # no size that can be had: an error, and the next call starts afresh
    starved = Fit(fit.lib, 200)
    starved.memory(largest=1)
    with pytest.raises(abi.GargantuaError):
        starved.gradient()
    assert starved.memory()[1] == 0
    assert close_to(starved.gradient(), want) and starved.memory()[0] == 1
    fresh.r.close()
    starved.r.close()
