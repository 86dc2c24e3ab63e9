"""The host arrays of a render's outcomes, on the CPU.

The arrays that a render fills have to be like those of RayOutputs(n): the same
names, shapes and types, and each its own memory, so that a caller who keeps
one keeps that one alone and may resize it."""
from __future__ import annotations

import gc
import weakref

import numpy as np
import pytest

from gargantua_b200.curved import RayOutputs

NAMES = ("cls", "x", "v", "lam", "attempts", "accepted", "intensity", "color_temp", "rgb", "cross")


@pytest.mark.parametrize("n", [1, 7, 65536])
def test_arrays_to_fill_are_like_the_initialised_ones(n):
    a, b = RayOutputs(n), RayOutputs._to_fill(n)
    assert a.n == b.n == n and (a.cls == -1).all()
    for name in NAMES:
        x, y = getattr(a, name), getattr(b, name)
        assert (x.shape, x.dtype) == (y.shape, y.dtype)
        assert y.flags.owndata and y.flags.c_contiguous and y.flags.writeable and y.base is None
    assert {k for k in vars(a)} == {k for k in vars(b)}


def test_a_kept_array_keeps_no_other():
    out = RayOutputs._to_fill(1000)
    cross, cls = weakref.ref(out.cross), out.cls
    del out
    gc.collect()
    assert cross() is None
    cls.resize(10, refcheck=False)
    assert cls.shape == (10,)
