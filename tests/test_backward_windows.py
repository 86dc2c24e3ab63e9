"""The windows of the adjoint's backward, on the CPU.

Rays are listed by their number of segments, longest first, and taken back in
windows of at most `most` segments, or one ray where it alone has more.  The
library's windows have to be the greedy ones, whatever the counts: bins of one
ray and of many, rays longer than a window, at the front and alone in their bin."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

from gargantua_b200 import abi


def windows(gglib, counts, most):
    n_keys = len(counts)
    cap = int(sum(counts)) + 1
    out = np.zeros((cap, 6), np.uint64)
    n = C.c_uint64()
    c = (C.c_uint32 * n_keys)(*counts)
    st = gglib.gg_check_backward_windows(c, n_keys, most,
                                         out.ctypes.data_as(C.POINTER(C.c_uint64)), cap, C.byref(n))
    assert st == abi.GG_OK
    return out[:n.value].astype(np.int64)


def greedy(counts, most):
    """(first entry, end entry, first item, end item) of each window."""
    segs = [len(counts) - k for k, c in enumerate(counts) for _ in range(c)]
    out, e, item = [], 0, 0
    while e < len(segs):
        first, g0 = e, item
        while e < len(segs) and (e == first or item + segs[e] - g0 <= most):
            item += segs[e]
            e += 1
        out.append((first, e, g0, item))
    return out


def key_counts(pairs, n_keys):
    c = [0] * n_keys
    for segs, n in pairs:
        c[n_keys - segs] = n
    return c


CASES = [
    # (segments, rays) pairs, keys, most
    ([(1, 1)], 1, 1),
    ([(5, 3), (2, 7), (1, 40)], 6, 8),
    ([(3000, 1), (40, 50), (2, 900)], 3002, 2048),    # longer than a window, alone in its bin
    ([(3000, 2), (2500, 1), (2048, 1), (3, 11)], 3002, 2048),
    ([(3000, 1), (2999, 1)], 3002, 1),
    ([(314, 40), (22, 700), (2, 30000), (1, 5000)], 314, 1 << 11),
]


@pytest.mark.parametrize("pairs,n_keys,most", CASES)
def test_windows_are_the_greedy_ones(gglib, pairs, n_keys, most):
    counts = key_counts(pairs, n_keys)
    got = windows(gglib, counts, most)
    assert [tuple(w[:4]) for w in got] == greedy(counts, most)
    assert (got[:-1, 5] == got[1:, 4]).all()  # parallel segments follow on


def test_windows_random_counts(gglib):
    rng = np.random.default_rng(3)
    for _ in range(60):
        n_keys = int(rng.integers(1, 60))
        counts = [int(x) for x in rng.integers(0, 4, n_keys) * (rng.random(n_keys) < 0.4)]
        if not any(counts):
            counts[0] = 1
        most = int(rng.integers(1, 80))
        got = windows(gglib, counts, most)
        assert [tuple(w[:4]) for w in got] == greedy(counts, most), (counts, most)
