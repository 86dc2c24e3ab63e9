"""The backward's split of a ray's chain, on one GPU.

A listed ray's last segments go to one lane in sequence and its earlier ones
to six lanes each; how many depends on the number of rays, and images of very
many segments are taken in windows.  The gradient of an image has to be the
sum of its row shards' gradients (the same per-pixel terms, summed in another
order, so to 1e-9 as for any row split), whose ray counts put them on other
sides of those rules: 768^2 is three windows and its shards one each, small
steps make chains of hundreds of segments, and the smallest images leave
warps part empty.  A loss that looks at one disk pixel, or at none, lists one
ray, or none."""
from __future__ import annotations

import numpy as np
import pytest

from gargantua_b200 import abi, diff
from gargantua_b200.gr_core import RK45Integrator

pytestmark = pytest.mark.gpu


def scene(side, max_step):
    integ = RK45Integrator(max_radius=200.0, rtol=1e-8, atol=1e-10, max_step=max_step,
                           stepper=abi.GG_STEPPER_DP45)
    return diff.DiffScene(width=side, height=side, integrator=integ)


def gradient(renderer, s, p, dl):
    import torch
    dr = diff.DiffRenderer(s, renderer)
    dr.render(p)
    dl = dl.contiguous()
    torch.cuda.current_stream().synchronize()
    return dr.backward(dl.data_ptr(), torch.cuda.current_stream().cuda_stream)


@pytest.mark.parametrize("side,world,max_step", [(768, 6, 1.0), (200, 9, 1.0), (160, 5, 0.05),
                                                 (33, 2, 1.0), (5, 2, 1.0)])
def test_shards_on_other_sides_of_the_split_rules(renderer, side, world, max_step):
    s = scene(side, max_step)
    p = diff.perturbed_params()
    target = diff.DiffRenderer(s, renderer).render(diff.target_params()).clone()
    img = diff.DiffRenderer(s, renderer).render(p).clone()
    dl = 2.0 * (img - target)
    whole = gradient(renderer, s, p, dl)
    parts = sum(gradient(renderer, s.shard(k, world), p, dl[k::world]) for k in range(world))
    assert np.isfinite(whole).all() and np.any(whole != 0.0)
    assert np.allclose(parts, whole, rtol=1e-9, atol=1e-12 * np.abs(whole).max()), (parts, whole)


def test_one_listed_ray_and_none(renderer):
    import torch
    s = scene(64, 1.0)
    p = diff.perturbed_params()
    img = diff.DiffRenderer(s, renderer).render(p).clone()
    assert np.array_equal(gradient(renderer, s, p, torch.zeros_like(img)), np.zeros(5))
    disk = diff.DiffRenderer(s, renderer).r.render(s.scene_at(p), rays=True)[1].cls == 2
    k = int(np.nonzero(disk)[0][disk.sum() // 2])
    dl = torch.zeros_like(img).view(-1, 3)
    dl[k] = 1.0
    g = gradient(renderer, s, p, dl.view_as(img))
    for i in (3, 4):  # r_in and q act on this pixel's colour alone
        h = 1e-6 * p[i]
        a, b = p.copy(), p.copy()
        a[i] += h
        b[i] -= h
        hi = diff.DiffRenderer(s, renderer).render(a).clone().view(-1, 3)[k].sum().item()
        lo = diff.DiffRenderer(s, renderer).render(b).clone().view(-1, 3)[k].sum().item()
        assert abs(g[i] - (hi - lo) / (2 * h)) <= 1e-4 * abs(g[i])
