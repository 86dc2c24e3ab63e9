"""What a step leaves out, against the oracle, which leaves nothing out.

A step of a volumetric render whose midpoint is inside r_inner or beyond the
radius from which the density underflows takes no sine, exponential or
redshift; a step whose chord's box misses the scene's tests no object.  The
cases put the boundaries of both rules where rays go: disks thinner than a
step and thicker than the picture, a disk of no width, a camera inside the
disk's height, objects whose box has no thickness, one object far smaller
than a step, and objects around the camera.  The bar is the FP64 form's: at
every threshold from 1e-9 to 1e-6 no more samples beyond it than twice those
of the oracle rebuilt with fused multiply-adds, plus 0.1 % (at least 3)."""
from __future__ import annotations

import math

import numpy as np
import pytest

from gargantua_b200 import abi
from gargantua_b200.curved import (AccretionDisk, Camera, DiffuseLight, Lambertian, ProceduralSky,
                                   Quad, RenderOptions, Scene, SceneObjects, Sphere)
from gargantua_b200.gr_core import Kerr, RK45Integrator, Schwarzschild

pytestmark = pytest.mark.gpu


def scene(metric, r_cam, incl, disk, objects=None):
    return Scene(metric, Camera.inclined(r_cam, math.radians(incl), math.radians(60.0), 4 / 3), 64, 48,
                 disk, RenderOptions(sky=ProceduralSky(), max_steps=5000,
                                     integrator=RK45Integrator(max_radius=200.0)), objects)


def hold(g, o, f, name, mask):
    def rel(a):
        x, y = np.atleast_2d(getattr(a, name).T)[..., mask], np.atleast_2d(getattr(o, name).T)[..., mask]
        return (np.abs(x - y) / np.maximum(np.abs(y).max(axis=0), 1e-300)).max(axis=0)
    e_gpu, e_fma = rel(g), rel(f)
    slack = max(3, int(0.001 * mask.sum()))
    for t in (1e-9, 1e-8, 1e-7, 1e-6):
        assert (e_gpu > t).sum() <= 2 * (e_fma > t).sum() + slack, (name, t)


@pytest.mark.parametrize("kerr", [False, True])
@pytest.mark.parametrize("disk,r_cam,incl", [
    (AccretionDisk(6.0, 20.0, 0.02), 30.0, 80.0),
    (AccretionDisk(6.0, 20.0, 1.0), 30.0, 20.0),
    (AccretionDisk(6.0, 20.0, 40.0), 30.0, 75.0),
    (AccretionDisk(12.0, 12.0, 2.0), 40.0, 70.0),
    (AccretionDisk(3.0, 60.0, 1.5), 45.0, 89.0),
])
def test_volumetric_disk_bounds(renderer, oracle_mod, kerr, disk, r_cam, incl):
    sc = scene(Kerr(1.0, 0.9) if kerr else Schwarzschild(1.0), r_cam, incl, disk)
    _, g = renderer.render(sc, rays=True)
    _, o = oracle_mod.render(sc)
    _, f = oracle_mod.render(sc, variant="fma")
    same = g.cls == o.cls
    assert same.mean() > 0.999, same.mean()
    both = same & (f.cls == o.cls) & (o.intensity > 0.0)
    hold(g, o, f, "intensity", both)


def objects(kind):
    red, light = Lambertian((0.8, 0.2, 0.1)), DiffuseLight((1.0, 2.0, 0.5))
    if kind == "flat":  # an axis-aligned plane: a box of no thickness
        return SceneObjects([Quad((-20.0, -15.0, -15.0), (0.0, 30.0, 0.0), (0.0, 0.0, 30.0), red)])
    if kind == "small":
        return SceneObjects([Sphere((-25.0, 1.0, 0.5), 0.3, light)])
    if kind == "two":
        return SceneObjects([Sphere((-60.0, 20.0, 5.0), 8.0, light), Sphere((-40.0, -14.0, 0.0), 3.5, red)])
    return SceneObjects([Sphere((30.0 * math.cos(a), 30.0 * math.sin(a), 3.0 * b), 4.0, red)
                         for a in np.linspace(0.3, 6.0, 9) for b in (-2.0, 2.0)])


@pytest.mark.parametrize("kind", ["flat", "small", "two", "around"])
@pytest.mark.parametrize("kerr,disk", [(False, None), (True, AccretionDisk())])
def test_scene_box(renderer, oracle_mod, kind, kerr, disk):
    sc = scene(Kerr(1.0, 0.7) if kerr else Schwarzschild(1.0), 30.0, 90.0 if kind != "around" else 85.0,
               disk, objects(kind))
    _, g = renderer.render(sc, rays=True)
    _, o = oracle_mod.render(sc)
    _, f = oracle_mod.render(sc, variant="fma")
    same = g.cls == o.cls
    assert same.mean() > 0.998, same.mean()
    both = same & (f.cls == o.cls) & (o.cls == abi.GG_CLASS_SCENE)
    if (o.cls == abi.GG_CLASS_SCENE).any():
        hold(g, o, f, "rgb", both)
    else:  # the small sphere falls between the Kerr frame's rays
        assert kind == "small" and not (g.cls == abi.GG_CLASS_SCENE).any()
