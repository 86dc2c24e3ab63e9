"""The renders and gradients that are timed: what a user of this package has it do.

A case names one call through the package's public entry points and its
sizes: the four synchronous image functions of the reference
(``render`` .. ``render_with_disk_and_scene``), the device-pointer render
with the image left on the GPU, the render with per-sample outcomes, the
batched render, and the differentiable render with its backward.  ``draw``
gives more of the same kinds over the ranges the listed ones stand for.

A seed moves the camera, the spin, the sky and the scene, so two seeds of a
case are two frames of the same kind.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from gargantua_b200 import abi, workloads
from gargantua_b200 import curved as gc
from gargantua_b200.diff import DiffRenderer, DiffScene, kerr_image, target_params
from gargantua_b200.gr_core import Kerr, RK45Integrator, Schwarzschild

R_ESCAPE = 200.0  # the renderer's escape radius
_DEV = "cuda"


def listed():
    return [
        # the reference's own sanity render: a thumbnail, where a call's fixed
        # cost and one ray's chain of steps are all there is
        {"name": "thumbnail_32x24", "kind": "image", "metric": "schwarzschild", "disk": "none",
         "sky": "procedural", "scene": False, "width": 32, "height": 24, "spa": 1},
        # the command line's default picture with its volumetric disk
        {"name": "cli_disk_800x600", "kind": "image", "metric": "schwarzschild",
         "disk": "volumetric", "sky": "procedural", "scene": False, "width": 800, "height": 600,
         "spa": 1},
        # the command line with --metric kerr and --hdri, an odd size
        {"name": "kerr_sky_map_803x601", "kind": "image", "metric": "kerr", "disk": "none",
         "sky": "map", "scene": False, "width": 803, "height": 601, "spa": 1},
        # --scene lensed-spheres with the disk, supersampled
        {"name": "kerr_spheres_disk_spa2", "kind": "image", "metric": "kerr",
         "disk": "volumetric", "sky": "procedural", "scene": True, "width": 401, "height": 300,
         "spa": 2},
        # every sample's outcome to the host, as a study of single rays reads it
        {"name": "outcomes_schw_256", "kind": "outcomes", "metric": "schwarzschild",
         "stepper": 0, "width": 256, "height": 256},
        # one frame of an animation with the drop-in stepper, the image kept on the GPU
        {"name": "frame_fp64_1080p", "kind": "device", "view": "far", "precision": 0,
         "stepper": 0, "width": 1920, "height": 1080, "spp": 1},
        # a small ragged preview of it in the mixed form
        {"name": "preview_mixed_321x181", "kind": "device", "view": "far", "precision": 1,
         "stepper": 1, "width": 321, "height": 181, "spp": 1},
        # the benchmark's headline frame: the same picture in the mixed form
        {"name": "frame_mixed_1080p", "kind": "device", "view": "far", "precision": 1,
         "stepper": 1, "width": 1920, "height": 1080, "spp": 1},
        # the stress view: near-extremal hole, near camera, jittered samples
        {"name": "stress_mixed_2048x4", "kind": "device", "view": "near", "precision": 1,
         "stepper": 1, "width": 2048, "height": 2048, "spp": 4},
        # a training set's worth of uneven scenes in one launch
        {"name": "batch_64", "kind": "batch", "scenes": 64, "max_side": 512},
        # a parameter fit: image, L2 loss and the five-parameter gradient
        {"name": "gradient_128", "kind": "gradient", "side": 128},
        {"name": "gradient_512", "kind": "gradient", "side": 512},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["image", "image", "outcomes", "device", "device", "batch", "gradient"])
    if kind == "image":
        w = _log_int(rng, 24, 1000)
        h = max(16, int(w * rng.uniform(0.5, 1.2)))
        return {"kind": kind, "metric": rng.choice(["schwarzschild", "kerr"]),
                "disk": rng.choice(["none", "volumetric", "thin"] if w % 2 else
                                   ["none", "volumetric"]),
                "sky": rng.choice(["procedural", "map", "checker"]),
                "scene": w % 2 == 0 and rng.random() < 0.4, "width": w, "height": h,
                "spa": 2 if w < 500 and rng.random() < 0.4 else 1}
    if kind == "outcomes":
        w = _log_int(rng, 24, 400)
        return {"kind": kind, "metric": rng.choice(["schwarzschild", "kerr"]),
                "stepper": rng.choice([0, 1]), "width": w,
                "height": max(16, int(w * rng.uniform(0.5, 1.2)))}
    if kind == "device":
        precision = rng.choice([0, 1])
        w = _log_int(rng, 64, 2200)
        return {"kind": kind, "view": rng.choice(["far", "near"]), "precision": precision,
                "stepper": 1 if precision else rng.choice([0, 1]), "width": w,
                "height": max(32, int(w * rng.uniform(0.5, 1.0))),
                "spp": rng.choice([1, 1, 3]) if w < 1200 else 1}
    if kind == "batch":
        return {"kind": kind, "scenes": _log_int(rng, 3, 96),
                "max_side": 64 * rng.randint(1, 6)}
    return {"kind": kind, "side": _log_int(rng, 48, 480)}


# ---- inputs ------------------------------------------------------------------
def _integrator(stepper):
    return workloads.disk_integrator(abi.GG_STEPPER_DP45 if stepper else
                                     abi.GG_STEPPER_REFERENCE)


def _image_scene(case, rng):
    """A picture of the command line's kind: camera near (30 M, the equator)."""
    kerr = case["metric"] == "kerr"
    metric = Kerr(1.0, 0.9 + 0.05 * rng.random()) if kerr else Schwarzschild(1.0)
    cam = gc.Camera((0.0, 30.0 + rng.uniform(-1.0, 1.0), math.pi / 2.0 + rng.uniform(-0.05, 0.05),
                     0.0), (-1.0, 0.0, 0.0), (0.0, 0.0, 1.0), math.radians(60.0),
                    case["width"] / case["height"])
    sky = {"procedural": gc.ProceduralSky, "checker": lambda: gc.CheckerSky(18, 36, int(rng.integers(1 << 30))),
           "map": lambda: gc.HdriSky(workloads.synthetic_sky_map(1024, 512, int(rng.integers(1 << 30))))}
    disk = {"none": lambda: None, "volumetric": gc.AccretionDisk,
            "thin": lambda: gc.ThinDisk(6.0, 20.0, 3.0)}[case["disk"]]()
    opts = gc.RenderOptions(samples_per_axis=case["spa"], sky=sky[case["sky"]]())
    return gc.Scene(metric, cam, case["width"], case["height"], disk, opts,
                    workloads.lensed_spheres() if case["scene"] else None)


def _outcome_scene(case, rng):
    kerr = case["metric"] == "kerr"
    spin = 0.9 + 0.05 * rng.random()
    metric = Kerr(1.0, spin) if kerr else Schwarzschild(1.0)
    cam = gc.Camera.inclined(30.0 + rng.uniform(-1.0, 1.0), math.radians(80.0 + rng.uniform(-1, 1)),
                             math.radians(60.0), case["width"] / case["height"])
    return gc.Scene(metric, cam, case["width"], case["height"], gc.ThinDisk(6.0, 20.0, 3.0),
                    gc.RenderOptions(sky=gc.CheckerSky(18, 36, int(rng.integers(1 << 30))),
                                     max_steps=10000, integrator=_integrator(case["stepper"])))


def _device_scene(case, rng):
    far = case["view"] == "far"
    k = Kerr(1.0, 0.9 + rng.uniform(-0.01, 0.01) if far else 0.998 - 0.002 * rng.random())
    cam = gc.Camera.inclined((50.0 if far else 15.0) + rng.uniform(-0.5, 0.5),
                             math.radians((75.0 if far else 85.0) + rng.uniform(-1, 1)),
                             math.radians(60.0), case["width"] / case["height"])
    opts = gc.RenderOptions(sky=gc.CheckerSky(18, 36, int(rng.integers(1 << 30))),
                            max_steps=10000 if far else 50000,
                            jitter_spp=0 if case["spp"] == 1 else case["spp"],
                            seed=int(rng.integers(1 << 30)),
                            integrator=_integrator(case["stepper"]), precision=case["precision"])
    return gc.Scene(k, cam, case["width"], case["height"],
                    gc.ThinDisk(k.isco(), 30.0 if far else 25.0, 3.0), opts)


def _fit_params(seed):
    """Parameters of a fit under way, and of the image it fits."""
    rng = np.random.default_rng(seed)
    target = target_params()
    return target * (1.0 + 0.05 * rng.standard_normal(5)), target


def _batch(case, seed):
    """New holes, cameras and disks; the image sizes are the batch's own."""
    scenes = workloads.batch_scenes(case["scenes"], seed=seed, max_side=case["max_side"])
    sizes = workloads.batch_scenes(case["scenes"], seed=case["scenes"], max_side=case["max_side"])
    for s, t in zip(scenes, sizes):
        s.width, s.height = t.width, t.height
    return scenes


def prepare(case, seed):
    kind = case["kind"]
    rng = np.random.default_rng(seed)
    s = {"kind": kind}
    if kind == "image":
        s["scene"] = _image_scene(case, rng)
        if isinstance(s["scene"].options.sky, gc.HdriSky):
            # a program with a sky map keeps a renderer that holds it
            s["renderer"] = gc.Renderer(0)
            s["renderer"].set_hdri(s["scene"].options.sky)
    elif kind == "outcomes":
        s["renderer"] = gc.Renderer(0)
        s["scene"] = _outcome_scene(case, rng)
    elif kind == "device":
        s["renderer"] = gc.Renderer(0)
        s["scene"] = _device_scene(case, rng)
        s["image"] = torch.empty(case["height"], case["width"], 3, dtype=torch.uint8, device=_DEV)
    elif kind == "batch":
        s["renderer"] = gc.Renderer(0)
        s["scenes"] = _batch(case, seed)
        s["images"] = torch.empty(3 * sum(x.width * x.height for x in s["scenes"]),
                                  dtype=torch.uint8, device=_DEV)
    else:
        p, target = _fit_params(seed)
        s["renderer"] = DiffRenderer(DiffScene(width=case["side"], height=case["side"]))
        s["target"] = s["renderer"].render(target)
        s["p"] = torch.tensor(p, dtype=torch.float64, requires_grad=True)
    return s


def run(s):
    kind = s["kind"]
    if kind == "image":
        c = s["scene"]
        if "renderer" in s:
            return s["renderer"].render(c)[0]
        if c.objects is not None and c.disk is not None:
            return gc.render_with_disk_and_scene(c.metric, c.camera, c.disk, c.objects, c.width,
                                                 c.height, c.options)
        if c.objects is not None:
            return gc.render_with_scene(c.metric, c.camera, c.objects, c.width, c.height, c.options)
        if c.disk is not None:
            return gc.render_with_disk(c.metric, c.camera, c.disk, c.width, c.height, c.options)
        return gc.render(c.metric, c.camera, c.width, c.height, c.options)
    if kind == "outcomes":
        img, o = s["renderer"].render(s["scene"], rays=True)
        return {"image": img, "cls": o.cls, "x": o.x, "v": o.v, "lam": o.lam,
                "attempts": o.attempts.astype(np.int64), "accepted": o.accepted.astype(np.int64),
                "intensity": o.intensity, "color_temp": o.color_temp, "rgb": o.rgb,
                "cross": o.cross}
    if kind == "device":
        s["renderer"].render_device(s["scene"], s["image"].data_ptr(),
                                    stream=torch.cuda.current_stream().cuda_stream)
        return s["image"]
    if kind == "batch":
        s["renderer"].render_batch_device(s["scenes"], s["images"].data_ptr(),
                                          stream=torch.cuda.current_stream().cuda_stream)
        return s["images"]
    s["p"].grad = None
    img = kerr_image(s["p"], s["renderer"])
    ((img - s["target"]) ** 2).sum().backward()
    return {"image": img.detach(), "grad": s["p"].grad}


def work(case):
    """Bytes of the results, and the arithmetic of the geodesic steps: about one
    step per M of a ray's path to the escape sphere (the near view and the
    disk end many rays early), at the operations one attempt's right-hand
    sides and sums take in the kernels' formulation (flops.py)."""
    kind = case["kind"]
    kerr = case.get("metric", "kerr") == "kerr"
    per = (1677.0 if case.get("stepper", 0) or kind in ("batch", "gradient") else 1394.0) if kerr \
        else (956.0 if case.get("stepper", 0) else 673.0)
    if kind == "image":
        n = case["width"] * case["height"]
        return {"bytes": 3.0 * n, "flops": n * case["spa"] ** 2 * 230.0 * per}
    if kind == "outcomes":
        n = case["width"] * case["height"]
        return {"bytes": (3 + 4 + 8 * (4 + 4 + 1 + 1 + 1 + 3 + 8) + 8.0) * n,
                "flops": n * 190.0 * per}
    if kind == "device":
        n = case["width"] * case["height"]
        return {"bytes": 3.0 * n,
                "flops": n * case["spp"] * (200.0 if case["view"] == "far" else 70.0) * per}
    if kind == "batch":  # sides are uniform over 64, 128 .. max_side
        k = case["max_side"] // 64
        n = case["scenes"] * 4096.0 * (k + 1) * (2 * k + 1) / 6.0
        return {"bytes": 3.0 * n, "flops": n * 170.0 * per}
    n = float(case["side"] ** 2)
    # forward; the 44 % of the rays that end on the disk are gone back over,
    # each step's stages at about three times their forward work
    return {"bytes": 2 * 24.0 * n + 40.0, "flops": n * 165.0 * per + 0.44 * n * 60.0 * 3.0 * per}


# ---- the same in 64 bits, with torch alone ------------------------------------
# A batch of rays through the Dormand-Prince steps, all in double precision;
# for the gradient every quantity carries five imaginary parts (complex-step
# derivatives in the five parameters, exact to rounding), while the real parts
# alone decide which steps are taken.
_B = [[], [1 / 5], [3 / 40, 9 / 40], [44 / 45, -56 / 15, 32 / 9],
      [19372 / 6561, -25360 / 2187, 64448 / 6561, -212 / 729],
      [9017 / 3168, -355 / 33, 46732 / 5247, 49 / 176, -5103 / 18656],
      [35 / 384, 0.0, 500 / 1113, 125 / 192, -2187 / 6784, 11 / 84]]
_A = [0.0, 1 / 5, 3 / 10, 4 / 5, 8 / 9, 1.0, 1.0]
_D = [5179 / 57600, 0.0, 7571 / 16695, 393 / 640, -92097 / 339200, 187 / 2100, 1 / 40]
_DENSE = [-12715105075 / 11282082432, 0.0, 87487479700 / 32700410799, -10690763975 / 1880347072,
          701980252875 / 199316789632, -1453857185 / 822651844, 69997945 / 29380423]
_EPS = 1e-25  # the imaginary parts' size


def _re(z):
    return z.real if torch.is_complex(z) else z


def _first(z):
    """The real value: one per ray (all five derivative rows share it)."""
    return z.real[0] if torch.is_complex(z) else z


def _sincos(z):
    if not torch.is_complex(z):
        return torch.sin(z), torch.cos(z)
    s, c = torch.sin(z.real), torch.cos(z.real)
    return torch.complex(s, c * z.imag), torch.complex(c, -s * z.imag)


def _fn(z, f, df):
    if not torch.is_complex(z):
        return f(z)
    return torch.complex(f(z.real), df(z.real) * z.imag)


def _inv(z):
    return _fn(z, lambda x: 1.0 / x, lambda x: -1.0 / (x * x))


def _sqrt(z):
    return _fn(z, torch.sqrt, lambda x: 0.5 / torch.sqrt(x))


def _accel(a, r, th, v):
    """-Gamma v v of the Kerr metric (M = 1; a = 0 is Schwarzschild)."""
    s, c = _sincos(th)
    s2, sc, a2, r2 = s * s, s * c, a * a, r * r
    sig, dlt = r2 + a2 * (c * c), r2 - 2.0 * r + a2
    isg = _inv(sig)
    idl = _inv(dlt)
    f = 2.0 * r * isg                                   # 2 M r / Sigma
    f_r = 2.0 * isg - 2.0 * r * f * isg
    f_t = 2.0 * a2 * sc * f * isg
    sig_t = -2.0 * a2 * sc
    gtt_r, gtt_t = f_r, f_t                             # g_tt = -1 + f
    gtp_r, gtp_t = -a * s2 * f_r, -a * (2.0 * sc * f + s2 * f_t)
    gpp_r = s2 * (2.0 * r + a2 * s2 * f_r)
    gpp_t = 2.0 * sc * (r2 + a2 + a2 * s2 * f) + a2 * s2 * (2.0 * sc * f + s2 * f_t)
    grr_r = (2.0 * r - sig * (2.0 * r - 2.0) * idl) * idl
    grr_t = sig_t * idl
    isd = isg * idl
    utt = -((r2 + a2) * (r2 + a2) - a2 * dlt * s2) * isd
    utp = -2.0 * a * r * isd
    upp = (dlt - a2 * s2) * isd * _inv(s2)
    t, x, y, p = v
    e_t = x * (gtt_r * t + gtp_r * p) + y * (gtt_t * t + gtp_t * p)
    e_p = x * (gtp_r * t + gpp_r * p) + y * (gtp_t * t + gpp_t * p)
    q_r = gtt_r * t * t + 2.0 * gtp_r * t * p + gpp_r * p * p
    q_t = gtt_t * t * t + 2.0 * gtp_t * t * p + gpp_t * p * p
    a_r = -0.5 * dlt * isg * (grr_r * x * x + 2.0 * grr_t * x * y - 2.0 * r * y * y - q_r)
    a_t = -0.5 * isg * (sig_t * y * y + 4.0 * r * x * y - grr_t * x * x - q_t)
    return torch.stack([-(utt * e_t + utp * e_p), a_r, a_t, -(utp * e_t + upp * e_p)])


def _lin(ws, ks):
    out = None
    for w, k in zip(ws, ks):
        if w:
            out = w * k if out is None else out + w * k
    return out


def _wrap(x):
    """Polar angles reflected into [0, pi], azimuths into [0, 2 pi); in place."""
    th = x[2]
    lo, hi = _re(th) < 0.0, _re(th) > math.pi
    x[2] = torch.where(lo, -th, torch.where(hi, 2.0 * math.pi - th, th))
    ph = x[3] + math.pi * (lo | hi).to(x.dtype)
    x[3] = ph - 2.0 * math.pi * torch.floor(_re(ph) / (2.0 * math.pi)).to(x.dtype)
    return x


def _poly(c, s):
    y0, r2, r3, r4, r5 = c
    t = 1.0 - s
    return y0 + s * (r2 + t * (r3 + s * (r4 + t * r5)))


def _cross_dense(x, v, xa, va, ks, ws, h, comp, target):
    """Where component `comp` of the steps' continuous extension meets the target."""
    def coef(y0, y1, f):
        r2 = y1 - y0
        r3 = h * f[0] - r2
        return y0, r2, r3, r2 - h * f[6] - r3, h * _lin(_DENSE, f)
    # the weights sum to zero, so the position's sum may be taken over w - v
    cx = list(coef(x, xa, ws))
    cx[4] = h * _lin(_DENSE, [w - v for w in ws])
    cv = coef(v, va, ks)
    c = [_first(q[comp]) for q in cx]
    lo, hi = torch.zeros_like(c[0]), torch.ones_like(c[0])
    f_lo = c[0] - target
    s = 0.5 * lo + 0.5
    for k in range(80):  # bisection, then Newton's method inside the bracket
        f = _poly(c, s) - target
        below = (f < 0.0) == (f_lo < 0.0)
        lo, hi = torch.where(below, s, lo), torch.where(below, hi, s)
        t = 1.0 - s
        d = c[1] + (1 - 2 * s) * c[2] + s * (2 - 3 * s) * c[3] + 2 * s * t * (1 - 2 * s) * c[4]
        n = s - f / d
        s = torch.where((n > lo) & (n < hi) & (k > 5), n, 0.5 * (lo + hi)) if k < 79 else s
    if torch.is_complex(x):
        z = torch.complex(s, torch.zeros_like(s))
        t = 1.0 - s
        d = c[1] + (1 - 2 * s) * c[2] + s * (2 - 3 * s) * c[3] + 2 * s * t * (1 - 2 * s) * c[4]
        f = _poly([q[comp] for q in cx], z) - target
        s_all = z - f * (1.0 / d)
    else:
        s_all = s
    return s, _wrap(_poly(cx, s_all)), _poly(cv, s_all)


def _trace(a, x, v, stepper, r_in, r_out, max_steps, rtol=1e-8, atol=1e-10, h_max=1.0, h_min=1e-8,
           horizon_buffer=0.01):
    """Ends of the rays (x, v): a dict of class (0 horizon, 1 escaped, 2 disk, 3 out of
    steps), final x, v, lam and the crossing state (NaN where there is none)."""
    n = x.shape[-1]
    dev = x.device
    out = {"cls": torch.full((n,), 3, dtype=torch.int64, device=dev), "x": x.clone(),
           "v": v.clone(), "lam": torch.zeros(n, dtype=torch.float64, device=dev),
           "cx": torch.full_like(x, float("nan")), "cv": torch.full_like(v, float("nan"))}
    a_re = float(_re(torch.as_tensor(a)).reshape(-1)[0])
    r_h = 1.0 + math.sqrt(1.0 - a_re * a_re)
    live = torch.arange(n, device=dev)
    x, v = x.clone(), v.clone()
    h = torch.full((n,), 0.1, dtype=torch.float64, device=dev)
    lam = torch.zeros_like(h)
    ended = torch.zeros(n, dtype=torch.bool, device=dev)
    half_pi = 0.5 * math.pi

    def end(mask, cls, xs, vs, ls):
        i = live[mask]
        out["cls"][i] = cls
        out["x"][..., i], out["v"][..., i], out["lam"][i] = xs[..., mask], vs[..., mask], ls[mask]

    for step in range(max_steps):
        r = _first(x[1])
        esc, hor = (r > R_ESCAPE) & ~ended, (r < r_h + horizon_buffer) & ~ended
        end(esc, 1, x, v, lam)
        end(hor, 0, x, v, lam)
        ended = ended | esc | hor
        if step % 8 == 0:
            keep = ~ended
            if not bool(keep.any()):
                return out
            if float(keep.double().mean()) < 0.9:
                live, x, v, h, lam = live[keep], x[..., keep], v[..., keep], h[keep], lam[keep]
                ended = ended[keep]
        bad = torch.zeros_like(ended)
        ks, ws, xs = [], [], x
        for s in range(7):
            if stepper:
                w = v + h * _lin(_B[s], ks) if s else v
                xs = x + h * _lin(_B[s], ws) if s else x
            elif s < 6:
                xs, w = x + (h * _A[s]) * v, (v + h * _lin(_B[s], ks) if s else v)
            else:
                w = v + h * _lin(_B[6], ks)
            bad = bad | ~(torch.isfinite(_re(xs)).all(0).reshape(-1, h.numel())[0] & (_first(xs[1]) > 0.0))
            ws.append(w)
            ks.append(_accel(a, xs[1], xs[2], [w[0], w[1], w[2], w[3]]))
        vn, xn = ws[6], xs
        e = [c - d for c, d in zip(_B[6] + [0.0], _D)]
        vr, vnr = _real_rows(v), _real_rows(vn)
        q = h * _lin(e, [_real_rows(k) for k in ks]) / (atol + rtol * torch.maximum(vr.abs(), vnr.abs()))
        if stepper:
            xr, xnr = _real_rows(x), _real_rows(xn)
            qx = h * _lin(e, [_real_rows(w) - vr for w in ws]) / (atol + rtol * torch.maximum(xr.abs(), xnr.abs()))
            err = torch.sqrt(((q * q).sum(0) + (qx * qx).sum(0)) / 8.0)
        else:
            err = torch.sqrt((q * q).sum(0) / 4.0)
        acc = ((err < 1.0) | (h <= h_min)) & ~bad & ~ended
        grown = torch.where(err > 0.0, (h * 0.9 * (1.0 / err) ** 0.2).clamp(h_min, h_max), h)
        shrunk = torch.clamp(h * 0.9 * (1.0 / err) ** 0.25, min=h_min)
        h_new = torch.where(bad, 0.5 * h, torch.where(acc, grown, shrunk))
        raw_r = _first(xn[1])
        wrapped = _wrap(xn.clone())
        leaves = acc & (_first(x[1]) <= R_ESCAPE) & (raw_r > R_ESCAPE)
        d_b, d_a = _first(x[2]) - half_pi, _first(wrapped[2]) - half_pi
        meets = acc & (((d_b < 0.0) & (d_a >= 0.0)) | ((d_b > 0.0) & (d_a <= 0.0)))
        x_next = torch.where(acc, wrapped, x)
        v_next = torch.where(acc, vn, v)
        lam_next = torch.where(acc, lam + h, lam)
        for mask, comp, target in ((leaves, 1, R_ESCAPE), (meets, 2, half_pi)):
            if not bool(mask.any()):
                continue
            i = live[mask]
            pick = lambda z: z[..., mask]  # noqa: E731
            if stepper:
                sc, cx, cv = _cross_dense(pick(x), pick(v), pick(xn), pick(vn), [pick(k) for k in ks],
                                          [pick(w) for w in ws], h[mask], comp, target)
            else:
                sc = (target - _first(pick(x)[1])) / (pick(raw_r) - _first(pick(x)[1])) if comp == 1 \
                    else d_b[mask] / (d_b[mask] - d_a[mask])
                cx = _wrap(pick(x) + sc * (pick(xn) - pick(x)))
                cv = pick(v) + sc * (pick(vn) - pick(v))
            if comp == 1:
                out["cx"][..., i], out["cv"][..., i] = cx, cv
                if stepper:
                    end(mask, 1, x_next, v_next, lam_next)
                    ended = ended | mask
            else:
                on = (_first(cx[1]) >= r_in) & (_first(cx[1]) <= r_out) & ~ended[mask]
                j = i[on]
                cx[2] = torch.where(on, torch.full_like(cx[2], half_pi), cx[2])
                out["cls"][j] = 2
                for key, z in (("x", cx), ("cx", cx), ("v", cv), ("cv", cv)):
                    out[key][..., j] = z[..., on]
                out["lam"][j] = (lam[mask] + sc * h[mask])[on]
                hit = torch.zeros_like(ended)
                hit[mask.nonzero()[:, 0][on]] = True
                ended = ended | hit
        x, v, lam, h = x_next, v_next, lam_next, torch.where(ended, h, h_new)
    end(~ended, 3, x, v, lam)
    return out


def _real_rows(z):
    return z.real[:, 0] if torch.is_complex(z) else z


def _camera_rays(a, th, r, width, height, fov):
    """Initial (x, v) of the inclined camera's pixels, row-major, and sqrt(-g_tt) there."""
    dev = th.device
    px = torch.arange(width * height, device=dev)
    u = ((px % width).double() + 0.5) / width * 2.0 - 1.0
    w = 1.0 - ((px // width).double() + 0.5) / height * 2.0
    half_h = math.tan(0.5 * fov)
    half_w = half_h * (width / height)
    st, ct = _sincos(th)
    # forward (-st, 0, -ct), right (0, st, 0) / st, up (-ct, 0, st)
    dx, dy, dz = -st - w * half_h * ct, u * half_w + 0.0 * st, -ct + w * half_h * st
    norm = _sqrt(dx * dx + dy * dy + dz * dz)
    n_r, n_t, n_p = (dx * st + dz * ct) / norm, (dx * ct - dz * st) / norm, dy / norm
    sig, dlt = r * r + a * a * ct * ct, r * r - 2.0 * r + a * a
    g_tt = -(1.0 - 2.0 * r / sig)
    g_pp = (r * r + a * a + 2.0 * a * a * r * st * st / sig) * st * st
    one = torch.ones_like(n_r)
    x = torch.stack([0.0 * one, r * one, th * one, 0.0 * one])
    v = torch.stack([_sqrt(-1.0 / g_tt) * _sqrt(n_r * n_r + n_t * n_t + n_p * n_p),
                     n_r / _sqrt(sig / dlt), n_t / _sqrt(sig), n_p / _sqrt(g_pp)])
    return x, v, _sqrt(-g_tt)


def _redshift(a, s_obs, r, v, schwarzschild):
    """g of a circular equatorial orbiter at r, seen along v."""
    g_tt, g_tp = -(1.0 - 2.0 / r), -2.0 * a / r
    g_pp = r * r + a * a + 2.0 * a * a / r
    p_t, p_p = g_tt * v[0] + g_tp * v[3], g_tp * v[0] + g_pp * v[3]
    om = 1.0 / (r * _sqrt(r) + a)
    den = -(g_tt + 2.0 * g_tp * om + g_pp * om * om)
    moving = (_re(den) > 0.0) & (_re(r) > 3.0 if schwarzschild else _re(r) > 0.0)
    u_t = 1.0 / _sqrt(torch.where(moving, den, torch.ones_like(den)))
    e = torch.where(moving, -(p_t + p_p * om) * u_t, -p_t / _sqrt(torch.clamp(-_re(g_tt), min=1e-300).to(g_tt.dtype)))
    return (-p_t / s_obs) / e


def _checker(theta, phi, rows, cols, seed):
    """The seeded checkerboard's colours (n, 3) at the escape angles."""
    i = np.clip(np.floor(theta / (math.pi / rows)), 0, rows - 1).astype(np.uint64)
    j = np.clip(np.floor(phi / (2.0 * math.pi / cols)), 0, cols - 1).astype(np.uint64)

    def mix(z):
        z = z + np.uint64(0x9E3779B97F4A7C15)
        z = (z ^ (z >> np.uint64(30))) * np.uint64(0xBF58476D1CE4E5B9)
        z = (z ^ (z >> np.uint64(27))) * np.uint64(0x94D049BB133111EB)
        return z ^ (z >> np.uint64(31))
    z = mix(np.uint64(seed) ^ mix(i * np.uint64(cols) + j))
    base = np.where(((i + j) & np.uint64(1)) == 1, 0.9, 0.1)
    f = [((z >> np.uint64(21 * k)) & np.uint64(0x1FFFFF)).astype(np.float64) / 2097152.0 for k in range(3)]
    return np.stack([base * (0.75 + 0.25 * u) for u in f], axis=1)


def _colours(o, intensity, sky, stepper):
    """Linear colours (n, 3) of the ends, the disk's given its intensity."""
    cls = o["cls"].cpu().numpy()
    x = _real_rows(o["cx"] if stepper else o["x"]).cpu().numpy()
    rgb = np.zeros((cls.size, 3))
    m = cls == 1
    rgb[m] = _checker(x[2][m], x[3][m], sky.rows, sky.cols, sky.seed)
    t = (intensity / (1.0 + intensity))[cls == 2]
    rgb[cls == 2] = np.stack([t ** 0.5, t ** 1.2, t ** 2.5], axis=1)
    rgb[cls == 3] = (0.0, 0.0, 10.0 / 255.0)
    return rgb


def _exact_outcomes(case, seed):
    c = _outcome_scene(case, np.random.default_rng(seed))
    a = c.metric.spin if case["metric"] == "kerr" else 0.0
    th = torch.tensor([c.camera.position[2]], dtype=torch.float64, device=_DEV)
    r = torch.tensor([c.camera.position[1]], dtype=torch.float64, device=_DEV)
    x, v, s_obs = _camera_rays(a, th, r, c.width, c.height, c.camera.fov_y_radians)
    o = _trace(a, x, v, case["stepper"], 6.0, 20.0, 10000)
    disk = o["cls"] == 2
    rc = torch.where(disk, o["x"][1], torch.full_like(o["x"][1], 10.0))
    g = _redshift(a, s_obs, rc, o["v"], a == 0.0)
    q = 6.0 / rc
    zero = torch.zeros_like(g)
    inten = torch.where(disk, g ** 4 * q ** 3.0, zero).cpu().numpy()
    return {"image": None, "cls": None, "x": o["x"].cpu().numpy(), "v": o["v"].cpu().numpy(),
            "lam": o["lam"].cpu().numpy(), "attempts": None, "accepted": None, "intensity": inten,
            "color_temp": torch.where(disk, g * q ** 0.75, zero).cpu().numpy(),
            "rgb": _colours(o, inten, c.options.sky, case["stepper"]),
            "cross": torch.cat([o["cx"], o["cv"]]).cpu().numpy()}


def _exact_image(case, p, derivatives):
    """The differentiable render's linear image (n, 3) at p and, if asked, its
    derivative with respect to the five parameters (5, n, 3)."""
    sc = DiffScene(width=case["side"], height=case["side"])
    if derivatives:
        z = torch.tensor(p, dtype=torch.complex128, device=_DEV).reshape(5, 1, 1).repeat(1, 5, 1)
        z = z + 1j * _EPS * torch.eye(5, dtype=torch.float64, device=_DEV).reshape(5, 5, 1)
    else:
        z = torch.tensor(p, dtype=torch.float64, device=_DEV).reshape(5, 1)
    a, incl, r_cam, r_in, q_em = z
    x, v, s_obs = _camera_rays(a, incl, r_cam, sc.width, sc.height, sc.fov_y)
    o = _trace(a, x, v, 1, float(p[3]), sc.r_outer, sc.max_steps)
    disk = o["cls"] == 2
    rc = torch.where(disk, o["cx"][1], torch.full_like(o["cx"][1], 10.0))
    vc = torch.where(disk, o["cv"], torch.ones_like(o["cv"]))
    g = _redshift(a, s_obs, rc, vc, False)
    g2 = g * g
    log_q = _fn(r_in / rc, torch.log, lambda t: 1.0 / t)
    inten = g2 * g2 * _fn(q_em * log_q, torch.exp, torch.exp)
    i = torch.where(disk, _first(inten), torch.zeros_like(_first(inten)))
    rgb = torch.from_numpy(_colours(o, i.cpu().numpy(), sc.sky, 1)).to(i.device)
    if not derivatives:
        return rgb, None
    t = torch.where(disk, i / (1.0 + i), torch.ones_like(i))
    di = torch.where(disk, inten.imag / _EPS, torch.zeros_like(inten.imag)) / (1.0 + i) ** 2
    return rgb, torch.stack([0.5 * t ** -0.5 * di, 1.2 * t ** 0.2 * di, 2.5 * t ** 1.5 * di], dim=-1)


def exact(case, seed):
    """What ``run`` returns, in 64 bits by torch alone; image bytes have no such value."""
    if case["kind"] == "outcomes" and case["width"] * case["height"] <= 120000:
        return _exact_outcomes(case, seed)
    if case["kind"] == "gradient" and case["side"] <= 520:
        p, target = _fit_params(seed)
        want = _exact_image(case, target, False)[0]
        img, d = _exact_image(case, p, True)
        grad = (2.0 * (img - want) * d).sum(dim=(1, 2))
        return {"image": img.reshape(case["side"], case["side"], 3), "grad": grad}
    return None
