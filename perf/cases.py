"""The work this engine is used for, as cases that can be timed and checked.

    listed()            the cases: dicts of plain values
    draw(rng)           one more case of the ranges the listed ones stand for
    prepare(case, seed) what a program has in hand before the call (views, buffers, prepared tiles)
    run(state)          one pass through the public entry points; returns its outputs
    work(case)          bytes and operations the pass cannot do without
    exact(case, seed)   the outputs in 64 bits from plain torch, without the engine

Kinds of cases: "frame" (engine.render_frame_ssaa on every precision tier), "probe"
(engine.probe_iter_map, the depth probe a viewer runs before a frame), "recolor"
(engine.recolor_frame of a rendered iteration map), "batch" (a prepared batch's
persistent launch) and "grad" (adjoint.smooth_escape forward and backward).
A frame is rendered as an application does: the smooth map stays in the caller's device
buffer, the RGB image goes to the caller's pinned host buffer, and the call returns when
it is there.  The seed moves each view by up to 2 % of its width; a frame with a reference orbit by
a multiple of 0.45 widths besides, so that it has an orbit of its own.
"""
import json
import math
import os
import random
from decimal import Decimal, localcontext

import numpy as np
import torch

from fractura_b200 import adjoint, batch, engine, high_precision

BAILOUT = 65536.0
LN_BAILOUT_LOG = 1.7129177284488854  # ln(8 ln 2) as the engine's smooth value has it

# Views: centre, width, formula, depth and the iterations a pixel runs one at a time there
# on average (rounded; what `work` counts).  "deep" is the repository's 600-digit centre.
VIEWS = {
    # the whole sets, the first thing a viewer shows
    "home": dict(cx="-0.65", cy="0.0", width="4.0", ft=0, steps=25),
    "valley": dict(cx="-0.7436", cy="0.1318", width="0.02", ft=0, steps=150),
    "ship": dict(cx="-0.45", cy="-0.5", width="3.6", ft=1, steps=40),
    "julia": dict(cx="0.0", cy="0.0", width="3.0", ft=2, jx=-0.8, jy=0.156, steps=55),
    "multi3": dict(cx="0.0", cy="0.0", width="3.0", ft=4, n=3, kr=0.1, ki=0.2, steps=30),
    # double-double: boundary points of the Burning Ship and of the Mandelbrot set
    "ship_dd": dict(cx="0.124358169196707612717600709063601165799139991463562182617", cy="-0.396319792291520078678949617149807043564591069184643856716",
                    width="2e-17", ft=1, steps=300),
    "mandel_dd": dict(cx="-0.743643887037158704752191506114774", cy="0.131825904205311970493132056385139",
                      width="1e-18", ft=0, steps=8150),
    # perturbation, FP64 deltas
    "seahorse": dict(cx="-0.743643887037158704752191506114774", cy="0.131825904205311970493132056385139",
                     width="1e-26", ft=0, steps=1200),
    "deep": dict(cx="deep", cy="deep", width="1e-160", ft=0, steps=340),
    # FloatExp deltas: the spiral around c = i
    "abyss": dict(cx="0.0", cy="1.0", width="1e-1000", ft=0, steps=60),
}


def _frame(name, view, W, H, max_iter, **kw):
    c = dict(kind="frame", view=view, W=W, H=H, max_iter=max_iter, ssaa=1, scheme=0, mode="1e-300 (Perturbation)",
             glitch="Off (Single-Ref)", order=32, tol=1e-6, arith="ref_cpu", bla="reference", delta="fp64", hdr=False)
    c.update(kw)
    if name:
        c["name"] = name
    return c


DEEP_FORM = dict(glitch="One-Pass Rebasing", arith="fast", bla="accurate")


def listed():
    return [
        # the depth probe before every frame of a viewer with adaptive depth: the smallest call
        dict(name="probe_128x72", kind="probe", view="valley", W=128, H=72, max_iter=2000),
        # the first view of the set, histogram colours: an interactive frame
        _frame("home_640x360_hist", "home", 640, 360, 1000, scheme=11, mode="1e-12 (FP64)"),
        # a Julia set for print: odd size, 2x adaptive supersampling, the CUDA profile
        _frame("julia_1283x721_ssaa2", "julia", 1283, 721, 2000, ssaa=2, scheme=2, mode="1e-12 (FP64)", arith="ref_cuda"),
        # a Multibrot with large bounded regions at full HD, deep enough to cost
        _frame("multibrot_1920x1080", "multi3", 1920, 1080, 5000, scheme=6, mode="1e-12 (FP64)"),
        # double-double, both profiles
        _frame("ship_dd_1280x720_ssaa2", "ship_dd", 1280, 720, 20000, ssaa=2, mode="1e-24 (DD)"),
        _frame("mandel_dd_960x540", "mandel_dd", 960, 540, 10000, scheme=5, mode="1e-24 (DD)", arith="ref_cuda"),
        # perturbation with the application's default series start and one reference
        _frame("seahorse_1279x719_series4", "seahorse", 1279, 719, 30000, scheme=5, order=4, tol=1e-4),
        # the deep zoom this engine is for: leaps, rebasing, 200000 iterations
        _frame("deep_1920x1080", "deep", 1920, 1080, 200000, **DEEP_FORM),
        # below 1e-300: FloatExp deltas
        _frame("abyss_1920x1080", "abyss", 1920, 1080, 200000, arith="ref_cuda", bla="accurate"),
        # a mixed batch (a mosaic export, a tile server): formulas, sizes and depths mixed
        dict(name="batch_21_tiles", kind="batch", tiles=21, first=0, stride=3, arith="fast", delta="fp64"),
        # gradient step of a fit of a Julia and a Multibrot view
        dict(name="grad_512x512", kind="grad", W=512, H=512, max_iter=2000, julia=True, multi=3),
        # moving a palette slider over a 4K map with histogram colours
        dict(name="recolor_3840x2160_hist", kind="recolor", view="valley", W=3840, H=2160, max_iter=1000, scheme=11,
             contrast=1.0, hdr=False),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _size(rng, lo, hi):
    """A width log-uniform in [lo, hi], and a height for an aspect between 4:3 and 21:9; odd ones among them."""
    W = _log_int(rng, lo, hi)
    return W, max(8, int(W / rng.uniform(1.33, 2.33)))


def draw(rng):
    kind = rng.choice(["direct", "direct", "dd", "pert", "deep", "abyss", "batch", "grad", "recolor", "probe"])
    arith = rng.choice(["ref_cpu", "ref_cuda"])
    scheme = rng.choice([0, 1, 2, 5, 6, 8, 11])
    if kind == "probe":
        return dict(kind="probe", view=rng.choice(["home", "valley", "ship", "julia"]), W=rng.randint(96, 160),
                    H=rng.randint(54, 90), max_iter=_log_int(rng, 1000, 4000))
    if kind == "direct":
        W, H = _size(rng, 97, 1920)
        return _frame(None, rng.choice(["home", "valley", "ship", "julia", "multi3"]), W, H, _log_int(rng, 500, 4000),
                      scheme=scheme, ssaa=rng.choice([1, 1, 2]) if W < 1300 else 1, mode="1e-12 (FP64)", arith=arith,
                      hdr=rng.random() < 0.2)
    if kind == "dd":
        W, H = _size(rng, 97, 1000)
        view = rng.choice(["ship_dd", "mandel_dd"])  # the Mandelbrot point escapes from step 8048 on
        return _frame(None, view, W, H, _log_int(rng, 2000 if view == "ship_dd" else 8500, 10000), scheme=scheme,
                      ssaa=rng.choice([1, 2]) if W < 600 else 1, mode="1e-24 (DD)", arith=arith)
    if kind == "pert":
        W, H = _size(rng, 97, 1280)
        return _frame(None, "seahorse", W, H, _log_int(rng, 18000, 30000), scheme=scheme, arith=arith,
                      **rng.choice([dict(order=4, tol=1e-4), dict(order=8, tol=1e-4), dict(order=32, tol=1e-6)]))
    if kind == "deep":
        W, H = _size(rng, 97, 1920)
        f = rng.choice([DEEP_FORM, dict(DEEP_FORM, arith=arith), dict(bla="accurate", arith=arith),
                        dict(DEEP_FORM, delta="fp32", arith=arith)])
        return _frame(None, "deep", W, H, _log_int(rng, 20000, 200000), scheme=rng.choice([0, 5, 6]), **f)
    if kind == "abyss":
        W, H = _size(rng, 97, 1920)
        f = rng.choice([dict(arith=arith, bla="accurate"), dict(glitch="One-Pass Rebasing", delta="fp32", bla="accurate")])
        return _frame(None, "abyss", W, H, _log_int(rng, 20000, 200000), scheme=rng.choice([0, 5, 6]), **f)
    if kind == "batch":
        return dict(kind="batch", tiles=rng.randint(4, 10), first=rng.randrange(64), stride=rng.choice([3, 5, 7]),
                    arith=rng.choice(["fast", "ref_cuda"]), delta="fp64")
    if kind == "grad":
        n = _log_int(rng, 96, 512)
        julia = rng.random() < 0.6
        return dict(kind="grad", W=n, H=max(8, n - rng.randint(0, n // 2)), max_iter=_log_int(rng, 200, 2000), julia=julia,
                    multi=rng.choice([0, 3]) if julia else rng.choice([2, 3, 4]))
    W, H = _size(rng, 200, 3840)
    return dict(kind="recolor", view=rng.choice(["home", "valley", "julia"]), W=W, H=H, max_iter=1000, scheme=scheme,
                contrast=rng.choice([1.0, 0.8]), hdr=rng.random() < 0.3)


# ------------------------------------------------------------------ views
def _workloads():
    with open(os.path.join("tests", "golden", "workloads.json")) as f:
        return json.load(f)


def _move(cx, cy, w, seed, r, own_orbit):
    """The centre moved by the seed: up to 2 % of the width, and with own_orbit by a place of a grid of 0.45 widths
    (the engine shares an orbit between views within 0.4 widths of one another)."""
    step, i, j = (Decimal("0.45"), seed % 4, seed // 4 % 4) if own_orbit else (Decimal(0), 0, 0)
    with localcontext() as ctx:
        ctx.prec = 1200
        mx = step * (Decimal(i) - Decimal("1.5")) + Decimal(round(r.uniform(-0.02, 0.02), 9))
        my = step * (Decimal(j) - Decimal("1.5")) + Decimal(round(r.uniform(-0.02, 0.02), 9))
        return Decimal(cx) + w * mx, Decimal(cy) + w * my


def _view(name, seed, key):
    """(centre x, centre y, width) as Decimals, the centre moved by the seed, and the view's formula."""
    v = VIEWS[name]
    r = random.Random(f"{key} {name} {seed}")
    w = Decimal(v["width"])
    cx, cy = _workloads()["config3_centre"] if v["cx"] == "deep" else (v["cx"], v["cy"])
    x, y = _move(cx, cy, w, seed, r, name in ("seahorse", "deep", "abyss"))
    return x, y, w, v


def _formula(v):
    return dict(fractal_type=v["ft"], julia_cx=v.get("jx", 0.0), julia_cy=v.get("jy", 0.0), gen_n=v.get("n", 3),
                gen_kr=v.get("kr", 0.25), gen_ki=v.get("ki", 1.0))


def _host_rgb(H, W, hdr):
    return torch.empty((H, W, 3), dtype=torch.uint16 if hdr else torch.uint8).pin_memory().numpy()


def _thetas(case, seed):
    """The (theta, target theta, formula, degree) of each view of a gradient case: the target's parameters are
    N(0, 1e-3) away."""
    r = random.Random(f"grad {seed}")
    start = []
    if case["julia"]:
        start.append(([0.0, 0.0, math.log(3.0), -0.8, 0.156], 2, 2))
    if case["multi"]:
        start.append(([0.0, 0.0, math.log(3.0), 0.1, 0.2], 4, case["multi"]))
    out = []
    for th, ft, n in start:
        th = [t + r.gauss(0.0, 1e-3) for t in th]
        out.append((th, [t + r.gauss(0.0, 1e-3) for t in th], ft, n))
    return out


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("frame", "probe", "recolor"):
        x, y, w, v = _view(case["view"], seed, kind)
    if kind == "probe":
        return dict(kind=kind, args=(x, y, w, case["max_iter"], case["W"], case["H"]), kw=_formula(v))
    if kind == "frame":
        W, H = case["W"], case["H"]
        it = torch.empty((H, W), dtype=torch.float32, device="cuda")
        kw = dict(_formula(v), cmap_name="inferno", ssaa_factor=case["ssaa"], color_scheme_id=case["scheme"],
                  precision_mode=case["mode"], bbsa_tol=case["tol"], bbsa_order=case["order"], glitch_mode=case["glitch"],
                  is_hdr=case["hdr"], arith=case["arith"], bla_form=case["bla"], delta_form=case["delta"],
                  d_iter_buf=it, h_rgb_buf=_host_rgb(H, W, case["hdr"]))
        return dict(kind=kind, args=(W, H, case["max_iter"], x, y, w), kw=kw, iter=it)
    if kind == "recolor":
        W, H = case["W"], case["H"]
        it = torch.empty((H, W), dtype=torch.float32, device="cuda")
        engine.render_frame_ssaa(W, H, case["max_iter"], x, y, w, "inferno", d_iter_buf=it, **_formula(v))
        p = engine.RenderParameters(target_w=W, target_h=H, max_iter=case["max_iter"], color_scheme_id=case["scheme"],
                                    palette_offset=random.Random(seed).random(), color_contrast=case["contrast"],
                                    is_hdr=case["hdr"], d_iter_buf=it, h_rgb_buf=_host_rgb(H, W, case["hdr"]))
        return dict(kind=kind, params=p)
    if kind == "batch":
        high_precision.clear_reference_orbit_cache()  # the tiles' references are searched, not an earlier batch's
        all_tiles, r, tiles = _workloads()["config4_tiles"], random.Random(f"batch {seed}"), []
        for q in range(case["tiles"]):
            t = all_tiles[(case["first"] + q * case["stride"]) % len(all_tiles)]
            w = Decimal(t["width"])
            x, y = _move(t["cx"], t["cy"], w, seed, r, False)
            tiles.append(batch.Tile(cx=x, cy=y, width=w, W=t["W"], H=t["H"], max_iter=t["max_iter"],
                                    fractal_type=t["fractal_type"], julia_cx=t["julia_cx"], julia_cy=t["julia_cy"],
                                    gen_n=t["gen_n"], gen_kr=t["gen_kr"], gen_ki=t["gen_ki"],
                                    rebase=t["fractal_type"] in (0, 1, 4), delta_form=case["delta"]))
        return dict(kind=kind, batch=batch.prepare_batch(tiles, arith=case["arith"], bla_form="accurate"))
    views = []
    for th, target, ft, n in _thetas(case, seed):
        goal = adjoint.smooth_escape(torch.tensor(target, dtype=torch.float64), case["W"], case["H"], case["max_iter"], ft, n)
        theta = torch.tensor(th, dtype=torch.float64, device="cuda", requires_grad=True)
        views.append((theta, goal, ft, n))
    return dict(kind=kind, views=views, size=(case["W"], case["H"], case["max_iter"]))


def _loss(s, goal):
    """Mean squared difference over the pixels that escape in both."""
    return torch.where((s >= 0) & (goal >= 0), (s - goal) ** 2, torch.zeros_like(s)).mean()


def run(state):
    kind = state["kind"]
    if kind == "probe":
        return {"iter": engine.probe_iter_map(*state["args"], **state["kw"])}
    if kind == "frame":
        rgb = engine.render_frame_ssaa(*state["args"], **state["kw"])
        return {"iter": state["iter"], "rgb": rgb}
    if kind == "recolor":
        return {"rgb": engine.recolor_frame(state["params"])}
    if kind == "batch":
        state["batch"].render()
        return [[o["iter"], o["kmap"], o["glitch"]] for o in state["batch"].tiles_out]
    out = []
    for theta, goal, ft, n in state["views"]:
        theta.grad = None
        s = adjoint.smooth_escape(theta, *state["size"], ft, n)
        _loss(s, goal).backward()
        out.append({"s": s.detach(), "grad": theta.grad})
    return out


# ------------------------------------------------------------------- work
def _step_flops(ft, n, tier):
    """Operations of one iteration: the formula and its escape test."""
    direct = 8 if ft != 4 else 6 * (n - 1) + 10
    return {"fp64": direct, "dd": 62, "pert": direct + 5}[tier]


def work(case):
    kind = case["kind"]
    if kind == "batch":
        tiles = _workloads()["config4_tiles"]
        bytes_, flops = 0.0, 0.0
        for q in range(case["tiles"]):
            t = tiles[(case["first"] + q * case["stride"]) % len(tiles)]
            px, ft = t["W"] * t["H"], t["fractal_type"]
            bytes_ += px * 9.0
            # iterations a pixel runs one at a time: few where leaps carry the view, most of them in Multibrot views
            steps = {0: 300.0, 1: 500.0, 2: 60.0, 3: 60.0, 4: min(2000.0, 0.1 * t["max_iter"] + 500.0)}[ft]
            flops += px * steps * _step_flops(ft, t["gen_n"], "pert")
        return {"bytes": bytes_, "flops": flops}
    px = case["W"] * case["H"]
    if kind == "grad":
        flops = 0.0
        for on, n, steps in ((case["julia"], 2, 60.0), (bool(case["multi"]), case["multi"], 300.0)):
            if on:  # the orbit, then two complex derivative recurrences beside it
                flops += px * steps * (2 * (6 * (n - 1) + 6) + 16)
        views = int(case["julia"]) + int(bool(case["multi"]))
        return {"bytes": px * views * (8.0 + 8.0 + 8.0), "flops": flops}
    rgb = 6.0 if case.get("hdr") else 3.0
    if kind == "recolor":
        return {"bytes": px * (4.0 + rgb), "flops": px * 30.0}
    v = VIEWS[case["view"]]
    if kind == "probe":
        return {"bytes": px * 4.0, "flops": px * v["steps"] * _step_flops(v["ft"], v.get("n", 3), "fp64")}
    tier = "dd" if "DD" in case["mode"] else "fp64" if "FP64" in case["mode"] else "pert"
    return {"bytes": px * (4.0 + rgb), "flops": px * v["steps"] * _step_flops(v["ft"], v.get("n", 3), tier)}


# ------------------------------------------------------------------ exact
DEVICE = "cuda" if torch.cuda.is_available() else "cpu"


def _inv_ln(ft, n):
    return float(np.float32(1.0 / math.log(n))) if ft == 4 and n > 1 else 1.0 / math.log(2.0)


def _smooth(k, m, inv_ln):
    lm = torch.log(m)
    return torch.where(lm > 1.0, (k + 1.0) - (torch.log(0.5 * lm) - LN_BAILOUT_LOG) * inv_ln, k)


def _power(zx, zy, n):
    rx, ry = zx, zy
    for _ in range(n - 1):
        rx, ry = rx * zx - ry * zy, rx * zy + ry * zx
    return rx, ry


def _step(ft, n, kr, ki, zx, zy, cx, cy, order=0):
    """One iteration; order 1 rounds in another order."""
    if order:
        if ft != 4:
            ax, ay, sg = (zx, zy, 1.0) if ft in (0, 2) else (zx.abs(), zy.abs(), -1.0)
            return (zx - zy) * (zx + zy) + cx, (ax + ax) * ay + sg * cy
        px, py = _power(zx, zy, n)
        return px + (cx + (kr * zx - ki * zy)), py + (cy + (kr * zy + ki * zx))
    if ft in (0, 2):
        return zx * zx - zy * zy + cx, 2.0 * zx * zy + cy
    if ft in (1, 3):
        return zx * zx - zy * zy + cx, 2.0 * zx.abs() * zy.abs() - cy
    px, py = _power(zx, zy, n)
    return px + (kr * zx - ki * zy) + cx, py + (kr * zy + ki * zx) + cy


def _alive(keep, *ts):
    return [t[keep] if torch.is_tensor(t) else t for t in ts]


def _exact_direct(W, H, max_iter, x, y, w, v, f=1, order=0):
    """Smooth values [H, W] (float64) of direct iteration of a view in 64 bits."""
    dx, dy = float(w) / max(1, W - 1), float(w) * H / W / max(1, H - 1)
    off = (f - 1) * 0.5 / f
    i = torch.arange(W, dtype=torch.float64, device=DEVICE) + off
    j = torch.arange(H, dtype=torch.float64, device=DEVICE) + off
    px = ((float(x) - 0.5 * float(w)) + i * dx).expand(H, W).reshape(-1)
    py = ((float(y) + 0.5 * float(w) * H / W) - j * dy).reshape(H, 1).expand(H, W).reshape(-1)
    ft, n, kr, ki = v["ft"], v.get("n", 3), v.get("kr", 0.25), v.get("ki", 1.0)
    if ft in (2, 3):
        zx, zy, cx, cy = px, py, v["jx"], v["jy"]
    else:
        zx, zy, cx, cy = torch.zeros_like(px), torch.zeros_like(py), px, py
    s = torch.full((H * W,), -1.0, dtype=torch.float64, device=DEVICE)
    idx = torch.arange(H * W, device=DEVICE)
    for k in range(max_iter):
        if k % 8 == 0:  # an escaped orbit stays above the bailout or leaves the doubles: eight steps, then look
            if k > 0:
                keep = zx * zx + zy * zy <= BAILOUT
                if not bool(keep.all()):
                    sx, sy, scx, scy, sidx = _alive(~keep, zx0, zy0, cx0, cy0, idx)
                    for t in range(k - 8, k + 1):
                        sm = sx * sx + sy * sy
                        out = sm > BAILOUT
                        s[sidx[out]] = _smooth(torch.full_like(sm[out], float(t)), sm[out], _inv_ln(ft, n))
                        sx, sy, scx, scy, sidx = _alive(~out, sx, sy, scx, scy, sidx)
                        sx, sy = _step(ft, n, kr, ki, sx, sy, scx, scy, order)
                    zx, zy, cx, cy, idx = _alive(keep, zx, zy, cx, cy, idx)
                    if idx.numel() == 0:
                        break
            zx0, zy0, cx0, cy0 = zx, zy, cx, cy
        zx, zy = _step(ft, n, kr, ki, zx, zy, cx, cy, order)
    else:
        sx, sy, scx, scy, sidx = zx0, zy0, cx0, cy0, idx
        for t in range((max_iter - 1) // 8 * 8, max_iter):
            sm = sx * sx + sy * sy
            out = sm > BAILOUT
            s[sidx[out]] = _smooth(torch.full_like(sm[out], float(t)), sm[out], _inv_ln(ft, n))
            sx, sy, scx, scy, sidx = _alive(~out, sx, sy, scx, scy, sidx)
            sx, sy = _step(ft, n, kr, ki, sx, sy, scx, scy, order)
    return s.reshape(H, W)


def _orbit(ft, x, y, max_iter, bits):
    """The orbit of 0 at x + iy in fixed point with that many fractional bits: float64 values, escape included."""
    with localcontext() as ctx:
        ctx.prec = bits
        cx, cy = int((x * 2 ** bits).to_integral_value()), int((y * 2 ** bits).to_integral_value())
    zx = zy = 0
    re, im, one = [], [], 1 << bits

    def to_float(a):
        sh = max(0, a.bit_length() - 64)
        return math.ldexp(float(a >> sh), sh - bits)

    for _ in range(max_iter + 1):
        re.append(to_float(zx))
        im.append(to_float(zy))
        x2, y2 = (zx * zx) >> bits, (zy * zy) >> bits
        if x2 + y2 > 65536 * one:
            break
        xy = (zx * zy) >> bits
        zx, zy = (x2 - y2 + cx, 2 * xy + cy) if ft == 0 else (x2 - y2 + cx, 2 * abs(xy) - cy)
    return re, im


def _exact_delta(W, H, max_iter, x, y, w, v, f=1):
    """Smooth values [H, W] of a deep Mandelbrot or Burning Ship view: 64-bit deltas around a high-precision orbit of the
    view's centre, restarted from the orbit's start whenever |z| < |dz| or the orbit ends.  Far below the doubles'
    range a Mandelbrot delta is A dc until it can be held; None when that takes too many steps."""
    ft = v["ft"]
    depth = max(0, -w.adjusted())
    re, im = _orbit(ft, x, y, max_iter, int(depth * 3.33) + 128)
    scale = int(depth * 3.33) if depth > 290 else 0  # dc in units of 2^-scale
    with localcontext() as ctx:
        ctx.prec = depth + 60
        ws = float(w * 2 ** scale)
    off = (f - 1) * 0.5 / f
    i = (torch.arange(W, dtype=torch.float64, device=DEVICE) + off - (W - 1) * 0.5) * (ws / max(1, W - 1))
    j = (torch.arange(H, dtype=torch.float64, device=DEVICE) + off - (H - 1) * 0.5) * (ws * H / W / max(1, H - 1))
    dcx = i.expand(H, W).reshape(-1).contiguous()
    dcy = (-j).reshape(H, 1).expand(H, W).reshape(-1).contiguous()
    Z = torch.tensor([re, im], dtype=torch.float64, device=DEVICE)
    last = len(re) - 1
    dx, dy = torch.zeros_like(dcx), torch.zeros_like(dcy)
    k0 = 0
    if scale:
        if ft != 0:
            return None
        a, e = 0j, 0  # dz_k = a 2^e dc
        while k0 < last and (a == 0 or e + math.log2(abs(a)) < scale - 700):
            a = 2.0 * complex(re[k0], im[k0]) * a + math.ldexp(1.0, -e if -e > -1070 else -1070)
            k0 += 1
            if a != 0:
                _, ex = math.frexp(abs(a))
                a, e = a * math.ldexp(1.0, -ex), e + ex
        fct = math.ldexp(1.0, e - scale)
        dx, dy = (a.real * dcx - a.imag * dcy) * fct, (a.real * dcy + a.imag * dcx) * fct
        dcx, dcy = dcx * 0.0, dcy * 0.0
    s = torch.full((H * W,), -1.0, dtype=torch.float64, device=DEVICE)
    idx = torch.arange(H * W, device=DEVICE)
    m = torch.full((H * W,), k0, dtype=torch.int64, device=DEVICE)
    inv = _inv_ln(ft, 2)
    spent = 0
    for k in range(k0, max_iter):
        zx, zy = Z[0][m], Z[1][m]
        fx, fy = zx + dx, zy + dy
        m2 = fx * fx + fy * fy
        out = m2 > BAILOUT
        if bool(out.any()):
            s[idx[out]] = _smooth(torch.full_like(m2[out], float(k)), m2[out], inv)
            dx, dy, dcx, dcy, m, idx, zx, zy, fx, fy, m2 = _alive(~out, dx, dy, dcx, dcy, m, idx, zx, zy, fx, fy, m2)
            if idx.numel() == 0:
                break
        again = (m2 < dx * dx + dy * dy) | (m >= last)
        dx, dy = torch.where(again, fx, dx), torch.where(again, fy, dy)
        m = torch.where(again, torch.zeros_like(m), m)
        zx, zy = torch.where(again, torch.full_like(zx, re[0]), zx), torch.where(again, torch.full_like(zy, im[0]), zy)
        if ft == 0:
            dx, dy = (2.0 * zx + dx) * dx - (2.0 * zy + dy) * dy + dcx, 2.0 * ((zx + dx) * dy + zy * dx) + dcy
        else:
            sx, sy = torch.where(zx >= 0, 1.0, -1.0).double(), torch.where(zy >= 0, 1.0, -1.0).double()
            ax = torch.where((zx + dx) * sx >= 0, sx * dx, -sx * (2.0 * zx + dx))
            ay = torch.where((zy + dy) * sy >= 0, sy * dy, -sy * (2.0 * zy + dy))
            dx, dy = ((2.0 * zx + dx) * dx - (2.0 * zy + dy) * dy + dcx,
                      2.0 * (zx.abs() * ay + zy.abs() * ax + ax * ay) - dcy)
        m = m + 1
        spent += idx.numel() + 60000
        if spent > 6e10:
            return None
    return s.reshape(H, W)


def _exact_grad(case, seed, order=0):
    """Smooth values and d loss / d(cx, cy, ln w, Re P, Im P): the orbit with dz/dpixel and dz/dP beside it."""
    W, H, max_iter = case["W"], case["H"], case["max_iter"]

    def forward(th, ft, n):
        w = math.exp(th[2])
        i = torch.arange(W, dtype=torch.float64, device=DEVICE) / max(1, W - 1)
        j = torch.arange(H, dtype=torch.float64, device=DEVICE) / max(1, H - 1)
        gx, gy = i.expand(H, W).reshape(-1), j.reshape(H, 1).expand(H, W).reshape(-1)
        ux, uy = gx - 0.5, (H / W) * (0.5 - gy)
        x, y = th[0] + w * ux, th[1] + w * uy
        c = torch.complex(x, y)
        P = complex(th[3], th[4])
        z = c.clone() if ft == 2 else torch.zeros_like(c)
        A = torch.ones_like(c) if ft == 2 else torch.zeros_like(c)  # dz/dpixel
        B = torch.zeros_like(c)                                     # dz/dP
        s = torch.full((H * W,), -1.0, dtype=torch.float64, device=DEVICE)
        g = torch.zeros((H * W, 5), dtype=torch.float64, device=DEVICE)
        idx = torch.arange(H * W, device=DEVICE)
        inv = 1.0 / math.log(n)
        for k in range(max_iter):
            m = z.real * z.real + z.imag * z.imag
            out = m > BAILOUT
            if bool(out.any()):
                mo, zo, Ao, Bo, io = m[out], z[out], A[out], B[out], idx[out]
                lm = torch.log(mo)
                s[io] = _smooth(torch.full_like(mo, float(k)), mo, inv)
                q = (-2.0 * inv / (mo * lm)) * zo  # ds/dz as a 2-vector
                qa, qb = q.conj() * Ao, q.conj() * Bo
                g[io] = torch.stack([qa.real, -qa.imag, w * (qa.real * ux[io] - qa.imag * uy[io]), qb.real, -qb.imag], 1)
                z, A, B, c, idx = _alive(~out, z, A, B, c, idx)
                if idx.numel() == 0:
                    break
            if ft == 2:
                sq = torch.complex((z.real - z.imag) * (z.real + z.imag), (z.real + z.real) * z.imag) if order else z * z
                z, A, B = sq + P, 2.0 * z * A, 2.0 * z * B + 1.0
            else:
                zn = torch.ones_like(z)
                for _ in range(n - 1):
                    zn = zn * z
                d = n * zn + P
                z, A, B = (zn * z + (P * z + c) if order else zn * z + P * z + c), d * A + 1.0, d * B + z
        return s.reshape(H, W), g.reshape(H, W, 5)

    res = []
    for th, target, ft, n in _thetas(case, seed):
        s, g = forward(th, ft, n)
        goal, _ = forward(target, ft, n)
        up = torch.where((s >= 0) & (goal >= 0), 2.0 * (s - goal), torch.zeros_like(s)) / s.numel()
        res.append({"s": s, "grad": (up[..., None] * g).sum((0, 1))})
    return res


def _settled(values):
    """`values` of two orders of rounding: the first, or None where they differ by over 3 %.  Beside a boundary the escape
    step of a pixel is decided by rounding, and a view of such pixels has no value in 64 bits."""
    a, b = values
    return a if float((a - b).norm()) <= 0.03 * float(a.norm()) else None


def exact(case, seed):
    kind = case["kind"]
    if kind == "grad":
        both = [_exact_grad(case, seed, order) for order in (0, 1)]
        res = [{k: _settled([a[k], b[k]]) for k in a} for a, b in zip(*both)]
        return res if any(t is not None for r in res for t in r.values()) else None
    if kind in ("batch", "recolor"):  # over 20 s in plain torch; bytes only
        return None
    W, H, max_iter = case["W"], case["H"], case["max_iter"]
    x, y, w, v = _view(case["view"], seed, kind)
    if kind == "probe" or "FP64" in case["mode"]:
        s = _settled([_exact_direct(W, H, max_iter, x, y, w, v, case.get("ssaa", 1), order) for order in (0, 1)])
    else:
        s = _exact_delta(W, H, max_iter, x, y, w, v, case["ssaa"])
    if s is None:
        return None
    return {"iter": s} if kind == "probe" else {"iter": s, "rgb": None}
