# SPDX-License-Identifier: 0BSD
"""Timing cases of the framework's public entry points.

Each case is one call (or one short run of calls) that a program using this
package makes, over the sizes it makes them on: the FP64 step through
``Solver`` from the reference's default domain up to the 8192^2 raster, the
two FP32 fields, the extended physics, the batched process map, the
reference's own per-step call sequence, and the learned super-stepper's
inference and gradients.

``listed()`` names the cases, ``draw(rng)`` makes one more of the same ranges,
``prepare(case, seed)`` builds what the caller holds beforehand, ``run(state)``
is one pass and returns its results, ``work(case)`` what a pass cannot do
without, and ``exact(case, seed)`` the same results in plain 64-bit torch.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from hedgehog_lpbf_b200 import dropin
from hedgehog_lpbf_b200 import params as P
from hedgehog_lpbf_b200 import plan as PL
from hedgehog_lpbf_b200 import process_map as PM
from hedgehog_lpbf_b200 import surrogate as SG
from hedgehog_lpbf_b200.batch import Batch, Scenario, batch_opts
from hedgehog_lpbf_b200.solver import Solver, SolverF32, SolverF32K

DEVICE = "cuda:0"
SIDES = (256, 512, 1024, 2048)
LARGEST = 8192 * 8192 * 60           # cell-updates of the largest stepping case


def listed():
    return [
        # The reference's default single-track domain (1.6 x 0.6 mm, AMB2022
        # case 0 constants), one 64-step batch of its task: launches and the
        # laser's rows are all there is.
        {"name": "fp64_amb_240x120", "kind": "step", "nx": 240, "ny": 120, "steps": 64,
         "amb": True, "bc": 0, "preheat": 0.0},
        # The 512^2 workload: edges held at 300 K, laser along a track.
        {"name": "fp64_512_fixed", "kind": "step", "nx": 512, "ny": 512, "steps": 200,
         "amb": False, "bc": 1, "preheat": 0.0},
        # A part-sized domain whose sides are no multiple of anything (odd rows).
        {"name": "fp64_1021x763", "kind": "step", "nx": 1021, "ny": 763, "steps": 100,
         "amb": False, "bc": 0, "preheat": 0.0},
        # An ordinary field (the process map's largest side, run by itself).
        {"name": "fp64_2048", "kind": "step", "nx": 2048, "ny": 2048, "steps": 90,
         "amb": False, "bc": 0, "preheat": 0.0},
        # The large raster field.
        {"name": "fp64_8192", "kind": "step", "nx": 8192, "ny": 8192, "steps": 60,
         "amb": False, "bc": 0, "preheat": 0.0},
        # The same raster held in FP32, plain and compensated.
        {"name": "f32_8192", "kind": "f32", "nx": 8192, "ny": 8192, "steps": 48, "bc": 0},
        {"name": "f32k_4096", "kind": "f32k", "nx": 4096, "ny": 4096, "steps": 60, "bc": 0},
        # Temperature-dependent properties, one launch per step.
        {"name": "ext_4096", "kind": "ext", "nx": 4096, "ny": 4096, "steps": 16, "bc": 0},
        # A process map of mixed grid sides from one captured graph.
        {"name": "process_map_256", "kind": "map", "n256": 64, "n512": 64, "n1024": 64,
         "n2048": 64, "steps": 40, "tuned": True},
        # A reference build's per-step loop over the five launch wrappers.
        {"name": "wrappers_1024", "kind": "wrappers", "nx": 1024, "ny": 1024, "steps": 64,
         "fused": False},
        # One super-step of the learned stepper: features, network, update.
        {"name": "superstep_2048", "kind": "superstep", "nx": 2048, "ny": 2048},
        # The training batch: loss and gradients of 32 patches of 256^2.
        {"name": "gradients_32x256", "kind": "gradients", "batch": 32, "nx": 256, "ny": 256},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["step", "step", "step", "step", "f32", "f32k", "ext", "map", "wrappers",
                       "superstep", "gradients"])
    if kind == "map":
        n = _log_int(rng, 4, 192)
        cut = sorted(rng.randint(0, n) for _ in range(3))
        return {"kind": kind, "n256": cut[0], "n512": cut[1] - cut[0], "n1024": cut[2] - cut[1],
                "n2048": max(0, min(64, n - cut[2])) + (0 if cut[2] else 1),
                "steps": 12 * rng.randint(1, 4), "tuned": rng.random() < 0.5}
    if kind == "gradients":
        b = _log_int(rng, 1, 32)
        return {"kind": kind, "batch": b, "nx": rng.randint(64, 256), "ny": rng.randint(64, 256)}
    nx = _log_int(rng, 120, 8192 if kind in ("step", "f32", "f32k") else 4096)
    ny = max(64, min(8192, int(nx * math.exp(rng.uniform(-0.9, 0.9)))))
    if kind in ("f32", "f32k") or rng.random() < 0.5:
        nx = max(4, nx // 4 * 4)          # whole vectors per row (required by the FP32 fields)
    if kind == "superstep":
        return {"kind": kind, "nx": min(nx, 3072), "ny": min(ny, 3072)}
    steps = _log_int(rng, 4, 240)
    steps = max(1, min(steps, LARGEST // 4 // (nx * ny)))
    if kind == "step":
        return {"kind": kind, "nx": nx, "ny": ny, "steps": steps, "amb": rng.random() < 0.2,
                "bc": 1 if rng.random() < 0.3 else 0,
                "preheat": 60.0 if rng.random() < 0.15 else 0.0}
    if kind == "wrappers":
        return {"kind": kind, "nx": nx, "ny": ny, "steps": min(steps, 128),
                "fused": rng.random() < 0.5}
    if kind == "ext":
        steps = max(1, min(steps, 48))
    return {"kind": kind, "nx": nx, "ny": ny, "steps": steps, "bc": 1 if rng.random() < 0.2 else 0}


# ---- inputs ------------------------------------------------------------------


def _problem(case, seed):
    """Constants, plan and melt threshold of a single-field case.  The seed
    draws the laser (power, speed, spot as in the process map) and where on
    its scan the run starts; returns (k, plan, Tm, domain, past) with `past`
    the laser positions before the run (oldest last) and their spacing."""
    r = np.random.default_rng([seed, 11])
    nx, ny, n = case["nx"], case["ny"], case.get("steps", SG.STEPS)
    if case.get("amb"):
        mat, pr = P.Material(), P.apply_case("0", P.Process())
        dx = 1.6e-3 / 239
        dom = P.Domain(Lx=(nx - 1) * dx, Ly=(ny - 1) * 0.6e-3 / 119, nx=nx, ny=ny)
        dt = P.dt_cfl(mat, dom)
    else:
        mat, pr = P.benchmark_material_process(P=100.0 + 300.0 * r.random(),
                                               V=0.5 + 1.5 * r.random(),
                                               r0=35e-6 + 35e-6 * r.random())
        dom = P.Domain(Lx=(nx - 1) * 5e-6, Ly=(ny - 1) * 5e-6, nx=nx, ny=ny)
        dt = P.dt_fraction(mat, dom, 0.1 if case["kind"] == "ext" else 0.2)
    pr.Tsub = pr.Tamb + case.get("preheat", 0.0)
    k = P.make_const(mat, pr, dom, dt)
    # a serpentine over the middle of the domain; start somewhere inside a track
    track = 0.6 * dom.Lx
    tracks = max(1, min(10, int(0.6 * dom.Ly / 100e-6)))
    t_track = track / pr.V
    t0 = (int(r.integers(0, tracks)) + 0.25 + 0.5 * r.random()) * t_track
    plan = PL.raster(dom, dt, n, V=pr.V, hatch=100e-6, track_len=track, n_tracks=tracks,
                     angle=0.0, center=(0.5 * dom.Lx, (0.5 + 0.02 * r.random()) * dom.Ly), t0=t0)
    gap = 0.5 * pr.r0 / pr.V
    m = max(1, min(64, int(t0 / gap)))
    times = t0 - gap * (np.arange(m) + 0.5)
    past = [PL.raster(dom, dt, 1, V=pr.V, hatch=100e-6, track_len=track, n_tracks=tracks,
                      angle=0.0, center=(0.5 * dom.Lx, float(plan["y_l"][0])), t0=float(t))
            for t in times]
    return k, plan, mat.Tm, dom, (past, gap)


def _heated(k, past, gap):
    """A field as a scan leaves it: the heat of the laser's last positions,
    each spread by diffusion and decayed by the substrate loss since."""
    dev = torch.device(DEVICE)
    x = torch.arange(k.nx, dtype=torch.float64, device=dev) * k.dx
    y = torch.arange(k.ny, dtype=torch.float64, device=dev) * k.dy
    rate = k.peak_S / (k.rho_cp * k.h)
    tau = k.rho_cp * k.h * k.dSub / k.K
    gx, gy = [], []
    for i, tick in enumerate(past):
        t = gap * (i + 0.5)
        w0 = 0.5 / k.inv_r0_sq
        w = w0 + 4.0 * k.alpha * t
        gy.append(rate * gap * (w0 / w) * math.exp(-t / tau)
                  * torch.exp(-(y - float(tick["y_l"][0])) ** 2 / w))
        gx.append(torch.exp(-(x - float(tick["x_l"][0])) ** 2 / w))
    return k.Tamb + torch.stack(gy, 1) @ torch.stack(gx, 0)


def _map_scenarios(case, seed):
    out = []
    i = 1000 * (seed + 1)
    for side in SIDES:
        for _ in range(case["n%d" % side]):
            d = PM.draw(i)
            i += 1
            k, plan, mat = PM.scenario_inputs(d, case["steps"], side=side)
            out.append(Scenario(k=k, plan=plan, Tm=mat.Tm))
    return out


def _net_params(seed):
    r = np.random.default_rng([seed, 5])
    ps = SG.init_params(seed)
    return [(w, r.normal(0.0, 0.05, b.shape)) for w, b in ps]


def _patches(case, seed):
    """A training batch: features around a laser and the changes to learn."""
    b, ny, nx = case["batch"], case["ny"], case["nx"]
    dev = torch.device(DEVICE)
    r = np.random.default_rng([seed, 7])
    g = torch.Generator(device="cpu").manual_seed(int(seed) + 17)
    col = lambda a: torch.as_tensor(a, dtype=torch.float32, device=dev).view(b, 1, 1)   # noqa: E731
    cy, cx = col(r.uniform(0.2, 0.8, b) * ny), col(r.uniform(0.2, 0.8, b) * nx)
    amp, src = col(r.uniform(0.5, 2.0, b)), col(r.uniform(0.5, 1.5, b))
    Y = torch.arange(ny, dtype=torch.float32, device=dev).view(1, ny, 1)
    X = torch.arange(nx, dtype=torch.float32, device=dev).view(1, 1, nx)
    r2 = (Y - cy) ** 2 + (X - cx) ** 2
    tail = torch.exp(-((Y - cy) ** 2) / 300.0) * torch.sigmoid((cx - X) / 4.0)
    T = amp * (tail * torch.exp(-(cx - X).clamp(min=0.0) / 80.0) + 0.3 * torch.exp(-r2 / 800.0))
    S = src * torch.exp(-r2 / 50.0)
    px = ((X - cx) * 0.05).clamp(-8.0, 8.0).expand(b, ny, nx)
    py = ((Y - cy) * 0.05).clamp(-8.0, 8.0).expand(b, ny, nx)
    x4 = torch.stack([T, S, px, py], -1).to(torch.bfloat16).contiguous()
    noise = torch.randn((b, ny, nx), generator=g).to(dev)
    tgt = (8.0 * S - 0.5 * T + 0.05 * noise).contiguous()
    return x4, tgt


def prepare(case, seed):
    kind = case["kind"]
    st = {"kind": kind}
    if kind == "map":
        # rows as the autotuner picks them for the mixed batch, or the defaults
        opts = batch_opts(depth=2, rows=(48, 48, 96, 384)) if case["tuned"] else batch_opts()
        b = Batch(_map_scenarios(case, seed), case["steps"], opts=opts, device=DEVICE)
        b.capture(0, case["steps"])
        return {**st, "batch": b, "Tamb": [s.k.Tamb for s in b.scenarios]}
    if kind == "gradients":
        x4, tgt = _patches(case, seed)
        return {**st, "net": SG.Net(_net_params(seed), device=DEVICE), "x4": x4, "target": tgt}
    k, plan, Tm, dom, past = _problem(case, seed)
    if kind == "wrappers":
        return {**st, "k": k, "dom": dom, "plan": plan, "Tm": Tm, "fused": case["fused"]}
    if kind == "superstep":
        T0 = _heated(k, *past)
        return {**st, "k": k, "plan": plan, "T0": T0, "T": torch.empty_like(T0),
                "net": SG.Net(_net_params(seed), device=DEVICE)}
    if kind in ("f32", "f32k"):
        cls = SolverF32 if kind == "f32" else SolverF32K
        s = cls(k, bc=case["bc"], T_edge=k.Tamb, Tm=Tm, device=DEVICE)
        return {**st, "solver": s, "plan": plan, "Tamb": k.Tamb, "ring": s.new_ring(len(plan))}
    s = Solver(k, phys=1 if kind == "ext" else 0, bc=case["bc"], T_edge=k.Tamb, Tm=Tm,
               device=DEVICE)
    return {**st, "solver": s, "plan": plan, "T0": _heated(k, *past),
            "ring": s.new_ring(len(plan))}


# ---- one pass ----------------------------------------------------------------


def _ring_views(ring, n):
    """Peak temperatures, argmax indices and molten rows of a device ring."""
    return {"tmax": ring.view(torch.float64).view(n, 3)[:, 0],
            "arg": ring.view(torch.int64).view(n, 3)[:, 1],
            "rows": ring.view(torch.int32).view(n, 6)[:, 4:6]}


def run(state):
    kind = state["kind"]
    if kind == "map":
        b = state["batch"]
        for i, t in enumerate(state["Tamb"]):
            b.set_field(i, t)
        b.run(0, b.n_steps, use_graph=True)
        sides = {}
        for i, s in enumerate(b.scenarios):
            sides.setdefault(s.k.nx, []).append(b.field(i))
        rings = torch.stack(b.rings)
        return {"fields": {str(n): torch.stack(f) for n, f in sides.items()},
                "rings": _ring_views(rings.view(-1), rings.numel() // 24)}
    if kind == "gradients":
        loss = state["net"].gradients(state["x4"], state["target"])
        return {"loss": loss, "grads": state["net"].grads_vector()}
    if kind == "wrappers":
        r = dropin.run(state["k"], state["dom"], state["plan"], state["Tm"],
                       fused=state["fused"], device=DEVICE)
        p = r["partials"]
        return {"field": r["field"], "tmax": p["tmax"], "arg": p["arg"], "ymin": p["ymin"],
                "ymax": p["ymax"]}
    if kind == "superstep":
        T = state["T"]
        T.copy_(state["T0"])
        x4 = SG.features(T, state["k"], state["plan"])
        y = state["net"].forward(x4[None])
        SG.apply(T, y[0])
        return {"y": y, "T": T}
    s, plan, ring = state["solver"], state["plan"], state["ring"]
    if kind in ("f32", "f32k"):
        s.set_field(state["Tamb"])
        s.advance(plan, ring)
        f = s.field if kind == "f32" else {"hi": s.hi[s.cur], "lo": s.lo[s.cur]}
        return {"field": f, "ring": _ring_views(ring, len(plan))}
    s.set_field(state["T0"])
    s.advance(plan, ring)
    return {"field": s.field, "ring": _ring_views(ring, len(plan))}


# ---- the work of a pass ------------------------------------------------------

STEP_FLOPS = 15          # Laplacian 5, loss 7, update 3 per cell and step
EXT_FLOPS = 41           # two face fluxes, k and cp lines, losses, division, update
NET_FLOPS = 2 * 9 * (4 * 32 + 3 * 32 * 32 + 32)


def work(case):
    kind = case["kind"]
    if kind == "map":
        cells = sum(case["n%d" % s] * s * s for s in SIDES)
        n = sum(case["n%d" % s] for s in SIDES)
        return {"bytes": 16.0 * cells + 24.0 * n * case["steps"],
                "flops": float(STEP_FLOPS) * cells * case["steps"]}
    if kind == "gradients":
        px = case["batch"] * case["ny"] * case["nx"]
        w = 4.0 * sum(32 * (9 * c + 1) for c in (4, 32, 32, 32))
        return {"bytes": 12.0 * px + 2 * w,
                "flops": (3.0 * NET_FLOPS - 2 * 9 * 4 * 32) * px}
    px = case["nx"] * case["ny"]
    if kind == "superstep":
        return {"bytes": 20.0 * px, "flops": float(NET_FLOPS) * px}
    n = case["steps"]
    cell = 8 if kind == "f32" else 16
    return {"bytes": float(cell) * px + 24.0 * n,
            "flops": float(EXT_FLOPS if kind == "ext" else STEP_FLOPS) * px * n}


# ---- the same results in plain 64-bit arithmetic ------------------------------

_TS = (298.0, 473.0, 673.0, 873.0, 1073.0, 1273.0, 1473.0, 1533.0, 1609.0)
_KS = (8.9, 12.9, 15.8, 18.7, 21.9, 25.6, 28.6, 29.3, 29.6)
_CS = (435.0, 479.0, 515.0, 558.0, 580.0, 628.0, 670.0, 685.0, 720.0)


def _table(T, ys):
    ts = torch.tensor(_TS, dtype=torch.float64, device=T.device)
    ys = torch.tensor(ys, dtype=torch.float64, device=T.device)
    c = T.clamp(_TS[0], _TS[-1])
    i = torch.bucketize(c, ts).clamp(1, len(_TS) - 1)
    f = (c - ts[i - 1]) / (ts[i] - ts[i - 1])
    return ys[i - 1] + f * (ys[i] - ys[i - 1])


def _edge_diffs(T):
    """Differences across the inner faces along x and along y."""
    return T[:, 1:] - T[:, :-1], T[1:] - T[:-1]


def _divergence(fx, fy, sx, sy):
    out = torch.zeros((fy.shape[0] + 1, fx.shape[1] + 1), dtype=torch.float64, device=fx.device)
    fx, fy = fx * sx, fy * sy
    out[:, :-1] += fx
    out[:, 1:] -= fx
    out[:-1] += fy
    out[1:] -= fy
    return out


def _exact_run(k, plan, T, bc, T_edge, phys=0):
    x = torch.arange(k.nx, dtype=torch.float64, device=T.device) * k.dx
    y = torch.arange(k.ny, dtype=torch.float64, device=T.device) * k.dy
    sigma = P.SIGMA_SB if k.radiation else 0.0
    peaks = []
    for tick in plan:
        gx = torch.exp(-2.0 * k.inv_r0_sq * (x - float(tick["x_l"])) ** 2)
        gy = torch.exp(-2.0 * k.inv_r0_sq * (y - float(tick["y_l"])) ** 2)
        q = float(tick["q_scale"]) * k.peak_S
        dx, dy = _edge_diffs(T)
        loss = k.hConv * (T - k.Tamb)
        loss += (k.eps * sigma) * ((T * T) ** 2 - (k.Tamb * k.Tamb) ** 2)
        if phys == 0:
            inc = _divergence(dx, dy, k.alpha * k.inv_dx2, k.alpha * k.inv_dy2)
            loss += (k.K / k.dSub) * (T - k.Tsub)
            inc -= loss * (k.inv_h / k.rho_cp)
            inc += torch.outer(gy * (q / (k.rho_cp * k.h)), gx)
            T = T + k.dt * inc
        else:
            kt = _table(T, _KS)
            inc = _divergence(0.5 * (kt[:, 1:] + kt[:, :-1]) * dx,
                              0.5 * (kt[1:] + kt[:-1]) * dy, k.inv_dx2, k.inv_dy2)
            loss += (kt / k.dSub) * (T - k.Tsub)
            inc += (torch.outer(gy * q, gx) - loss) * k.inv_h
            cp = _table(T, _CS) + ((T >= 1533.0) & (T <= 1609.0)).double() * (210.0e3 / 76.0)
            T = T + k.dt * inc / (k.rho * cp)
        if bc == 1:
            T[0], T[-1] = T_edge, T_edge
            T[:, 0], T[:, -1] = T_edge, T_edge
        peaks.append(T.max())
    return T, torch.stack(peaks)


def _gelu(x):
    return 0.5 * x * (1.0 + torch.tanh(math.sqrt(2.0 / math.pi) * (x + 0.044715 * x ** 3)))


def _exact_net(params, x):
    """x: f64 [B, H, W, 4] -> [B, H, W]; params: [(w [co, ci, 3, 3], b)] in f64."""
    h = x.permute(0, 3, 1, 2)
    for i, (w, b) in enumerate(params):
        h = torch.nn.functional.conv2d(h, w, b, padding=1)
        if i < 4:
            h = _gelu(h)
    return h[:, 0]


def _exact_params(seed, grad=False):
    out = []
    for w, b in _net_params(seed):
        w = torch.tensor(np.asarray(w, np.float32), device=DEVICE).double()
        b = torch.tensor(np.asarray(b, np.float32), device=DEVICE).double()
        w = w.reshape(w.shape[0], 3, 3, w.shape[2]).permute(0, 3, 1, 2).contiguous()
        out.append((w.requires_grad_(grad), b.requires_grad_(grad)))
    return out


def _exact_features(T, k, plan):
    x = torch.arange(k.nx, dtype=torch.float64, device=T.device) * k.dx
    y = torch.arange(k.ny, dtype=torch.float64, device=T.device) * k.dy
    S = torch.zeros_like(T)
    for t in plan[:SG.STEPS]:
        c = k.dt * float(t["q_scale"]) * k.peak_S / (k.rho_cp * k.h)
        S += torch.outer(c * torch.exp(-2.0 * k.inv_r0_sq * (y - float(t["y_l"])) ** 2),
                         torch.exp(-2.0 * k.inv_r0_sq * (x - float(t["x_l"])) ** 2))
    m = plan[SG.STEPS // 2]
    fx = ((x - float(m["x_l"])) / SG.POS_SCALE).clamp(-8.0, 8.0).expand_as(T)
    fy = ((y - float(m["y_l"])) / SG.POS_SCALE).clamp(-8.0, 8.0)[:, None].expand_as(T)
    return torch.stack([(T - k.Tamb) / SG.T_SCALE, S / SG.S_SCALE, fx, fy], -1)


def exact(case, seed):
    kind = case["kind"]
    with torch.no_grad():
        if kind == "map":
            sides, peaks = {}, []
            for s in _map_scenarios(case, seed):
                T = torch.full((s.k.ny, s.k.nx), s.k.Tamb, dtype=torch.float64, device=DEVICE)
                T, pk = _exact_run(s.k, s.plan, T, 0, 0.0)
                sides.setdefault(s.k.nx, []).append(T)
                peaks.append(pk)
            return {"fields": {str(n): torch.stack(f) for n, f in sides.items()},
                    "rings": {"tmax": torch.cat(peaks), "arg": None, "rows": None}}
        if kind == "superstep":
            k, plan, _, _, past = _problem(case, seed)
            T = _heated(k, *past)
            ps = _exact_params(seed)
            f = _exact_features(T, k, plan)
            y = torch.empty_like(T)
            for a in range(0, k.ny, 256):              # row blocks with the network's reach
                lo, hi = max(0, a - 5), min(k.ny, a + 256 + 5)
                part = _exact_rows(ps, f, lo, hi, k.ny)
                y[a:min(k.ny, a + 256)] = part[a - lo:min(k.ny, a + 256) - lo]
            return {"y": y[None], "T": T + y * SG.DT_SCALE}
        if kind != "gradients":
            k, plan, _, _, past = _problem(case, seed)
            uniform = kind in ("f32", "f32k", "wrappers")
            if uniform:
                T = torch.full((k.ny, k.nx), 300.0 if kind == "wrappers" else k.Tamb,
                               dtype=torch.float64, device=DEVICE)
            else:
                T = _heated(k, *past)
            T, pk = _exact_run(k, plan, T, case.get("bc", 0), k.Tamb, 1 if kind == "ext" else 0)
            if kind == "wrappers":
                return {"field": T, "tmax": pk, "arg": None, "ymin": None, "ymax": None}
            if kind == "f32k":
                T = T.reshape(-1)
                return {"field": {"hi": T, "lo": None}, "ring": {"tmax": pk, "arg": None,
                                                                 "rows": None}}
            return {"field": T, "ring": {"tmax": pk, "arg": None, "rows": None}}
    x4, tgt = _patches(case, seed)
    ps = _exact_params(seed, grad=True)
    n = tgt.numel()
    loss = torch.zeros((), dtype=torch.float64, device=DEVICE)
    for i in range(0, case["batch"], 4):
        y = _exact_net(ps, x4[i:i + 4].double())
        part = ((y - tgt[i:i + 4].double()) ** 2).sum() / n
        part.backward()
        loss += part.detach()
    grads = torch.cat([torch.cat([w.grad.permute(0, 2, 3, 1).reshape(-1), b.grad])
                       for w, b in ps])
    return {"loss": loss.reshape(1), "grads": grads}


def _exact_rows(ps, f, lo, hi, ny):
    """The network on rows [lo, hi) of the features; rows cut off there are
    five layers away from the ones kept, the field's own edges are exact."""
    return _exact_net(ps, f[None, lo:hi])[0]
