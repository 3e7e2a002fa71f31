"""Performance cases: what users of the library have it compute, through its
public entry points, from a few dozen sections to the largest single instance
and from one instance to thousands of cells.

A case names a `kind`:
  rhs         one right-hand side, aggregation + breakage (the drop-in calls)
  breakage    one breakage right-hand side alone (milling without aggregation)
  vjp         the vector-Jacobian products of both terms
  tape        checkpointed RK4 of one instance, forward and backward
  batch_rk4   RK4 steps of many cells, mixed section counts and grids
  batch_mesh  one RK4 step of many small cells held as mesh fields
  batch_tape  checkpointed RK4 of many cells, forward and backward
  batch_ros2  linearly implicit steps of many cells
and its sizes. Grids are x_i = x_0 2^(i/q) (q sections an octave), or, with
q = 0, irregular. `seed` moves the distributions and coefficients.
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                                "pbe-fixed-pivot-cuda_gb300"))
import pbe_gb300 as pg  # noqa: E402

X0 = 1e-21
F64 = torch.float64


def listed():
    return [
        # the calls an integrator of a small model makes thousands of times: latency and launches
        {"name": "rhs_n64", "kind": "rhs", "n": 64, "q": 4, "kernel": 5, "selection": 3,
         "daughter": "symmetric", "points": 1},
        # the flocculation example's section count: shear flocs with a power-law breakage rate
        {"name": "rhs_n960", "kind": "rhs", "n": 960, "q": 32, "kernel": 5, "selection": 2,
         "daughter": "uniform", "points": 8},
        # the headline instance: the finest grid in use, threshold breakage with 16 table entries
        {"name": "rhs_n16384", "kind": "rhs", "n": 16384, "q": 512, "kernel": 5, "selection": 3,
         "daughter": "split", "points": 16},
        # sections placed by hand (irregular), an odd count, the sum kernel, erosion
        {"name": "rhs_irregular_n2049", "kind": "rhs", "n": 2049, "q": 0, "kernel": 1, "selection": 1,
         "daughter": "erosion", "points": 2},
        # milling: breakage alone on a fine grid with a power-law daughter
        {"name": "breakage_n8191", "kind": "breakage", "n": 8191, "q": 256, "selection": 2,
         "daughter": "powerlaw", "points": 16},
        # sensitivities of the headline instance: one reverse-mode call of each term
        {"name": "vjp_n16384", "kind": "vjp", "n": 16384, "q": 512, "kernel": 5, "selection": 3,
         "daughter": "split", "points": 16},
        # parameter fitting on the two-stage flocculation run: a checkpointed stretch of RK4 and its adjoint
        {"name": "tape_n3840", "kind": "tape", "n": 3840, "q": 128, "steps": 10, "every": 5,
         "daughter": "powerlaw", "points": 8},
        # a flow solver's compartments: uneven section counts on shared grids, explicit steps
        {"name": "batch_rk4_256", "kind": "batch_rk4", "cells": 256, "n_max": 3840, "steps": 2},
        # a flow solver's mesh: thousands of cells of a few dozen sections, mesh fields in and out
        {"name": "batch_mesh_4096", "kind": "batch_mesh", "cells": 4096, "n": 48, "q": 4, "kernel": 3},
        # fitting many experiments at once: batched RK4 and its adjoint
        {"name": "batch_tape_48", "kind": "batch_tape", "cells": 48, "n_max": 2048, "steps": 4, "every": 2},
        # stiff cells: implicit steps, Jacobian-vector products inside GMRES
        {"name": "batch_ros2_64", "kind": "batch_ros2", "cells": 64, "n_max": 512, "steps": 1, "krylov": 8},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["rhs", "rhs", "rhs", "breakage", "vjp", "vjp", "tape", "batch_rk4", "batch_mesh",
                       "batch_tape", "batch_ros2"])
    daughter, points = rng.choice([("symmetric", 1), ("erosion", 2), ("uniform", 4), ("uniform", 8),
                                   ("powerlaw", 8), ("powerlaw", 16), ("split", 16)])
    if kind in ("rhs", "breakage", "vjp"):
        n = _log_int(rng, 48, 16384)
        # 20 to 40 octaves, as the listed grids span, or an irregular grid of at most 4096 sections
        q = max(2, int(round(n / rng.uniform(20.0, 40.0))))
        if n <= 4096 and rng.random() < 0.25:
            q = 0
        case = {"kind": kind, "n": n, "q": q, "selection": rng.randrange(4), "daughter": daughter, "points": points}
        if kind != "breakage":
            case["kernel"] = rng.randrange(6)
        return case
    if kind == "tape":
        n = _log_int(rng, 128, 3840)
        return {"kind": kind, "n": n, "q": max(4, n // 30), "steps": rng.randint(4, 10), "every": rng.randint(2, 5),
                "daughter": daughter, "points": points}
    if kind == "batch_rk4":
        return {"kind": kind, "cells": _log_int(rng, 1, 256), "n_max": 64 * rng.randint(4, 60), "steps": rng.randint(1, 2)}
    if kind == "batch_mesh":
        return {"kind": kind, "cells": _log_int(rng, 256, 4096), "n": rng.randint(24, 72), "q": rng.choice([3, 4, 5]),
                "kernel": rng.randrange(6)}
    if kind == "batch_tape":
        return {"kind": kind, "cells": _log_int(rng, 2, 48), "n_max": rng.randint(512, 2048), "steps": rng.randint(2, 4),
                "every": rng.randint(1, 3)}
    return {"kind": kind, "cells": _log_int(rng, 4, 64), "n_max": rng.randint(64, 512), "steps": 1, "krylov": rng.randint(4, 8)}


# -- inputs (host arrays from the seed) --------------------------------------------

def _table(case):
    d, p = case["daughter"], case["points"]
    if d == "symmetric":
        return pg.quadrature.symmetric_binary()
    if d == "erosion":
        return pg.quadrature.erosion(0.1)
    if d == "uniform":
        return pg.quadrature.uniform(p)
    if d == "powerlaw":
        return pg.quadrature.power_law(2.0, p // 2)
    return pg.quadrature.symmetric_binary_split(p)


def _pivots(n, q, rng):
    if q:
        return pg.grids.geometric_pow2(n, X0, float(q))
    steps = rng.uniform(0.2, 1.8, size=n) * (24.0 * math.log(2.0) / n)
    return X0 * np.exp(np.cumsum(steps))


def _lognormal(x, where, total, rng):
    """A lognormal population (sigma 1) around the pivot at `where` of the grid, moved and scaled a little by the
    seed, and empty beyond five sigma."""
    m = min(len(x) - 1, max(0, int(where * len(x))))
    z = np.log(x / x[m]) + rng.uniform(-0.3, 0.3)
    N = np.where(np.abs(z) <= 5.0, np.exp(-0.5 * z * z), 0.0)
    return N * (total * rng.uniform(0.5, 1.5) / N.sum())


_AGG = {0: dict(beta0=1e-15), 1: dict(beta0=1e4), 2: dict(beta0=1e24), 3: dict(beta_br=6.73e-18),
        4: dict(beta_sh=66.0), 5: dict(beta_br=6.73e-18, beta_sh=66.0)}


def _agg(kernel, rng):
    c = dict(beta0=0.0, beta_br=0.0, beta_sh=0.0)
    c.update(_AGG[kernel])
    f = rng.uniform(0.5, 1.5)
    return {k: v * f for k, v in c.items()}


def _host(case, seed):
    """The inputs of a case as numpy arrays and numbers."""
    rng = np.random.default_rng(seed)
    kind = case["kind"]
    if kind in ("rhs", "breakage", "vjp"):
        n = case["n"]
        x = _pivots(n, case["q"], rng)
        # the headline distribution is not cut: its tail falls below 1e-60 of the peak
        if n > 8192:
            N = pg.grids.lognormal_ic(x, n // 8 + int(rng.integers(-64, 65)), 1.0, 1e14 * rng.uniform(0.5, 1.5))
        else:
            N = _lognormal(x, 0.25, 1e14, rng)
        t, bw = _table(case)
        h = dict(x=x, N=N, t=t, bw=bw, kernel=case.get("kernel", -1),
                 sel=dict(selection=case["selection"], S0=1e-3 * rng.uniform(0.5, 1.5), v_ref=float(x[n // 2]),
                          alpha=float(rng.uniform(0.5, 1.5)), v_min=float(x[n // 2])))
        if "kernel" in case:
            h["agg"] = _agg(case["kernel"], rng)
        if kind == "vjp":
            h["lam"] = (x / x[n // 2]) ** (2.0 / 3.0) + 0.1 * rng.standard_normal(n)
        return h
    if kind == "tape":
        n = case["n"]
        x = _pivots(n, case["q"], rng)
        t, bw = _table(case)
        return dict(x=x, N=_lognormal(x, 1.0 / 6.0, 1e12, rng), t=t, bw=bw, lam=x ** (2.0 / 3.0), dt=0.5,
                    agg=[dict(beta0=0.0, beta_br=6.73e-18, beta_sh=4.0 * G / 3.0 * rng.uniform(0.8, 1.2))
                         for G in (100.0, 20.0)],
                    sel=dict(selection=2, S0=5e-4, v_ref=1e-18, alpha=1.0, v_min=0.0),
                    step_set=[0 if s < case["steps"] // 2 else 1 for s in range(case["steps"])])
    if kind == "batch_mesh":
        C, n = case["cells"], case["n"]
        x = _pivots(n, case["q"], rng)
        z = np.log(x[:, None] / x[n // 4]) + rng.uniform(-1.0, 1.0, size=(1, C))
        N = np.where(np.abs(z) <= 5.0, np.exp(-0.5 * z * z), 0.0)
        N *= 1e13 * rng.uniform(0.5, 1.5, size=(1, C)) / N.sum(axis=0, keepdims=True)
        c = _AGG[case["kernel"]]
        p = pg.batch.cell_params(C, beta0=c.get("beta0", 0.0), beta_br=c.get("beta_br", 0.0),
                                 beta_sh=c.get("beta_sh", 0.0) * np.exp(rng.uniform(-1.0, 1.0, size=C)),
                                 S0=1e-3, v_ref=float(x[n // 2]), alpha=1.0)
        t, bw = pg.quadrature.symmetric_binary()
        return dict(grids=[x], cell_n=np.full(C, n), cell_grid=np.zeros(C, int), params=p, soa=N, t=t, bw=bw,
                    kernel=case["kernel"], selection=2, dt=0.5)
    C = case["cells"]
    if kind == "batch_rk4":
        # sizes and grids are the case's; states and shear rates move with the seed
        cfg = pg.grids.config_batched_cells(C, n_max=case["n_max"])
        cfg["N"] = cfg["N"] * np.repeat(rng.uniform(0.5, 1.5, size=C), cfg["cell_n"])
        cfg["params"][:, 2] *= rng.uniform(0.8, 1.2, size=C)
    elif kind == "batch_tape":
        # sizes do not move with the seed (a fit keeps its experiments' grids); coefficients and states do
        sizes = np.random.default_rng(case["n_max"] * 131 + C)
        cell_n = sizes.integers(min(256, case["n_max"] // 2), case["n_max"] + 1, size=C)
        grids = [_pivots(int(k), 128, rng) for k in (case["n_max"] // 2, case["n_max"])]
        cell_grid = (cell_n > case["n_max"] // 2).astype(int)
        spread = lambda: np.exp(rng.normal(0.0, 0.5, size=C))  # noqa: E731
        p = pg.batch.cell_params(C, beta0=0.0, beta_br=6.73e-18 * spread(), beta_sh=66.0 * spread(), S0=1e-3 * spread(),
                                 v_ref=1e-18, alpha=1.0)
        t, bw = pg.quadrature.uniform(4)
        cfg = dict(grids=grids, cell_n=cell_n, cell_grid=cell_grid, params=p, t_q=t, bw_q=bw,
                   N=np.concatenate([_lognormal(grids[g][:n], 0.25, 1e13, rng) for g, n in zip(cell_grid, cell_n)]))
    else:
        sizes = np.random.default_rng(case["n_max"] * 137 + C)
        cell_n = sizes.integers(max(32, case["n_max"] // 4), case["n_max"] + 1, size=C)
        x = _pivots(case["n_max"], max(2, case["n_max"] // 30), rng)
        p = pg.batch.cell_params(C, beta0=0.0, beta_br=6.73e-18, beta_sh=66.0 * np.exp(rng.uniform(-1, 1, size=C)),
                                 S0=rng.uniform(0.5, 2.0, size=C), v_ref=1e-18, alpha=1.0)
        t, bw = pg.quadrature.uniform(4)
        cfg = dict(grids=[x], cell_n=cell_n, cell_grid=np.zeros(C, int), params=p, t_q=t, bw_q=bw,
                   N=np.concatenate([_lognormal(x[:n], 0.25, 1e13, rng) for n in cell_n]))
    h = dict(grids=cfg["grids"], cell_n=cfg["cell_n"], cell_grid=cfg["cell_grid"], params=cfg["params"], N=cfg["N"],
             t=cfg["t_q"], bw=cfg["bw_q"], kernel=5, selection=2, dt=0.5)
    if kind == "batch_tape":
        h["lam"] = rng.standard_normal(len(cfg["N"])) * 1e-13 + 1e-13
    return h


def _dev(a):
    return torch.tensor(np.ascontiguousarray(a, dtype=np.float64), device="cuda")


def _agg_params(h, c, n):
    p = pg.AggregationParams(n=n, kernel_type=h.get("kernel", 5), **c)
    p.log_x0, p.inv_log_r = pg.grids.geometric_params(h["x"])
    return p


def prepare(case, seed):
    h = _host(case, seed)
    kind = case["kind"]
    s = {"kind": kind}
    if kind in ("rhs", "breakage", "vjp", "tape"):
        n = case["n"]
        s.update(x=_dev(h["x"]), N0=_dev(h["N"]), t=_dev(h["t"]), bw=_dev(h["bw"]))
        bp = pg.BreakageParams(n=n, n_quad=len(h["t"]), **h["sel"])
        if kind == "tape":
            h["kernel"] = 5
            ap = [_agg_params(h, c, n) for c in h["agg"]]
            s.update(N=s["N0"].clone(), lam=_dev(h["lam"]), g=torch.zeros(n, dtype=F64, device="cuda"),
                     ga=torch.zeros((2, 3), dtype=F64, device="cuda"), gb=torch.zeros((2, 4), dtype=F64, device="cuda"),
                     tape=pg.Rk4Tape(case["steps"], h["dt"], case["every"], agg_sets=ap, brk_sets=[bp, bp],
                                     step_set=h["step_set"]))
            return s
        s["bp"] = bp
        if kind != "breakage":
            s["ap"] = _agg_params(h, h["agg"], n)
            if not case["q"]:
                s["ap"].inv_log_r = 0.0
        if kind == "vjp":
            s.update(lam=_dev(h["lam"]), ga=torch.zeros(3, dtype=F64, device="cuda"),
                     gb=torch.zeros(4, dtype=F64, device="cuda"))
        s["out"] = torch.zeros(n, dtype=F64, device="cuda")
        return s
    s["plan"] = pg.BatchPlan(h["grids"], h["cell_n"], h["cell_grid"], h["kernel"], h["selection"], h["t"], h["bw"])
    s["params"], s["dt"] = _dev(h["params"]), h["dt"]
    total = s["plan"].total
    s["N"] = torch.zeros(total, dtype=F64, device="cuda")
    if kind == "batch_mesh":
        s.update(soa=_dev(h["soa"]), out=torch.zeros_like(_dev(h["soa"])), ld=case["cells"])
        return s
    s["N0"] = _dev(h["N"])
    s["steps"] = case["steps"]
    if kind == "batch_tape":
        s.update(lam=_dev(h["lam"]), g=torch.zeros(total, dtype=F64, device="cuda"), every=case["every"],
                 gp=torch.zeros((case["cells"], 8), dtype=F64, device="cuda"))
    if kind == "batch_ros2":
        s.update(krylov=case["krylov"], resid=torch.zeros(case["cells"], dtype=F64, device="cuda"))
    return s


def run(s):
    kind = s["kind"]
    if kind == "rhs":
        s["out"].zero_()
        pg.check(pg.aggregation_rhs(s["N0"], s["x"], s["out"], s["ap"]))
        pg.check(pg.breakage_rhs(s["N0"], s["x"], s["t"], s["bw"], s["out"], s["bp"]))
        return s["out"]
    if kind == "breakage":
        s["out"].zero_()
        pg.check(pg.breakage_rhs(s["N0"], s["x"], s["t"], s["bw"], s["out"], s["bp"]))
        return s["out"]
    if kind == "vjp":
        for k in ("out", "ga", "gb"):
            s[k].zero_()
        pg.check(pg.aggregation_rhs_vjp(s["N0"], s["x"], s["lam"], s["out"], s["ga"], s["ap"]))
        pg.check(pg.breakage_rhs_vjp(s["N0"], s["x"], s["t"], s["bw"], s["lam"], s["out"], s["gb"], s["bp"]))
        return s["out"], s["ga"], s["gb"]
    if kind == "tape":
        s["N"].copy_(s["N0"])
        pg.check(s["tape"].forward(s["N"], s["x"], s["t"], s["bw"]))
        pg.check(s["tape"].backward(s["lam"], s["g"], s["ga"], s["gb"]))
        return s["N"], s["g"], s["ga"], s["gb"]
    plan = s["plan"]
    if kind == "batch_mesh":
        pg.check(plan.from_soa(s["soa"], s["ld"], s["N"]))
        pg.check(plan.rk4(s["N"], s["params"], s["dt"], 1))
        pg.check(plan.to_soa(s["N"], s["out"], s["ld"]))
        return s["out"]
    s["N"].copy_(s["N0"])
    if kind == "batch_rk4":
        pg.check(plan.rk4(s["N"], s["params"], s["dt"], s["steps"]))
        return s["N"]
    if kind == "batch_tape":
        pg.check(plan.tape_forward(s["N"], s["params"], s["dt"], s["steps"], s["every"]))
        pg.check(plan.tape_backward(s["lam"], s["g"], s["gp"]))
        return s["N"], s["g"], s["gp"]
    pg.check(plan.ros2(s["N"], s["params"], s["dt"], s["steps"], s["krylov"], s["resid"]))
    return s["N"]


# -- work ---------------------------------------------------------------------------

def _rhs_flops(n, q, points):
    """Operations one evaluation cannot do without: pairs that share their larger member and their bracket can be
    summed term by term (five separable terms of rate and weighted rate, a multiply-add each), and a section meets
    at most q + 1 brackets, or as many as it has partners; a fragment takes eight operations."""
    return 20.0 * n * min(q + 1, (n + 1) / 2) + 8.0 * n * points


def work(case):
    kind = case["kind"]
    if kind in ("rhs", "breakage", "vjp", "tape"):
        n, points = case["n"], case["points"]
        q = case["q"] or n / 24.0
        f = 8.0 * n * points if kind == "breakage" else _rhs_flops(n, q, points)
        if kind == "vjp":
            return {"bytes": 8.0 * (4 * n + 2 * points), "flops": 2 * f}
        if kind == "tape":
            return {"bytes": 8.0 * 5 * n, "flops": f * 4 * case["steps"] * 4}
        return {"bytes": 8.0 * (3 * n + 2 * points), "flops": f}
    h = _host(case, 0)
    qs = [round(math.log(2.0) / math.log(g[1] / g[0])) for g in h["grids"]]
    f = sum(_rhs_flops(int(n), qs[g], len(h["t"])) for n, g in zip(h["cell_n"], h["cell_grid"]))
    bins = float(np.sum(h["cell_n"]))
    evals = {"batch_mesh": 4, "batch_rk4": 4 * case.get("steps", 1), "batch_tape": 16 * case.get("steps", 1),
             "batch_ros2": (2 + 4 * case.get("krylov", 0)) * case.get("steps", 1)}[kind]
    return {"bytes": 8.0 * bins * (4 if kind == "batch_tape" else 2), "flops": f * evals}


# -- the same in plain torch, 64 bits -----------------------------------------------

def _beta_terms(kernel, c, xj, xk, aj, ak):
    """[(coefficient index, form)] with beta = sum of coefficient * form."""
    if kernel == 0:
        return [(0, torch.ones_like(xj * xk))]
    if kernel == 1:
        return [(0, xj + xk)]
    if kernel == 2:
        return [(0, xj * xk)]
    br = (1, aj / ak + ak / aj + 2.0)
    sh = (2, (aj + ak) ** 3)
    return {3: [br], 4: [sh], 5: [br, sh]}[kernel]


def _pairs(x, kernel, c):
    """Blocks of the pairs j <= k: (rows j, columns k, mask * 1/2 on the diagonal, forms, bracket, weight, clipped)."""
    n = len(x)
    a = x ** (1.0 / 3.0)
    rows = max(1, min(n, (1 << 23) // n))
    for j0 in range(0, n, rows):
        j = torch.arange(j0, min(n, j0 + rows), device=x.device)[:, None]
        k = torch.arange(j0, n, device=x.device)[None, :]
        half = (k > j).to(F64) + 0.5 * (k == j).to(F64)
        xj, xk = x[j], x[k]
        v = xj + xk
        lo = (torch.searchsorted(x, v.reshape(-1), right=True) - 1).reshape(v.shape)
        clip = lo >= n - 1
        lo = lo.clamp(max=n - 2) if n > 1 else lo * 0
        # (x_k - x_lo) + x_j: the two pivots are within a factor of two, so no bit of x_j is lost
        w = ((xk - x[lo]) + xj) / (x[(lo + 1).clamp(max=n - 1)] - x[lo]) if n > 1 else torch.zeros_like(v)
        yield j, k, half, _beta_terms(kernel, c, xj, xk, a[j], a[k]), lo, w, clip


def _exact_agg(N, x, kernel, c):
    n = len(x)
    out = torch.zeros_like(N)
    co = (c["beta0"], c["beta_br"], c["beta_sh"])
    for j, k, half, forms, lo, w, clip in _pairs(x, kernel, co):
        rate = sum(co[i] * f for i, f in forms) * half * N[j] * N[k]
        out.index_add_(0, j[:, 0], -rate.sum(1))
        out.index_add_(0, k[0], -rate.sum(0))
        inner = torch.where(clip, 0.0, rate)
        out.index_add_(0, lo.reshape(-1), ((1.0 - w) * inner).reshape(-1))
        out.index_add_(0, (lo + 1).clamp(max=n - 1).reshape(-1), (w * inner).reshape(-1))
        out[n - 1] += torch.where(clip, rate, 0.0).sum()
    return out


def _exact_agg_vjp(N, x, lam, kernel, c):
    n = len(x)
    g, gp = torch.zeros_like(N), torch.zeros(3, dtype=F64, device=N.device)
    co = (c["beta0"], c["beta_br"], c["beta_sh"])
    for j, k, half, forms, lo, w, clip in _pairs(x, kernel, co):
        hi = lam[(lo + 1).clamp(max=n - 1)]
        G = torch.where(clip, lam[n - 1], lam[lo] + w * (hi - lam[lo])) - lam[j] - lam[k]
        G = G * half
        B = sum(co[i] * f for i, f in forms) * G
        g.index_add_(0, j[:, 0], (B * N[k]).sum(1))
        g.index_add_(0, k[0], (B * N[j]).sum(0))
        for i, f in forms:
            gp[i] += (f * G * N[j] * N[k]).sum()
    return g, gp


def _selection(x, s):
    r = x / s["v_ref"]
    S = {0: torch.ones_like(x), 1: r, 2: r ** s["alpha"], 3: (x > s["v_min"]).to(F64)}[s["selection"]]
    return s["S0"] * S, S


def _fragments(x, t):
    n = len(x)
    v = x[:, None] * t[None, :]
    lo = (torch.searchsorted(x, v.reshape(-1), right=True) - 1).reshape(v.shape)
    low, high = v <= x[0], v >= x[n - 1]
    lo = lo.clamp(0, max(0, n - 2))
    w = (v - x[lo]) / (x[(lo + 1).clamp(max=n - 1)] - x[lo]) if n > 1 else torch.zeros_like(v)
    w = torch.where(low, 0.0, torch.where(high, 1.0, w))
    return torch.where(low, 0, lo), w


def _exact_brk(N, x, t, bw, s):
    S, _ = _selection(x, s)
    lo, w = _fragments(x, t)
    b = (S * N)[:, None] * bw[None, :]
    out = -S * N
    out.index_add_(0, lo.reshape(-1), ((1.0 - w) * b).reshape(-1))
    out.index_add_(0, (lo + 1).clamp(max=len(x) - 1).reshape(-1), (w * b).reshape(-1))
    return out


def _exact_brk_vjp(N, x, t, bw, lam, s):
    S, form = _selection(x, s)
    lo, w = _fragments(x, t)
    hi = lam[(lo + 1).clamp(max=len(x) - 1)]
    Q = (bw[None, :] * (lam[lo] + w * (hi - lam[lo]))).sum(1) - lam
    zero = torch.zeros((), dtype=F64, device=N.device)
    gp = [(form * N * Q).sum(), zero, zero, zero]
    if s["selection"] == 1:
        gp[1] = -(S * N * Q).sum() / s["v_ref"]
    if s["selection"] == 2:
        gp[1] = -(s["alpha"] / s["v_ref"]) * (S * N * Q).sum()
        gp[2] = (S * torch.log(x / s["v_ref"]) * N * Q).sum()
    return torch.where(N > 2.2e-308, S * Q, 0.0), torch.stack(gp)


def _exact_rk4(N, rhs, dt):
    """One step; its four stage states."""
    Y = [N]
    k = [rhs(N)]
    for c in (0.5, 0.5, 1.0):
        Y.append(N + c * dt * k[-1])
        k.append(rhs(Y[-1]))
    return N + dt / 6.0 * (k[0] + 2.0 * k[1] + 2.0 * k[2] + k[3]), Y


def _exact_back(lam, Y, vjp, dt):
    """lambda at the step's start and the parameter gradients of the step."""
    c, h = dt / 6.0, 0.5 * dt
    m4, p4 = vjp(Y[3], c * lam)
    m3, p3 = vjp(Y[2], 2.0 * c * lam + dt * m4)
    m2, p2 = vjp(Y[1], 2.0 * c * lam + h * m3)
    m1, p1 = vjp(Y[0], c * lam + h * m2)
    return lam + m1 + m2 + m3 + m4, p1 + p2 + p3 + p4


def exact(case, seed):
    kind = case["kind"]
    if kind == "batch_ros2":
        return None  # GMRES of a few steps: its value is the method's own
    h = _host(case, seed)
    t, bw = _dev(h["t"]), _dev(h["bw"])
    if kind in ("rhs", "breakage", "vjp"):
        x, N = _dev(h["x"]), _dev(h["N"])
        if kind == "vjp":
            lam = _dev(h["lam"])
            ga, pa = _exact_agg_vjp(N, x, lam, h["kernel"], h["agg"])
            gb, pb = _exact_brk_vjp(N, x, t, bw, lam, h["sel"])
            return ga + gb, pa, pb
        out = _exact_brk(N, x, t, bw, h["sel"])
        return out if kind == "breakage" else out + _exact_agg(N, x, h["kernel"], h["agg"])
    if kind == "tape":
        x, N, lam = _dev(h["x"]), _dev(h["N"]), _dev(h["lam"])

        def rhs(y, m):
            return _exact_agg(y, x, 5, h["agg"][m]) + _exact_brk(y, x, t, bw, h["sel"])

        def vjp(y, a, m):
            g, p = _exact_agg_vjp(y, x, a, 5, h["agg"][m])
            gb, pb = _exact_brk_vjp(y, x, t, bw, a, h["sel"])
            return g + gb, torch.cat([p, pb])

        stages = []
        for m in h["step_set"]:
            N, Y = _exact_rk4(N, lambda y: rhs(y, m), h["dt"])
            stages.append(Y)
        gp = torch.zeros((2, 7), dtype=F64, device="cuda")
        for m, Y in zip(reversed(h["step_set"]), reversed(stages)):
            lam, p = _exact_back(lam, Y, lambda y, a: vjp(y, a, m), h["dt"])
            gp[m] += p
        return N, lam, gp[:, :3].contiguous(), gp[:, 3:].contiguous()
    if kind == "batch_mesh":
        return _exact_mesh(h, t, bw)
    Ns, gs, ps, at = [], [], [], 0
    for c, (n, gi) in enumerate(zip(h["cell_n"], h["cell_grid"])):
        n = int(n)
        x, N = _dev(h["grids"][gi][:n]), _dev(h["N"][at:at + n])
        p = h["params"][c]
        ac = dict(beta0=float(p[0]), beta_br=float(p[1]), beta_sh=float(p[2]))
        sc = dict(selection=h["selection"], S0=float(p[3]), v_ref=float(p[4]), alpha=float(p[5]), v_min=float(p[6]))

        def rhs(y):
            return _exact_agg(y, x, h["kernel"], ac) + _exact_brk(y, x, t, bw, sc)

        def vjp(y, a):
            g, q = _exact_agg_vjp(y, x, a, h["kernel"], ac)
            gb, qb = _exact_brk_vjp(y, x, t, bw, a, sc)
            return g + gb, torch.cat([q, qb, qb.new_zeros(1)])

        stages = []
        for _ in range(case["steps"]):
            N, Y = _exact_rk4(N, rhs, h["dt"])
            stages.append(Y)
        Ns.append(N)
        if kind == "batch_tape":
            lam, gp = _dev(h["lam"][at:at + n]), torch.zeros(8, dtype=F64, device="cuda")
            for Y in reversed(stages):
                lam, q = _exact_back(lam, Y, vjp, h["dt"])
                gp += q
            gs.append(lam)
            ps.append(gp)
        at += n
    if kind == "batch_tape":
        return torch.cat(Ns), torch.cat(gs), torch.stack(ps)
    return torch.cat(Ns)


def _exact_mesh(h, t, bw):
    """All cells share one small grid: the pair and fragment sums as matrices over the cells."""
    x, N, p = _dev(h["grids"][0]), _dev(h["soa"]), _dev(h["params"])
    n = len(x)
    co = [p[:, i] for i in range(3)]
    lo_f, w_f = _fragments(x, t)
    S = (p[:, 3])[None, :] * (x[:, None] / p[:, 4][None, :]) ** p[:, 5][None, :]

    def rhs(y):
        out = torch.zeros_like(y)
        for j, k, half, forms, lo, w, clip in _pairs(x, h["kernel"], None):
            j, k = torch.broadcast_tensors(j, k)
            keep = (half > 0).reshape(-1)
            j, k, lo, w, clip, half = (v.reshape(-1)[keep] for v in (j, k, lo, w, clip, half))
            B = sum(co[i][None, :] * (f.reshape(-1)[keep] * half)[:, None] for i, f in forms)
            rate = B * y[j] * y[k]
            out.index_add_(0, j, -rate)
            out.index_add_(0, k, -rate)
            lw = torch.where(clip, 0.0, 1.0 - w)[:, None]
            hw = torch.where(clip, 1.0, w)[:, None]
            out.index_add_(0, lo, lw * rate)
            out.index_add_(0, torch.where(clip, n - 1, lo + 1), hw * rate)
        for q in range(len(t)):
            b = S * y * bw[q]
            out.index_add_(0, lo_f[:, q], (1.0 - w_f[:, q])[:, None] * b)
            out.index_add_(0, (lo_f[:, q] + 1).clamp(max=n - 1), w_f[:, q][:, None] * b)
        return out - S * y

    return _exact_rk4(N, rhs, h["dt"])[0]
