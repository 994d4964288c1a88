"""Timed cases: the work a user of this package has it do, at the sizes it is used at.

Each case is one call (or one short sequence of calls) of the public entry
points with everything in hand that a user's program keeps between calls:
ensembles packed on the device, the resident library, a running server.

    listed()             the cases
    draw(rng)            one more case of the same kinds, sizes spread over their ranges
    prepare(case, seed)  inputs and handles (another seed: other inputs)
    run(state)           one pass, whole outputs
    work(case)           bytes and operations of one pass
    exact(case, seed)    the outputs in 64-bit torch, where they are computed numbers
"""

from __future__ import annotations

import math

import numpy as np
import torch

from custom_madi_gb300 import _native as N
from custom_madi_gb300 import signal as S
from custom_madi_gb300 import workloads as WL
from custom_madi_gb300.config import SimConfig
from custom_madi_gb300.ensemble import create_ensemble
from custom_madi_gb300.fitters_gpu import bayes_fit_gpu, map_match_fits0_gpu, map_match_gpu, match_device
from custom_madi_gb300.serving import FitRequest, Server, SimRequest
from custom_madi_gb300.walker_gpu import WalkJob, kio_to_pp, pair_layout, simulate_jobs

STEPS = 4600                    # 46 ms at 0.01 ms, the acquisition of the benchmark
SI_STEPS = 128_000              # 128 ms at 0.001 ms, the reference's production grid
SI_COLUMNS = 1245 * 25
OPS_PER_STEP = 289.0            # random numbers, move, trapezoid, three-plane label test


def listed() -> list:
    return [
        # A library build: many (kio, rho, V) entries walked in one launch (the
        # headline workload, with fewer walkers each): the largest case.
        {"name": "walk_batch", "kind": "walk", "entries": 128, "walkers": 25_000, "cells_lo": 27, "cells_hi": 512,
         "precision": 32},
        # One entry asked for by itself, at the plain configuration's size:
        # 10,000 walkers leave the GPU part idle, the step chain's latency counts.
        {"name": "walk_entry", "kind": "entry", "rho": 2.0e5, "V": 4.0, "n_kio": 1, "walkers": 10_000,
         "directions": 24},
        # One ensemble of a production library entry: the SI domain with fatal
        # escape, 128,000 steps, stored Y reduced over the full 31,125-column grid.
        {"name": "walk_si_grid", "kind": "si_entry", "rho": 5.0e4, "V": 14.0, "walkers": 10_000},
        # The fp64 walker (reference arithmetic) used to check an entry.
        {"name": "walk_f64", "kind": "walk", "entries": 1, "walkers": 16_000, "cells_lo": 64,
         "cells_hi": 64, "precision": 64},
        # Column reduction of one production ensemble's stored Y.
        {"name": "reduce_grid", "kind": "reduce", "walkers": 50_000, "n_grid": 129, "all_columns": True},
        # Whole-brain voxel fit against a 20,000-entry library, exhaustive FP32 scan.
        {"name": "match_fp32", "kind": "match", "n_vox": 1_000_000, "n_lib": 20_000, "F": 20, "precision": "fp32",
         "topk": 32, "free_s0": False, "snr": 30.0},
        # The same fit on raw signals (free S0), one slab, a ragged size.
        {"name": "match_fp32_free", "kind": "match", "n_vox": 150_001, "n_lib": 20_000, "F": 20, "precision": "fp32",
         "topk": 32, "free_s0": True, "snr": 30.0},
        # The whole-brain fit on the tensor cores with FP32 rescoring of the top 32.
        {"name": "match_bf16", "kind": "match", "n_vox": 1_000_000, "n_lib": 20_000, "F": 20, "precision": "bf16",
         "topk": 32, "free_s0": False, "snr": 30.0},
        # A region of interest fitted from host arrays against a two-Delta
        # library: the smallest call, where launches and copies count.
        {"name": "match_roi", "kind": "match_host", "n_vox": 3_001, "n_lib": 5_000, "F": 10, "free_s0": False,
         "snr": 30.0},
        # Bayesian posterior means of a slab of voxels.
        {"name": "bayes_fit", "kind": "bayes", "n_vox": 100_000, "n_lib": 20_000, "F": 20, "free_s0": False,
         "sigma_m": 0.02, "snr": 30.0},
        # Labels of 200,000 points of an SI population (the v_i measurement of
        # every ensemble build).
        {"name": "classify_points", "kind": "classify", "rho": 5.0e4, "V": 14.0, "points": 200_000, "method": "grid"},
        # The serving loop with simulations and fits waiting at t = 0.
        {"name": "serve_mixed", "kind": "serve", "sims": 24, "walkers_lo": 10_000, "walkers_hi": 100_000, "fits": 3,
         "n_vox": 100_000, "n_lib": 20_000},
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def _ilog(rng, lo, hi):
    return int(min(hi, max(lo, round(_log(rng, lo, hi)))))


def draw(rng) -> dict:
    kind = rng.choice(["walk", "walk", "entry", "si_entry", "f64", "reduce", "match", "match", "match", "match_host",
                       "bayes", "bayes", "classify", "serve"])
    if kind == "walk":
        entries = _ilog(rng, 2, 128)
        lo = rng.randint(27, 256)
        return {"kind": "walk", "entries": entries, "walkers": _ilog(rng, 1_000, 3_200_000 // entries if entries > 32
                                                                     else 100_000),
                "cells_lo": lo, "cells_hi": rng.randint(lo, 1024), "precision": 32}
    if kind == "f64":
        nc = rng.randint(27, 512)
        return {"kind": "walk", "entries": 1, "walkers": _ilog(rng, 500, 8_000), "cells_lo": nc,
                "cells_hi": nc, "precision": 64}
    if kind == "entry":
        rho = _log(rng, 2.0e4, 2.0e7)
        return {"kind": "entry", "rho": rho, "V": rng.uniform(0.55, 0.95) / (rho * 1e-6),
                "n_kio": rng.randint(1, 4),
                "walkers": _ilog(rng, 200, 50_000), "directions": rng.choice([0, 6, 24, 32])}
    if kind == "si_entry":
        rho = _log(rng, 1.0e4, 1.0e5)
        return {"kind": "si_entry", "rho": rho, "V": rng.uniform(0.55, 0.9) / (rho * 1e-6),
                "walkers": _ilog(rng, 500, 12_000)}
    if kind == "reduce":
        full = rng.random() < 0.5
        return {"kind": "reduce", "walkers": _ilog(rng, 500, 50_000), "n_grid": 129, "all_columns": full}
    if kind == "match":
        prec = rng.choice(["fp32", "fp32", "bf16"])
        n_lib = _ilog(rng, 500, 40_000)
        return {"kind": "match", "n_vox": _ilog(rng, 2_000, 500_000), "n_lib": n_lib, "F": rng.choice([5, 10, 15, 20, 28]),
                "precision": prec, "topk": rng.choice([8, 16, 32]), "free_s0": rng.random() < 0.4,
                "snr": _log(rng, 15.0, 80.0)}
    if kind == "match_host":
        return {"kind": "match_host", "n_vox": _ilog(rng, 50, 50_000), "n_lib": _ilog(rng, 200, 20_000),
                "F": rng.choice([5, 10, 15, 20]), "free_s0": rng.random() < 0.5, "snr": _log(rng, 15.0, 80.0)}
    if kind == "bayes":
        return {"kind": "bayes", "n_vox": _ilog(rng, 500, 100_000), "n_lib": _ilog(rng, 500, 20_000),
                "F": rng.choice([5, 10, 15, 20]), "free_s0": rng.random() < 0.5, "sigma_m": _log(rng, 0.01, 0.05),
                "snr": _log(rng, 15.0, 80.0)}
    if kind == "classify":
        rho = _log(rng, 1.0e4, 1.0e5)
        return {"kind": "classify", "rho": rho, "V": rng.uniform(0.55, 0.9) / (rho * 1e-6),
                "points": _ilog(rng, 1_000, 200_000), "method": rng.choice(["grid", "kd"])}
    return {"kind": "serve", "sims": rng.randint(4, 24), "walkers_lo": 5_000, "walkers_hi": _ilog(rng, 20_000, 100_000),
            "fits": rng.randint(1, 4), "n_vox": _ilog(rng, 10_000, 100_000), "n_lib": _ilog(rng, 2_000, 20_000)}


# ---------------------------------------------------------------------------
# Inputs
# ---------------------------------------------------------------------------

def _pgse(n_walkers: int, directions: int = 24) -> SimConfig:
    return WL.plain_config(n_walkers=n_walkers, directions=directions)


def _kios(n: int) -> list:
    """n exchange rates [1/s] of the library's range."""
    return [20.0, 5.0, 60.0, 1.5][:n]


def _columns(cfg: SimConfig):
    c = S.build_columns(cfg)
    return c.j_delta, c.j_Delta, c.j_sum, c.phase_coef


def _walk_jobs(case, cfg, seed):
    """(kio, rho, V, cells) of the batched-build ranges; the geometry and the walk change with the seed."""
    trip = WL.batch_triplets(case["entries"], seed=1, cells=(case["cells_lo"], case["cells_hi"]))
    ens = WL.build_ensembles(trip, cfg, seed=1000 * seed, measure_vi=False)
    for e in ens:
        e.device()
    return [WalkJob(e, kio_to_pp(t[0], e.mean_AV, cfg), 17 + seed, int(case["walkers"])) for e, t in zip(ens, trip)]


def _decays(n_lib: int, F: int, gen) -> torch.Tensor:
    """Bi-exponential decays with exchange-like Delta dependence over F (Delta, b) columns, 1 at b = 0 (fp64)."""
    b = torch.tensor([0.0, 1.0, 2.5, 4.0, 6.0], dtype=torch.float64, device="cuda")
    n_delta = (F + 4) // 5
    deltas = torch.tensor([15.0, 25.0, 30.0, 40.0, 50.0, 60.0][:n_delta], dtype=torch.float64, device="cuda")

    def u(lo, hi):
        return lo + (hi - lo) * torch.rand((n_lib, 1, 1), generator=gen, dtype=torch.float64, device="cuda")
    f, d_in, d_ex, tau = u(0.3, 0.95), u(0.1, 1.2), u(1.0, 3.0), u(20.0, 400.0)
    x = torch.exp(-deltas[None, :, None] / tau)
    slow, fast = torch.exp(-b * d_in), torch.exp(-b * d_ex)
    s = f * (x * slow + (1.0 - x) * fast) + (1.0 - f) * fast
    return s.reshape(n_lib, -1)[:, :F].contiguous()


def _voxels(lib: torch.Tensor, n_vox: int, snr: float, free_s0: bool, gen) -> torch.Tensor:
    """Rician-noised library entries; free S0: scaled to raw scanner units."""
    pick = torch.randint(0, lib.shape[0], (n_vox,), generator=gen, device="cuda")
    s = lib[pick]
    n1 = torch.randn(s.shape, generator=gen, dtype=torch.float64, device="cuda") / snr
    n2 = torch.randn(s.shape, generator=gen, dtype=torch.float64, device="cuda") / snr
    v = torch.sqrt((s + n1) ** 2 + n2 ** 2)
    if free_s0:
        v = v * (200.0 + 1300.0 * torch.rand((n_vox, 1), generator=gen, dtype=torch.float64, device="cuda"))
    return v


def _fit_inputs(case, seed):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(7919 * seed + 11)
    lib = _decays(case["n_lib"], case.get("F", 20), gen)
    vox = _voxels(lib, case["n_vox"], case.get("snr", 30.0), case.get("free_s0", False), gen)
    return vox.float(), lib.float(), gen


def _params(n_lib: int, gen):
    r = torch.rand((n_lib, 3), generator=gen, dtype=torch.float64, device="cuda").cpu().numpy()
    lo, hi = np.log([1.0, 4.4e3, 0.01]), np.log([130.0, 5.8e7, 206.0])
    return np.exp(lo + (hi - lo) * r)


def _reduce_columns(case):
    """The production grid's (delta, Delta) x b columns, or the 200-column uncertainty subset."""
    cfg = SimConfig()
    if case["all_columns"]:
        return _columns(cfg)
    sub = [(5.0, 15.0), (7.0, 25.0), (10.0, 30.0), (12.0, 36.0), (15.0, 40.0), (20.0, 50.0), (25.0, 60.0), (30.0, 80.0)]
    c = S.build_columns(cfg, delta_pairs=sub)
    return c.j_delta, c.j_Delta, c.j_sum, c.phase_coef


def _stored_Y(case, seed) -> torch.Tensor:
    """Y(t) = int (x - L/2) dt of restricted walks: reflected displacements about a uniform start (um ms)."""
    gen = torch.Generator(device="cuda")
    gen.manual_seed(104_729 * seed + 3)
    n, g = case["walkers"], case["n_grid"]
    x0 = 220.0 * (torch.rand((n, 1, 3), generator=gen, dtype=torch.float64, device="cuda") - 0.5)
    step = math.sqrt(2.0 * 3.0) * torch.randn((n, g, 3), generator=gen, dtype=torch.float64, device="cuda")
    d = torch.cumsum(step, dim=1)
    w = 12.0                                            # reflecting cell width, um
    d = torch.abs(torch.remainder(d, 2.0 * w) - w) - 0.5 * w
    Y = torch.cumsum(x0 + d, dim=1)
    Y[:, 0] = 0.0
    return Y.contiguous()


def prepare(case: dict, seed: int) -> dict:
    kind = case["kind"]
    st = {"case": case}
    if kind == "walk":
        cfg = _pgse(case["walkers"], 24 if case["precision"] == 32 else 0)
        st.update(cfg=cfg, jobs=_walk_jobs(case, cfg, seed), columns=_columns(cfg))
    elif kind == "entry":
        cfg = _pgse(case["walkers"], case["directions"])
        e = create_ensemble(case["rho"], case["V"], cfg, seed=1000 + seed, verify_vi=False, measure_vi=False)
        e.device()
        st.update(cfg=cfg, ens=e, columns=S.build_columns(cfg), seed=17 + seed)
    elif kind == "si_entry":
        cfg = SimConfig(n_walkers=case["walkers"], n_ensembles=1)
        e = create_ensemble(case["rho"], case["V"], cfg, seed=1000 + seed, verify_vi=False, measure_vi=False)
        e.device()
        st.update(cfg=cfg, ens=e, columns=S.build_columns(cfg), seed=17 + seed)
    elif kind == "reduce":
        jd, jD, js, pc = _reduce_columns(case)
        st.update(Y=_stored_Y(case, seed), coef=torch.from_numpy(np.asarray(pc, np.float64)).cuda(),
                  **{k: torch.from_numpy(np.asarray(a, np.int32)).cuda() for k, a in (("jd", jd), ("jD", jD), ("js", js))})
    elif kind == "match":
        vox, lib, _ = _fit_inputs(case, seed)
        st.update(vox=vox, lib=lib)
    elif kind == "match_host":
        vox, lib, gen = _fit_inputs(case, seed)
        st.update(vox=vox.double().cpu().numpy(), lib=lib.double().cpu().numpy(), par=_params(case["n_lib"], gen))
    elif kind == "bayes":
        vox, lib, gen = _fit_inputs(case, seed)
        par = _params(case["n_lib"], gen)
        q = 0.2 + torch.rand(case["n_lib"], generator=gen, dtype=torch.float64, device="cuda").cpu().numpy()
        st.update(vox=vox.double().cpu().numpy(), lib=lib.double().cpu().numpy(), par=par, q=q)
    elif kind == "classify":
        cfg = SimConfig()
        e = create_ensemble(case["rho"], case["V"], cfg, seed=1000 + seed, verify_vi=False, measure_vi=False)
        e.device()
        st.update(ens=e, pts=np.random.default_rng(seed).uniform(0.0, e.L, size=(case["points"], 3)))
    elif kind == "serve":
        cfg = WL.batch_config()
        trip = WL.batch_triplets(case["sims"], seed=2)
        ens = WL.build_ensembles(trip, cfg, seed=1000 * seed, measure_vi=False)
        vox, lib, _ = _fit_inputs(case, seed)
        rng = np.random.default_rng(5)
        n = np.exp(rng.uniform(math.log(case["walkers_lo"]), math.log(case["walkers_hi"]), case["sims"])).astype(int)
        reqs = [SimRequest(e, kio_to_pp(t[0], e.mean_AV, cfg), 100 + seed, int(k)) for e, t, k in zip(ens, trip, n)]
        v = vox.cpu().numpy()
        for i in range(case["fits"]):
            reqs.insert((i + 1) * len(reqs) // (case["fits"] + 1),
                        FitRequest(v[: len(v) // (i + 1)], "fp32" if i % 3 == 2 else "bf16", 32))
        lay = pair_layout(*_columns(cfg))
        for e in ens:
            e.device()
        st.update(server=Server(cfg, lay, cfg.direction_array(), library=lib, n_slots=32), requests=reqs)
    else:
        raise ValueError(f"unknown kind {kind!r}")
    return st


# ---------------------------------------------------------------------------
# One pass
# ---------------------------------------------------------------------------

def run(state: dict):
    case = state["case"]
    kind = case["kind"]
    if kind == "walk":
        res = simulate_jobs(state["jobs"], state["cfg"], state["columns"], precision=case["precision"])
        return {k: np.stack([r[k] for r in res]) for k in ("cos", "sin", "occupancy")}
    if kind in ("entry", "si_entry"):
        out = S.compute_signals_multi_kio(case["rho"], case["V"], _kios(case.get("n_kio", 1)), state["cfg"],
                                          state["columns"], seed=state["seed"], verbose=False, ensembles=[state["ens"]])
        keep = ("S", "S_imag", "S_dir", "S_dir_imag", "ensemble_S", "occupancy_fraction")
        return [{k: r[k] for k in keep if k in r} for r in out.values()]
    if kind == "reduce":
        cs = torch.empty_like(state["coef"])
        sn = torch.empty_like(state["coef"])
        N.reduce_Y(state["Y"], case["walkers"], case["n_grid"], state["jd"], state["jD"], state["js"], state["coef"],
                   cs, sn, torch.cuda.current_stream())
        return cs, sn
    if kind == "match":
        idx, res, s0 = match_device(state["vox"], state["lib"], free_s0=case["free_s0"], precision=case["precision"],
                                    topk=case["topk"])
        return (idx, res, s0) if case["free_s0"] else (idx, res)
    if kind == "match_host":
        fit = map_match_fits0_gpu if case["free_s0"] else map_match_gpu
        par = state["par"]
        return fit(state["vox"], state["lib"], par[:, 0], par[:, 1], par[:, 2])
    if kind == "bayes":
        par = state["par"]
        return bayes_fit_gpu(state["vox"], state["lib"], par[:, 0], par[:, 1], par[:, 2], case["sigma_m"],
                             case["free_s0"], state["q"])
    if kind == "classify":
        return state["ens"].classify(state["pts"], method=case["method"])
    out = state["server"].run(state["requests"])
    recs = sorted(out["records"], key=lambda r: r.rid)
    sims = [r.result for r in recs if r.kind == "sim"]
    fits = [r.result for r in recs if r.kind == "fit"]
    return {**{k: np.stack([r[k] for r in sims]) for k in ("cos", "sin", "occupancy")},
            **{k: [r[k] for r in fits] for k in ("best_idx", "best_resid")}}


# ---------------------------------------------------------------------------
# Work of one pass
# ---------------------------------------------------------------------------

def _geometry_bytes(cells: float) -> float:
    """Seeds, facets (15.5 a cell, plane + neighbour) and the fp64 seeds of one geometry."""
    return cells * (16.0 + 15.5 * 20.0 + 32.0)


def _match_work(n_vox, n_lib, F, outs):
    return 4.0 * F * (n_vox + n_lib) + 4.0 * outs * n_vox, 2.0 * F * n_vox * n_lib


def work(case: dict) -> dict:
    kind = case["kind"]
    if kind == "walk":
        cells = 0.5 * (case["cells_lo"] + case["cells_hi"])
        cols = 20 * (24 if case["precision"] == 32 else 1)
        return {"bytes": case["entries"] * (_geometry_bytes(cells) + 16.0 * cols + 8.0 * 47),
                "flops": OPS_PER_STEP * case["entries"] * case["walkers"] * STEPS}
    if kind == "entry":
        return {"bytes": _geometry_bytes(64) + case["n_kio"] * (16.0 * 20 * max(3, case["directions"]) + 8.0 * 47),
                "flops": OPS_PER_STEP * case["n_kio"] * case["walkers"] * STEPS}
    if kind == "si_entry":
        cells = case["rho"] * 1e-9 * 520.0 ** 3
        return {"bytes": _geometry_bytes(cells) + 16.0 * SI_COLUMNS + 8.0 * 129,
                "flops": case["walkers"] * (OPS_PER_STEP * SI_STEPS + 30.0 * 3 * SI_COLUMNS)}
    if kind == "reduce":
        cols = SI_COLUMNS if case["all_columns"] else 200
        return {"bytes": 24.0 * case["walkers"] * case["n_grid"] + cols * (20.0 + 16.0),
                "flops": 30.0 * 3 * cols * case["walkers"]}
    if kind in ("match", "match_host", "bayes"):
        outs = {"match": 3 if case.get("free_s0") else 2, "match_host": 9, "bayes": 18}[kind]
        b, f = _match_work(case["n_vox"], case["n_lib"], case["F"], outs)
        return {"bytes": b, "flops": f}
    if kind == "classify":
        return {"bytes": (24.0 + 5.0) * case["points"] + _geometry_bytes(case["rho"] * 1e-9 * 520.0 ** 3),
                "flops": 500.0 * case["points"]}
    mid = (case["walkers_hi"] - case["walkers_lo"]) / math.log(case["walkers_hi"] / case["walkers_lo"])
    b, f = _match_work(sum(case["n_vox"] // (i + 1) for i in range(case["fits"])), case["n_lib"], 20, 2)
    return {"bytes": b + case["sims"] * (_geometry_bytes(270) + 16.0 * 480 + 8.0 * 47),
            "flops": f + OPS_PER_STEP * case["sims"] * mid * STEPS}


# ---------------------------------------------------------------------------
# The same outputs in 64 bits
# ---------------------------------------------------------------------------

def _exact_reduce(case, seed):
    jd, jD, js, pc = (torch.from_numpy(np.asarray(a)).cuda() for a in _reduce_columns(case))
    Y = _stored_Y(case, seed)
    key = torch.stack([jd, jD, js], 1).long()
    pairs, inv = torch.unique(key, dim=0, return_inverse=True)
    cs, sn = torch.zeros_like(pc), torch.zeros_like(pc)
    order = torch.argsort(inv)
    counts = torch.bincount(inv)
    beg = 0
    for p, c in enumerate(counts.tolist()):
        cols = order[beg:beg + c]
        beg += c
        a, b, s = pairs[p].tolist()
        dm = (Y[:, a] + Y[:, b] - Y[:, s]).reshape(-1)
        ph = pc[cols][:, None] * dm[None, :]
        cs[cols] = torch.cos(ph).sum(1)
        sn[cols] = torch.sin(ph).sum(1)
    return cs, sn


def _pair_blocks(m: torch.Tensor, rows: int = 8192):
    for i in range(0, m.shape[0], rows):
        yield i, m[i:i + rows]


def _exact_match(vox, lib, free_s0):
    """Residual (and S0) of the best entry per voxel; the index itself is a whole number."""
    m, L = vox.double(), lib.double()
    res = torch.empty(m.shape[0], dtype=torch.float64, device=m.device)
    s0 = torch.empty_like(res)
    idx = torch.empty(m.shape[0], dtype=torch.int64, device=m.device)
    ll = (L * L).sum(1)
    for i, x in _pair_blocks(m):
        dot = x @ L.T
        if free_s0:
            score = torch.where(dot > 0, -(dot * dot) / ll, torch.full_like(dot, math.inf))
        else:
            score = ll - 2.0 * dot
        j = torch.argmin(score, 1)
        r = L[j]
        k = (x * r).sum(1) / (r * r).sum(1) if free_s0 else torch.ones(len(x), dtype=torch.float64, device=m.device)
        idx[i:i + len(x)], s0[i:i + len(x)] = j, k
        res[i:i + len(x)] = ((x - k[:, None] * r) ** 2).sum(1)
    return idx, res, s0


def _exact_bayes(case, seed):
    vox, lib, gen = _fit_inputs(case, seed)
    par = torch.from_numpy(_params(case["n_lib"], gen)).cuda()
    q = 0.2 + torch.rand(case["n_lib"], generator=gen, dtype=torch.float64, device="cuda")
    m, L = vox.double(), lib.double()
    ll = (L * L).sum(1)
    inv = 1.0 / (2.0 * case["sigma_m"] ** 2)
    centre = par.mean(0)
    P = par - centre
    names = ("kio_mean", "rho_mean", "V_mean", "kio_std", "rho_std", "V_std", "residual", "n_eff", "s0_fit")
    out = {k: torch.empty(len(m), dtype=torch.float64, device=m.device) for k in names}
    for i, x in _pair_blocks(m, 4096):
        sl = slice(i, i + len(x))
        dot, mm = x @ L.T, (x * x).sum(1, keepdim=True)
        if case["free_s0"]:
            s0 = dot / ll
            resid = (mm - 2.0 * s0 * dot + s0 * s0 * ll).clamp_min(0.0)
            rw = torch.where(dot > 0, resid / (s0 * s0), torch.full_like(dot, math.inf))
        else:
            s0 = torch.ones_like(dot)
            resid = (mm + ll - 2.0 * dot).clamp_min(0.0)
            rw = resid
        e = torch.log(q) - rw * inv
        w = torch.exp(e - e.max(1, keepdim=True).values)
        W = w.sum(1)
        for k, name in enumerate(("kio", "rho", "V")):
            mean = (w @ P[:, k]) / W
            second = (w * (P[None, :, k] - mean[:, None]) ** 2).sum(1) / W
            out[name + "_mean"][sl] = mean + centre[k]
            out[name + "_std"][sl] = second.clamp_min(0.0).sqrt()
        out["residual"][sl] = (w * torch.where(w > 0, resid, torch.zeros_like(resid))).sum(1) / W
        out["n_eff"][sl] = W * W / (w * w).sum(1)
        out["s0_fit"][sl] = (w * torch.where(w > 0, s0, torch.zeros_like(s0))).sum(1) / W
    if not case["free_s0"]:
        del out["s0_fit"]
    return {k: v.cpu().numpy() for k, v in out.items()}


def exact(case: dict, seed: int):
    kind = case["kind"]
    if kind == "reduce":
        return _exact_reduce(case, seed)
    if kind == "match":
        vox, lib, _ = _fit_inputs(case, seed)
        _, res, s0 = _exact_match(vox, lib, case["free_s0"])
        return (None, res, s0) if case["free_s0"] else (None, res)
    if kind == "match_host":
        vox, lib, gen = _fit_inputs(case, seed)
        idx, res, s0 = _exact_match(vox, lib, case["free_s0"])
        par = _params(case["n_lib"], gen)[idx.cpu().numpy()]
        out = (par[:, 0], par[:, 1], par[:, 2], res.cpu().numpy())
        return out + (s0.cpu().numpy(),) if case["free_s0"] else out
    if kind == "bayes":
        return _exact_bayes(case, seed)
    return None     # walks, labels and served sums: chains of accept / reject decisions, compared as they are
