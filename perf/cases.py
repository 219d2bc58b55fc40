"""The work that a user of the library has it do, through its public entry
points: simulation of prior draws and parameter sets, acceptance of simulated
particles for observed genes with the posterior summaries that follow, the
error matrix, the deterministic (moment) simulation, the statistics of
observed counts, and the learned pre-screen (training and screening).

Sizes come from the repository's own benchmark, tests and pipeline: 2,000
synthetic cells, 53 statistics (72 in the wide distance workload), five-model
batches with theta padded to 9 columns, 4 to 2,000 genes.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from abc_inference_transcription_gb300 import FP32, FP64, make_config, synthetic_cells
from abc_inference_transcription_gb300.config import REF_FAMILIES, beta_moments
from abc_inference_transcription_gb300.host import Context
from abc_inference_transcription_gb300.surrogate import Surrogate

LD = 9          # theta columns of a five-model batch
N_STATS = 53    # statistics per particle: 4 x 5 ages + 3 x 11 conditions
MODEL_ROW = 14  # surrogate input: padded theta (9) and one-hot model (5)
MEMBERS = 4     # networks of the surrogate ensemble


def listed():
    return [
        # one parameter set re-simulated, as the reference does for a gene's best
        # fit or its example genes: a single abc_sim call, where latency counts
        {"name": "sim_one_gene", "kind": "sim", "model": 1, "prior": "example", "particles": 1, "cells": 2000,
         "device": False, "graph": False},
        # a handful of draws of all five models (a first look, a unit of a sharded
        # run) on an odd number of cells
        {"name": "sim_few_draws", "kind": "sim", "model": 0, "prior": "factor", "particles": 101, "cells": 1437,
         "device": False, "graph": False},
        # an ordinary chunk of the ABC simulation loop, host arrays in and out
        {"name": "sim_batch", "kind": "sim", "model": 0, "prior": "factor", "particles": 2000, "cells": 2000,
         "device": False, "graph": False},
        # a large chunk kept on the device, as the screened pipeline runs it
        {"name": "sim_large_device", "kind": "sim", "model": 0, "prior": "factor", "particles": 10000, "cells": 2000,
         "device": True, "graph": False},
        # acceptance for a few genes at a small quantile, errors kept (the
        # threshold-setting selection of the screened pipeline)
        {"name": "accept_few_genes", "kind": "accept", "particles": 100000, "genes": 4, "stats": 53, "mode": 1,
         "value": 0.002, "errors": True, "device": True, "posterior": False},
        # the reference's acceptance at eps = 4.8 from host arrays, then the
        # posterior summaries and model probabilities of the accepted particles
        {"name": "accept_eps_posterior", "kind": "accept", "particles": 100003, "genes": 487, "stats": 53, "mode": 0,
         "value": 4.8, "errors": True, "device": False, "posterior": True},
        # the wide rejection step: 5 x 10^6 particles x 2,000 genes, top 0.1 %,
        # indices only, as the reference's acceptance writes them
        {"name": "accept_topq_wide", "kind": "accept", "particles": 5000000, "genes": 2000, "stats": 72, "mode": 1,
         "value": 0.001, "errors": False, "device": True, "posterior": False},
        # the full error matrix that compute_trunc_errors writes to file
        {"name": "error_matrix", "kind": "errors", "particles": 3001, "genes": 500, "stats": 53},
        # the reference's deterministic simulation over prior draws of one model
        {"name": "moment_draws", "kind": "moment", "model": 4, "particles": 10000, "exact_mode": False},
        # statistics of observed counts with 100 bootstrap resamples
        {"name": "data_stats", "kind": "data", "genes": 2000, "cells": 2000, "resamples": 100},
        # training of the pre-screen: two passes over simulated draws
        {"name": "screen_train", "kind": "train", "particles": 40000, "epochs": 2, "batch": 4096},
        # screening of fresh draws for a few genes, survivors compacted, and the
        # predictions of a calibration subset
        {"name": "screen_draws", "kind": "screen", "particles": 500000, "genes": 4, "predict": 20000},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["sim", "sim", "sim", "accept", "accept", "accept", "errors", "moment", "data", "train",
                       "screen"])
    if kind == "sim":
        cells = rng.randint(220, 4000)
        device = rng.random() < 0.5
        if rng.random() < 0.25:  # a few parameter sets near the reference's example genes
            return {"kind": "sim", "model": rng.randint(1, 2), "prior": "example", "particles": _log_int(rng, 1, 64),
                    "cells": cells, "device": device, "graph": device and rng.random() < 0.5}
        most = min(8000, int(1.6e7 // cells))
        return {"kind": "sim", "model": rng.choice([0, 0, 0, 1, 2, 3, 4, 5]), "prior": rng.choice(["factor", "reference"]),
                "particles": _log_int(rng, 5, most), "cells": cells, "device": device,
                "graph": device and rng.random() < 0.5}
    if kind == "accept":
        genes = _log_int(rng, 1, 2000)
        particles = _log_int(rng, 1000, min(4e6, 8e9 / genes))
        mode = rng.randint(0, 1)
        device = particles > 300000 or rng.random() < 0.5
        if mode == 1:
            value = math.exp(rng.uniform(math.log(5e-4), math.log(1e-2)))
        else:
            value = rng.uniform(2.0, 4.8)
        return {"kind": "accept", "particles": particles, "genes": genes, "stats": rng.choice([53, 53, 72]),
                "mode": mode, "value": value, "errors": rng.random() < 0.5, "device": device,
                "posterior": particles * genes < 2e8 and rng.random() < 0.5}
    if kind == "errors":
        genes = _log_int(rng, 4, 2000)
        return {"kind": "errors", "particles": _log_int(rng, 100, min(20000, 4e6 / genes)), "genes": genes,
                "stats": rng.choice([53, 72])}
    if kind == "moment":
        exact_mode = rng.random() < 0.25
        return {"kind": "moment", "model": rng.randint(1, 5),
                "particles": _log_int(rng, 1, 500 if exact_mode else 20000), "exact_mode": exact_mode}
    if kind == "data":
        return {"kind": "data", "genes": _log_int(rng, 20, 2000), "cells": rng.randint(220, 4000),
                "resamples": rng.choice([0, 20, 50, 100])}
    if kind == "train":
        return {"kind": "train", "particles": _log_int(rng, 4000, 60000), "epochs": rng.randint(1, 2),
                "batch": rng.choice([512, 1000, 2048, 4096])}
    return {"kind": "screen", "particles": _log_int(rng, 5000, 600000), "genes": _log_int(rng, 1, 50),
            "predict": rng.randint(500, 20000)}


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _cells(n):
    """n synthetic cells over 6 pulse and 5 chase conditions (sizes 5 : 4, as 200 and 160)."""
    full = synthetic_cells(n_per_pulse=math.ceil(n / 2000 * 200) + 2, n_per_chase=math.ceil(n / 2000 * 160) + 2,
                           seed=1)
    keep = np.sort(np.random.default_rng(7).permutation(full.n)[:n])
    cond, age = full.cond[keep].copy(), full.age[keep].copy()
    age[:] = 0
    for j in range(11):  # every (condition, age) group is populated
        sel = np.flatnonzero(cond == j)
        age[sel] = np.random.default_rng(j).permutation(np.arange(sel.size) % 5)
    full.cond, full.age, full.beta = cond, age.astype(np.int32), full.beta[keep].copy()
    w = np.zeros((5, 11))
    np.add.at(w, (full.age, full.cond), 1.0)
    full.age_dist = w / full.n
    return full


def _thetas(rng, model, n, prior):
    """log10 rates (kon, koff, alpha, gamma, labelling), the varying one over five age steps."""
    if prior == "example":  # rates of the reference's example genes, a tenth of a decade around them
        return np.log10([0.5, 1.0, 20.0, 0.1, 0.7]) + rng.uniform(-0.1, 0.1, (n, 5)) * [1, 1, 1, 1, 0.5]
    lo, hi = np.array([-3.0, -3.0, -3.0, -3.0, -0.7]), np.array([3.0, 3.0, 3.0, 2.0, 0.0])
    base = rng.uniform(lo, hi, (n, 5))
    cols = []
    for r in range(5):
        if {3: 0, 4: 2, 5: 3}.get(model) != r:
            cols.append(base[:, r:r + 1])
        elif prior == "factor":  # a base draw times a factor in [0.2, 5] per age step
            cols.append(base[:, r:r + 1] + rng.uniform(math.log10(0.2), math.log10(5.0), (n, 5)))
        else:                    # independent draws per age step
            cols.append(rng.uniform(lo[r], hi[r], (n, 5)))
    return np.ascontiguousarray(np.hstack(cols))


def _batch(rng, n, prior):
    """A five-model batch: theta padded to 9 columns, and the model of each row."""
    models = (1 + np.arange(n) * 5 // n).astype(np.int32)
    theta = np.zeros((n, LD))
    for m in range(1, 6):
        rows = np.flatnonzero(models == m)
        if rows.size:
            th = _thetas(rng, m, rows.size, prior)
            theta[rows, :th.shape[1]] = th
    return theta, models


def _genes_and_stats(case, seed):
    """Particle statistics (log-normal around 256 base vectors), genes near base
    vectors with 5 % noise, and standard errors around 10 % of the statistic."""
    P, G, K = case["particles"], case["genes"], case["stats"]
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    base = torch.exp(1.5 * torch.randn((256, K), device="cuda", dtype=torch.float64, generator=g))
    pick = torch.randint(0, 256, (P,), device="cuda", generator=g)
    stats = torch.randn((P, K), device="cuda", dtype=torch.float64, generator=g).mul_(0.25).exp_()
    for p0 in range(0, P, 1 << 19):
        stats[p0:p0 + (1 << 19)] *= base[pick[p0:p0 + (1 << 19)]]
    rng = np.random.default_rng(seed)
    b = base.cpu().numpy()
    data = b[rng.integers(0, 256, G)] * (1.0 + 0.05 * rng.normal(size=(G, K)))
    se = 0.1 * np.abs(data) * rng.lognormal(0.0, 0.5, (G, K))
    return stats, data, se


def _families(K):
    return list(REF_FAMILIES) if K == N_STATS else None


def _counts(seed, G, cells):
    """Observed counts: gamma-distributed gene levels, Poisson around them."""
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    rng = np.random.default_rng(seed)
    age, cond, beta = (torch.as_tensor(x, device="cuda", dtype=torch.float64) for x in (cells.age, cells.cond, cells.beta))
    mu_u = torch.as_tensor(rng.gamma(2.0, 3.0, (G, 1)), device="cuda") * (1.0 + 0.1 * age)[None, :] * beta[None, :] * 5
    mu_l = torch.as_tensor(rng.gamma(1.5, 1.0, (G, 1)), device="cuda") * (1.0 + 0.03 * cond)[None, :] * beta[None, :] * 5
    return tuple(torch.poisson(m, generator=g).to(torch.int32).cpu().numpy() for m in (mu_u, mu_l))


def _screen_stats(theta, rng):
    """Statistics that vary with the rates as simulated ones do: means, Fano
    factors and correlations of a bursty gene, with sampling noise."""
    kon, koff, alpha, gamma, lam = (10.0 ** theta[:, c] for c in range(5))
    pon = kon / (kon + koff)
    mean = alpha * pon / (gamma + 0.03)
    fano = 1.0 + alpha * koff / ((kon + koff) * (kon + koff + gamma))
    out = np.zeros((theta.shape[0], N_STATS))
    for k in range(5):
        out[:, k] = 0.2 * mean * (1 + 0.1 * k)
        out[:, 5 + k] = 1.0 + 0.2 * (fano - 1.0)
        out[:, 10 + k] = 0.15 * mean * (1 + 0.1 * k)
        out[:, 15 + k] = 1.0 + 0.15 * (fano - 1.0)
    for j in range(11):
        out[:, 20 + j] = lam * (1.0 - np.exp(-gamma * (0.25 + j)))
        out[:, 31 + j] = (fano - 1.0) / (fano + 1.0 + j)
        out[:, 42 + j] = mean / (mean + 10.0 + j)
    return out * np.exp(0.05 * rng.normal(size=out.shape))


def _screen_rows(rng, n):
    theta, models = _batch(rng, n, "factor")
    onehot = np.zeros((n, 5))
    onehot[np.arange(n), models - 1] = 1.0
    return np.ascontiguousarray(np.hstack([theta, onehot])), theta


def prepare(case, seed):
    rng = np.random.default_rng([seed, 11])
    kind = case["kind"]
    s = {"kind": kind, "case": case}
    if kind == "sim":
        s["ctx"] = Context(make_config("hour", precision=FP32), _cells(case["cells"]))
        P = case["particles"]
        if case["model"]:
            s["theta"] = _thetas(rng, case["model"], P, case["prior"])
            s["models"] = None
        else:
            s["theta"], s["models"] = _batch(rng, P, case["prior"])
        s["seed"] = int(rng.integers(1, 1 << 40))
        if case["device"]:
            s["d_theta"] = torch.as_tensor(s["theta"], device="cuda")
            s["d_models"] = None if s["models"] is None else torch.as_tensor(s["models"], device="cuda")
            s["d_stats"] = torch.empty((P, N_STATS), device="cuda", dtype=torch.float64)
            s["ctx"].set_graph(case["graph"])
    elif kind == "accept":
        s["ctx"] = Context(make_config("hour", precision=FP32), None)
        stats, s["data"], s["se"] = _genes_and_stats(case, seed)
        s["stats"] = stats if case["device"] else stats.cpu().numpy()
        if case["mode"] == 0:  # about one particle in 256 is near a gene
            room = case["particles"] * case["genes"] // 100 + 500
            s["indices"], s["errors"] = np.zeros(room, np.int64), np.zeros(room)
        if case["posterior"]:
            s["theta"] = rng.uniform(-3.0, 3.0, (case["particles"], LD))
    elif kind == "errors":
        s["ctx"] = Context(make_config("hour", precision=FP32), None)
        stats, s["data"], s["se"] = _genes_and_stats(case, seed)
        s["stats"] = stats.cpu().numpy()
    elif kind == "moment":
        cells = _cells(2000)
        s["ctx"] = Context(make_config("hour", precision=FP64 if case["exact_mode"] else FP32), cells)
        s["theta"] = _thetas(rng, case["model"], case["particles"], "factor")
        s["iv"] = np.array([0.0, 0.5, 0, 0, 0, 0, 0, 0, 0])
        s["beta"] = beta_moments(cells, 5)
        s["age_dist"] = cells.age_dist
    elif kind == "data":
        cells = _cells(case["cells"])
        s["ctx"] = Context(make_config("hour", precision=FP32), cells)
        s["u"], s["l"] = _counts(seed, case["genes"], cells)
    elif kind == "train":
        s["net"] = Surrogate(MODEL_ROW, N_STATS, ensemble=MEMBERS, seed=seed)
        s["rows"], theta = _screen_rows(rng, case["particles"])
        s["stats"] = _screen_stats(theta, rng)
    elif kind == "screen":
        s["net"] = Surrogate(MODEL_ROW, N_STATS, ensemble=MEMBERS, seed=seed)
        rows, theta = _screen_rows(rng, 8192)
        stats = _screen_stats(theta, rng)
        s["net"].train(rows, stats, epochs=40, batch=2048, lr=2e-3)
        # observed genes: the statistics of ordinary draws (both rates of switching and
        # expression near the middle of the prior), with 5 % noise
        G = case["genes"]
        near = theta.copy()[:G] * 0.3
        d = _screen_stats(near, rng)
        s["data"], s["se"] = d, 0.1 * np.abs(d) * rng.lognormal(0.0, 0.5, d.shape)
        # thresholds and the disagreement bound as the pipeline calibrates them on simulated
        # draws: each gene keeps a few per cent of the prior, the bound passes 99 %
        d_rows = torch.as_tensor(rows, device="cuda")
        keep = torch.empty(8192, device="cuda", dtype=torch.uint8)
        low = np.zeros((8192, G))
        s["thr"], s["disagree"] = np.zeros(G), float(np.quantile(s["net"].predict(rows)[2], 0.99))
        torch.cuda.synchronize()
        s["net"].screen_device(d_rows.data_ptr(), MODEL_ROW, 8192, s["data"], s["se"], s["thr"], 0.0, s["disagree"],
                               keep.data_ptr(), err_out=low, z=1.0)
        s["thr"] = np.quantile(low, 0.06 / G ** 0.5, axis=0)
        fresh, _ = _screen_rows(rng, case["particles"])
        s["rows"] = fresh[:case["predict"]].copy()
        s["d_rows"] = torch.as_tensor(fresh, device="cuda")
        n = case["particles"]
        s["keep"] = torch.empty(n, device="cuda", dtype=torch.uint8)
        s["out"] = torch.zeros((n, MODEL_ROW), device="cuda", dtype=torch.float64)
        s["idx"] = torch.zeros(n, device="cuda", dtype=torch.int64)
    torch.cuda.synchronize()
    return s


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------
def run(s):
    kind, case = s["kind"], s["case"]
    if kind == "sim":
        ctx = s["ctx"]
        if case["device"]:
            P, out = case["particles"], s["d_stats"]
            if s["models"] is None:
                ctx.simulate_device(case["model"], s["d_theta"].data_ptr(), P, s["seed"], out.data_ptr())
            else:
                ctx.simulate_batch_device(s["d_models"].data_ptr(), s["d_theta"].data_ptr(), LD, P, s["seed"],
                                          out.data_ptr())
            ctx.synchronize()  # reports a simulation's status; later work may run on another stream
            return {"stats": out}
        if s["models"] is None:
            return {"stats": ctx.simulate(case["model"], s["theta"], s["seed"])}
        return {"stats": ctx.simulate_batch(s["models"], s["theta"], s["seed"])}
    if kind == "accept":
        ctx, fam = s["ctx"], _families(case["stats"])
        if case["device"]:
            off, idx, err = ctx.select_device(s["data"], s["se"], s["stats"].data_ptr(), case["particles"],
                                              case["mode"], case["value"], families=fam, errors=case["errors"])
        else:
            off, idx, err = ctx.select(s["data"], s["se"], s["stats"], case["mode"], case["value"], fam,
                                       errors=case["errors"])
        if case["mode"] == 0:  # lists of any length, gathered in the program's own arrays
            n = min(idx.size, s["indices"].size)
            s["indices"][:n] = idx[:n]
            idx = s["indices"]
            if case["errors"]:
                s["errors"][:n] = err[:n]
                err = s["errors"]
        out = {"offsets": off, "indices": idx, "errors": err}
        if case["posterior"]:
            out["posterior"] = ctx.posterior_summary(s["theta"])
            n = np.diff(off)
            out["probability"] = ctx.model_probs(np.stack([n // 3, n - n // 3], axis=1))
        return out
    if kind == "errors":
        return {"errors": s["ctx"].errors(s["data"], s["se"], s["stats"], _families(case["stats"]))}
    if kind == "moment":
        return s["ctx"].moment_simulate(case["model"], s["theta"], s["iv"], s["beta"], s["age_dist"])
    if kind == "data":
        st, se = s["ctx"].data_stats(s["u"], s["l"], n_boot=case["resamples"])
        return {"stats": st, "se": se}
    if kind == "train":
        loss = s["net"].train(s["rows"], s["stats"], epochs=case["epochs"], batch=case["batch"])
        return {"loss": loss, "params": s["net"].params()}
    n = case["particles"]
    kept = s["net"].screen_device(s["d_rows"].data_ptr(), MODEL_ROW, n, s["data"], s["se"], s["thr"], 0.0,
                                  s["disagree"], s["keep"].data_ptr(), z=1.0)
    m = s["net"].compact_device(s["keep"].data_ptr(), s["d_rows"].data_ptr(), MODEL_ROW, n, s["out"].data_ptr(),
                                s["idx"].data_ptr())
    mean, var, dis = s["net"].predict(s["rows"])
    return {"kept": kept, "compacted": m, "keep": s["keep"], "rows": s["out"], "indices": s["idx"], "mean": mean,
            "var": var, "disagreement": dis}


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
def work(case):
    kind = case["kind"]
    if kind == "sim":
        P, C = case["particles"], case["cells"]
        # expected fired events per trajectory: about 8,000 under the prior, 1,700 for the
        # example rates; 60 operations each (half a Philox block, log, division, channel, update)
        events = 1700.0 if case["prior"] == "example" else 8000.0
        return {"bytes": 8.0 * P * (LD + N_STATS) + 16.0 * C, "flops": 60.0 * events * P * C}
    if kind in ("accept", "errors"):
        P, G, K = case["particles"], case["genes"], case["stats"]
        if kind == "errors":
            out = 8.0 * P * G
        else:
            out = (16.0 if case["errors"] else 8.0) * P * G * (case["value"] if case["mode"] else 1.0 / 256.0)
        more = 8.0 * P * LD if case.get("posterior") else 0.0
        return {"bytes": 8.0 * P * K + 16.0 * G * K + out + more, "flops": 4.0 * P * G * K}
    if kind == "moment":
        P = case["particles"]
        n = 400 if case["exact_mode"] else 80  # substeps per cycle, with and without labelling
        # a triangular 10 x 10 exponential per substep (about 13 products of 440 operations)
        # and the (condition, age) trajectories from the start of their labelling
        return {"bytes": 8.0 * P * (LD + N_STATS), "flops": P * n * (2 * 13 * 440.0 + 37 * 110.0)}
    if kind == "data":
        G, C, B = case["genes"], case["cells"], case["resamples"]
        draws = 1.0 * G * (B * C * (1.0 + 2.0 / 11.0) + C)
        return {"bytes": 8.0 * G * C + 16.0 * G * N_STATS, "flops": 40.0 * draws}
    layers = 2.0 * (MODEL_ROW * 256 + 2 * 256 * 256 + 256 * 2 * N_STATS) * MEMBERS
    if kind == "train":
        rows = 1.0 * case["particles"] * case["epochs"]
        weights = layers / 2.0 * 4.0
        return {"bytes": 8.0 * case["particles"] * (MODEL_ROW + N_STATS) + 2.0 * weights, "flops": 3.0 * layers * rows}
    n = 1.0 * case["particles"]
    return {"bytes": 8.0 * n * MODEL_ROW * 1.05 + 9.0 * n + 8.0 * case["predict"] * (MODEL_ROW + 2 * N_STATS + 1),
            "flops": layers * (n + case["predict"]) + 5.0 * n * case["genes"] * N_STATS}


# ---------------------------------------------------------------------------
# the same outputs in plain FP64
# ---------------------------------------------------------------------------
def _errors64(data, se, stats):
    d, e = torch.as_tensor(data, device="cuda"), torch.as_tensor(se, device="cuda")
    den = e * e + 0.01 * d * d
    den = den + torch.where(e + d != 0, 0.0, 0.0001)
    st = torch.as_tensor(stats, device="cuda")
    out = torch.empty((st.shape[0], d.shape[0]), device="cuda", dtype=torch.float64)
    for g in range(d.shape[0]):
        out[:, g] = ((d[g] - st).square_() / den[g]).sum(dim=1) / d.shape[1]
    return out.clamp_(max=10.0)


def _posterior64(theta, off, idx, q=0.95):
    G = off.shape[0] - 1
    out = {k: np.full((G, theta.shape[1]), np.nan) for k in ("map", "mean", "lower", "upper")}
    for g in range(G):
        th = theta[idx[off[g]:off[g + 1]] - 1]
        if th.shape[0]:
            out["map"][g], out["mean"][g] = th[0], th.mean(axis=0)
            out["lower"][g], out["upper"][g] = np.quantile(th, 1 - q, axis=0), np.quantile(th, q, axis=0)
    return {**out, "n_particles": None}


def _exact_accept(case, seed):
    s = prepare(case, seed)
    err = _errors64(s["data"], s["se"], s["stats"]).t().contiguous()
    val, order = torch.sort(err, dim=1, stable=True)
    P, G = case["particles"], case["genes"]
    n = (val <= case["value"]).sum(dim=1).cpu().numpy() if case["mode"] == 0 else np.full(G, math.ceil(case["value"] * P))
    off = np.concatenate([[0], np.cumsum(n)])
    val, order = val.cpu().numpy(), order.cpu().numpy()
    out = {"offsets": None, "indices": None, "errors": None}
    if case["errors"]:
        lists = np.concatenate([val[g, :n[g]] for g in range(G)])
        out["errors"] = np.zeros(s["errors"].size) if case["mode"] == 0 else lists
        out["errors"][:lists.size] = lists
    if case["posterior"]:
        idx = np.concatenate([order[g, :n[g]] for g in range(G)]) + 1
        out["posterior"] = _posterior64(s["theta"], off, idx)
        cnt = np.stack([n // 3, n - n // 3], axis=1).astype(np.float64)
        out["probability"] = (cnt / np.maximum(cnt.sum(axis=1, keepdims=True), 1.0), None, None)
    return out


def _stats64(mu, ml, vu, cv, vl, w):
    """Statistics from the moments of every (condition, age), arrays [..., 11, 5]; w [5, 11]."""
    wt = torch.as_tensor(w, device=mu.device).t()
    mean = lambda x: (wt * x).sum(-1)                                                       # noqa: E731
    cov = lambda x, y: (wt * (x - mean(x)[..., None]) * (y - mean(y)[..., None])).sum(-1)   # noqa: E731
    su, sl = mean(mu), mean(ml)
    std = ((mean(vu) + cov(mu, mu)) * (mean(vl) + cov(ml, ml))).abs().sqrt()
    tot, ff = mu + ml, vu + 2 * cv + vl
    fano = ff / torch.where(tot == 0, 0.0001, tot)
    return torch.cat([tot[..., 5, :], fano[..., 5, :], tot[..., 6, :], fano[..., 6, :], sl / (su + sl), mean(cv) / std,
                      cov(mu, ml) / std], dim=-1)


def _exact_moment(case, seed):
    s = prepare(case, seed)
    cfg, model = s["ctx"].cfg, case["model"]
    P, n = case["particles"], 400 if case["exact_mode"] else 80
    T, h, t0 = 20.0, 20.0 / n, -60.0
    dev = torch.device("cuda")
    th = torch.as_tensor(s["theta"], device=dev)
    cols, c = [], 0
    for r in range(5):
        wide = {3: 0, 4: 2, 5: 3}.get(model) == r
        cols.append(10.0 ** (th[:, c:c + 5] if wide else th[:, c:c + 1].expand(-1, 5)))
        c += 5 if wide else 1
    kon, koff, alp, gam, lam = cols
    scal = 0.0 if model == 2 else 1.0

    def generator(k, phase, lab):
        """Moment equations; state 1, EG, Eu, El, VarG, Cov Gu, Cov Gl, Var u, Cov ul, Var l."""
        a = alp[:, k] * (1.0 + phase / T) ** scal
        lb = lam[:, 0] if lab else torch.zeros_like(a)
        a1, a2, ks, g, ko = a * (1 - lb), a * lb, kon[:, k] + koff[:, k], gam[:, k], kon[:, k]
        M = torch.zeros((P, 10, 10), dtype=torch.float64, device=dev)
        for (r, q), v in {(1, 0): ko, (1, 1): -ks, (4, 0): ko, (4, 1): koff[:, k] - ko, (4, 4): -2 * ks, (2, 1): a1,
                          (2, 2): -g, (3, 1): a2, (3, 3): -g, (5, 4): a1, (5, 5): -(ks + g), (6, 4): a2,
                          (6, 6): -(ks + g), (7, 1): a1, (7, 2): g, (7, 5): 2 * a1, (7, 7): -2 * g, (8, 5): a2,
                          (8, 6): a1, (8, 8): -2 * g, (9, 1): a2, (9, 3): g, (9, 6): 2 * a2, (9, 9): -2 * g}.items():
            M[:, r, q] = v
        return M

    prop = [[torch.linalg.matrix_exp(h * generator(i * 5 // n, (i + 0.5) * h, lab)) for i in range(n)]
            for lab in (False, True)]

    def divide(y):
        z = y.clone()
        z[:, 2:4] = 0.5 * y[:, 2:4]
        z[:, 5:7] = 0.5 * y[:, 5:7]
        z[:, 7] = 0.25 * (y[:, 7] + y[:, 2])
        z[:, 9] = 0.25 * (y[:, 9] + y[:, 3])
        z[:, 8] = 0.25 * y[:, 8]
        return z

    cycle = prop[0][0]
    for m in prop[0][1:]:
        cycle = m @ cycle
    y = torch.zeros((P, 10, 1), dtype=torch.float64, device=dev)
    y[:, 0] = 1.0
    y[:, 1:, 0] = torch.as_tensor(s["iv"][[0, 1, 2, 3, 4, 5, 6, 7, 8]], device=dev)
    y = cycle @ y
    live = torch.ones(P, dtype=torch.bool, device=dev)
    for _ in range(101):
        z = cycle @ divide(y)
        old, new = y[:, [1, 2, 4, 5, 7], 0], z[:, [1, 2, 4, 5, 7], 0]
        off = ((old > 0) & ~(((old - new) / old).abs() <= 0.01)).any(dim=1)
        y = torch.where(live[:, None, None], z, y)
        live = live & off
        if not bool(live.any()):
            break
    ages = np.array([2.0, 6.0, 10.0, 14.0, 18.0])
    pulse, chase = (np.array(list(x)[:11]) for x in (cfg.pulse, cfg.chase))
    end = np.broadcast_to(np.rint((ages - t0) / h), (11, 5)).reshape(-1)
    lo = np.rint((ages[None, :] - pulse[:, None] - chase[:, None] - t0) / h).reshape(-1)
    hi = lo + np.rint(np.repeat(pulse, 5) / h)
    y = divide(y).expand(P, 10, 55).contiguous()
    lo, hi, end = (torch.as_tensor(x, device=dev) for x in (lo, hi, end))
    for k in range(int(end.max().item())):
        if k and k % n == 0:
            y = torch.where(k < end, divide(y), y)
        z = torch.where((k >= lo) & (k < hi), prop[1][k % n] @ y, prop[0][k % n] @ y)
        y = torch.where(k < end, z, y)
    m = y.reshape(P, 10, 11, 5)
    mu, ml, vu, cv, vl = (m[:, r] for r in (2, 3, 7, 8, 9))
    b = torch.as_tensor(s["beta"], device=dev)
    b = torch.cat([b[0].expand(6, 5, 3), b[1].expand(5, 5, 3)])
    mb, m2, vb = b[..., 0], b[..., 1], b[..., 2]
    cu = (mb - m2) * mu + vb * (mu * mu + vu) + mb * mb * vu
    cl = (mb - m2) * ml + vb * (ml * ml + vl) + mb * mb * vl
    cc = vb * (mu * ml + cv) + mb * mb * cv
    return {"stats": _stats64(mu * mb, ml * mb, cu, cc, cl, s["age_dist"]), "transient_iters": None}


def _exact_data(case, seed):
    s = prepare(case, seed)
    cells = s["ctx"].cells
    u, l = (torch.as_tensor(s[k], device="cuda").double() for k in ("u", "l"))
    member = torch.zeros((cells.n, 55), dtype=torch.float64, device="cuda")
    member[torch.arange(cells.n), torch.as_tensor(cells.cond.astype(np.int64) * 5 + cells.age)] = 1.0
    n = member.sum(0)
    mean = lambda x: x @ member / n                                                  # noqa: E731
    mu, ml = mean(u), mean(l)
    du, dl = u - mu @ member.t(), l - ml @ member.t()
    var = lambda x, y: ((x * y) @ member) / (n - 1)                                  # noqa: E731
    shape = (u.shape[0], 11, 5)
    st = _stats64(*(x.reshape(shape) for x in (mu, ml, var(du, du), var(du, dl), var(dl, dl))), cells.age_dist)
    # the ratio of a condition is that of all its cells, not of its age groups
    cond = torch.zeros((cells.n, 11), dtype=torch.float64, device="cuda")
    cond[torch.arange(cells.n), torch.as_tensor(cells.cond.astype(np.int64))] = 1.0
    a, b = u @ cond, l @ cond
    st[:, 20:31] = b / (a + b)
    return {"stats": torch.nan_to_num(st, nan=0.0), "se": None}


def exact(case, seed):
    kind = case["kind"]
    if kind == "accept" and 1.0 * case["particles"] * case["genes"] <= 1e8 and (case["errors"] or case["posterior"]):
        return _exact_accept(case, seed)
    if kind == "errors":
        s = prepare(case, seed)
        return {"errors": _errors64(s["data"], s["se"], s["stats"])}
    if kind == "moment" and 1.0 * case["particles"] * (4 if case["exact_mode"] else 1) <= 10000:
        return _exact_moment(case, seed)
    if kind == "data":
        return _exact_data(case, seed)
    return None  # random trajectories, and a trained network's outputs
