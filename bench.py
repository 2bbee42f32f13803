"""Benchmark: plain VEGAS on one GB300 (and N independent replicas on N GPUs).

Workload (the configuration the headline metric is quoted on): VEGAS+,
dim 6, N = 1e7 evaluations budget (max_iterations 20), 50 map intervals per
dimension, default stratification (6^6 cubes), fp32 points with fp64
compensated sums, integrand prod_i N(x_i; 0.5, 0.05) on [0,1]^6 (value ~1),
seeds 0, 1, 2, ... per step.  A step is one full VEGAS integration.

  python bench.py [--gpus N] [--steps K] [--warmup W] [--impl reference]

Our arm prints one JSON line: ``value`` = integrand evaluations per second
over the timed steps with inputs resident on the device; ``e2e`` = the same
metric through the public API with the domain given as a host list and the
result read back to the host every step; ``roofline`` for the dominant
kernel (the fused VEGAS sampler) against an FP32 FMA peak measured in the
same run; ``cpu_baseline`` = the CPU oracle (numpy restatement of the
reference) on the host, one process.

``--impl reference`` times the reference algorithm on the host cores
instead (the numpy restatement; the reference itself is pure Python over
torch and not installable on the GPU host): each step runs one integration
per host core in parallel processes.
"""
from __future__ import annotations

import argparse
import ctypes
import json
import math
import os
import statistics
import subprocess
import sys
import time
from pathlib import Path

ROOT = Path(__file__).resolve().parent
sys.path.insert(0, str(ROOT))

DIM, N_EVALS, N_BINS, SIGMA = 6, 10_000_000, 50, 0.05
METRIC = "integrand evals/s (plain VEGAS, dim 6, N=1e7, 50 bins, fp32 + fp64 sums)"
UNIT = "evals/s"
CONFIG = {
    "workload": "plain VEGAS+ dim=6 N=1e7 budget, 50 map bins/dim, default stratification (6^6 cubes), "
                "Gaussian peak sigma=0.05 on [0,1]^6, fp32 points with fp64 compensated sums, one integration per step",
    "dim": DIM,
    "N": N_EVALS,
    "n_bins": N_BINS,
    "max_iterations": 20,
    "integrand": "prod_i exp(-(x_i-0.5)^2/(2*0.05^2))/(0.05*sqrt(2*pi))",
    "l2": "flushed (256 MiB write) between timed steps, outside the per-step CUDA events",
}


def reduce_over_ranks(t_local, e2e_t, evals, e2e_evals, ws, device):
    """Replicas: the slowest rank's times (MAX) and all ranks' evaluations
    (SUM); value = all evaluations / the slowest time."""
    if ws <= 1:
        return t_local, e2e_t, evals, e2e_evals
    import torch
    import torch.distributed as dist

    t = torch.tensor([t_local, e2e_t], dtype=torch.float64, device=device)
    dist.all_reduce(t, op=dist.ReduceOp.MAX)
    n = torch.tensor([float(evals), float(e2e_evals)], dtype=torch.float64, device=device)
    dist.all_reduce(n, op=dist.ReduceOp.SUM)
    return float(t[0]), float(t[1]), int(n[0]), int(n[1])


def rank_seed(rank, k):
    """Seed of timed integration k on a rank: distinct across ranks and steps."""
    return rank * 1_000_003 + k


def _dist_env():
    ws = int(os.environ.get("WORLD_SIZE", "1"))
    rank = int(os.environ.get("RANK", "0"))
    local = int(os.environ.get("LOCAL_RANK", "0"))
    return ws, rank, local


# ------------------------------------------------------------ helpers
HBM_FALLBACK_GBS = 6800.0


def hbm_peak():
    """(GB/s, source): the measured copy bandwidth of the GB300s
    (MEASURED_PEAKS.json next to this file), else the fallback figure."""
    try:
        with open(ROOT / "MEASURED_PEAKS.json") as fh:
            v = float(json.load(fh)["hbm_gbs"])
        return v, "of measured (MEASURED_PEAKS.json hbm_gbs)"
    except (OSError, KeyError, ValueError):
        return HBM_FALLBACK_GBS, "of fallback (6.8 TB/s)"


def fp_peaks(L, torch):
    """FP32 and FP64 FMA peaks (TFLOP/s) measured in this run by the probe
    kernels (best of three launches)."""
    out = {}
    for name, dt, fn in (("fp32", torch.float32, "tq_fp32_fma_probe"), ("fp64", torch.float64, "tq_fp64_fma_probe")):
        buf = torch.zeros(1, dtype=dt, device="cuda")
        flops = ctypes.c_double(0.0)
        best = 0.0
        iters = 4096 if name == "fp32" else 64
        for _ in range(3):
            e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            e0.record()
            L.check(getattr(L.lib(), fn)(iters, 8, buf.data_ptr(), ctypes.byref(flops), L.stream_handle()), fn)
            e1.record()
            torch.cuda.synchronize()
            best = max(best, flops.value / (e0.elapsed_time(e1) / 1000.0) / 1e12)
        out[name] = best
    return out


def timed_launches(torch, fn, reps, flush=None):
    """Mean device time (s) of fn over reps launches (CUDA events on the
    current stream); with flush, L2 is overwritten before every launch and
    each launch is timed on its own."""
    fn()
    torch.cuda.synchronize()
    if flush is None:
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        e0.record()
        for _ in range(reps):
            fn()
        e1.record()
        torch.cuda.synchronize()
        return e0.elapsed_time(e1) / reps / 1000.0
    tot = 0.0
    for k in range(reps):
        flush.fill_(k & 0xFF)
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        e0.record()
        fn()
        e1.record()
        torch.cuda.synchronize()
        tot += e0.elapsed_time(e1) / 1000.0
    return tot / reps


def cpu_cores_used():
    return 1


def c2_accuracy(results, errors):
    """Relative error of the timed plain-VEGAS integrations against the
    analytic integral erf(0.5 / (0.05 sqrt 2))^6 (the normal densities
    truncated to [0, 1]^6), with VEGAS's own error estimate beside it."""
    import numpy as np

    exact = math.erf(0.5 / (SIGMA * math.sqrt(2.0))) ** DIM
    rel = np.abs(np.array(results) - exact) / exact
    est = np.array(errors) / exact
    return {"analytic": exact, "rel_err_median": float(np.median(rel)), "rel_err_max": float(np.max(rel)),
            "frac_within_1e-4": float(np.mean(rel <= 1e-4)), "reported_rel_error_median": float(np.median(est)),
            "integrations": len(results)}


# ------------------------------------------------- batched workload (C3)
def c3_workload(n=4096, seed=1):
    """4096 independent Gaussian-peak integrals: dims U{1..4}, rule U{trapezoid,
    simpson, boole, gausslegendre}, N log-uniform 1e3..1e6 (points per
    dimension then made valid for the rule), f = exp(-sum a_i (x_i-u_i)^2),
    a_i ~ U[0.5, 5], u_i ~ U[0, 1], domains [l, l+w], l ~ U[-1, 0],
    w ~ U[0.5, 2]; returns (specs, analytic values).  Gauss-Legendre
    integrals use at most 256 nodes per dimension: the nodes come from
    numpy's leggauss (as in the reference), which builds an n x n matrix."""
    import numpy as np

    rng = np.random.default_rng(seed)
    rules = ["trapezoid", "simpson", "boole", "gausslegendre"]
    out, exact = [], []
    for _ in range(n):
        d = int(rng.integers(1, 5))
        rule = rules[int(rng.integers(0, 4))]
        N = int(10 ** rng.uniform(3, 6))
        if rule == "gausslegendre":
            N = min(N, 256**d)
        a = rng.uniform(0.5, 5.0, d)
        u = rng.uniform(0.0, 1.0, d)
        lo = rng.uniform(-1.0, 0.0, d)
        w = rng.uniform(0.5, 2.0, d)
        dom = np.stack([lo, lo + w], axis=1)
        out.append((rule, d, N, dom, a, u))
        v = 1.0
        for k in range(d):
            s = math.sqrt(a[k])
            v *= math.sqrt(math.pi / a[k]) / 2.0 * (math.erf(s * (lo[k] + w[k] - u[k])) - math.erf(s * (lo[k] - u[k])))
        exact.append(v)
    return out, exact


def c3_cpu_baseline(specs, budget_s=6.0):
    """The oracle port (numpy restatement of the reference's per-call grid
    rules) over the integrals of the workload in order, until budget_s."""
    import numpy as np

    from oracle import grid as OG
    from oracle import integrands as OI

    rid = {"trapezoid": OG.TRAPEZOID, "simpson": OG.SIMPSON, "boole": OG.BOOLE, "gausslegendre": OG.GAUSS}
    t0 = time.perf_counter()
    k = 0
    nodes = 0
    while k < len(specs) and time.perf_counter() - t0 < budget_s:
        rule, d, N, dom, a, u = specs[k]
        params = np.concatenate([[1.0, 0.0], a, u])
        OG.integrate(lambda x: OI.evaluate(2, params, x), rid[rule], d, N, dom)
        nodes += OG.n_per_dim(OG.adjust_N(rid[rule], d, N), d) ** d
        k += 1
    t = time.perf_counter() - t0
    return {"integrals_per_s": k / t, "unit": "integrals/s", "cores": cpu_cores_used(), "kind": "port",
            "sample": f"the first {k} integrals of the workload ({nodes} nodes), numpy restatement of the "
                      "reference's per-call grid rules, one process"}


def measure_batched(tq, dev, L, peaks, reps=5):
    """Batched (one persistent launch) vs plain per-call integration of the
    4096-integral workload, fp32 and fp64; integrals/s and accuracy."""
    import warnings

    import numpy as np
    import torch
    from torchquad_gb300 import batch as B

    specs, exact = c3_workload()
    exact = np.array(exact)
    cls = {"trapezoid": tq.Trapezoid, "simpson": tq.Simpson, "boole": tq.Boole, "gausslegendre": tq.GaussLegendre}
    out = {"workload": "4096 Gaussian-peak integrals, dims 1-4, trapezoid/simpson/boole/gausslegendre, "
                       "N log-uniform 1e3-1e6, seed 1"}
    for dtype in (torch.float32, torch.float64):
        name = "fp32" if dtype == torch.float32 else "fp64"
        fs = [tq.GaussianPeak(d, a=a.tolist(), u=u.tolist()) for (_, d, _, _, a, u) in specs]
        rules = [sp[0] for sp in specs]
        Ns = [sp[2] for sp in specs]
        doms = [sp[3] for sp in specs]
        bg = B.BatchedGrid(dtype=dtype, autotune=True)
        plan = bg.plan(fs, rules, Ns, doms)
        shape = bg.tuned_shape(plan)
        plan = bg.retile(plan, shape[2])
        vals = bg.run(plan, shape)
        t_batch = timed_launches(torch, lambda: bg.run(plan, shape), reps)
        torch.cuda.synchronize()
        t0 = time.perf_counter()
        v_e2e = bg.integrate(fs, rules, Ns, doms).cpu()
        t_e2e = time.perf_counter() - t0
        vb = vals.double().cpu().numpy()
        dtens = [torch.tensor(dm, dtype=dtype, device=dev) for dm in doms]
        with warnings.catch_warnings():
            warnings.simplefilter("ignore")
            for i in range(64):  # warm-up
                cls[rules[i]]().integrate(fs[i], fs[i].dim, N=Ns[i], integration_domain=dtens[i])
            torch.cuda.synchronize()
            t0 = time.perf_counter()
            plain = [cls[r]().integrate(f, f.dim, N=N, integration_domain=dt)
                     for r, f, N, dt in zip(rules, fs, Ns, dtens)]
            torch.cuda.synchronize()
            t_plain = time.perf_counter() - t0
        vp = np.array([float(x) for x in plain])
        rel = np.abs(vb - exact) / np.abs(exact)
        d = plan.desc_np
        terms = int(np.sum(d["n"] * d["dim"]))
        rec = {
            "batched_integrals_per_s": len(specs) / t_batch,
            "batched_ms": t_batch * 1000.0,
            "batched_e2e_integrals_per_s": len(specs) / t_e2e,
            "plain_integrals_per_s": len(specs) / t_plain,
            "speedup_batched_vs_plain": t_plain / t_batch,
            "speedup_batched_e2e_vs_plain": t_plain / t_e2e,
            "nodes_per_s": plan.total_points / t_batch,
            "total_nodes": plan.total_points,
            "tuned_shape": {"block": shape[0], "strip": shape[1], "tile_points": shape[2], "ctas": shape[3]},
            "frac_within_1e-4_of_analytic": float(np.mean(rel <= 1e-4)),
            "median_rel_err_vs_analytic": float(np.median(rel)),
            "max_rel_diff_batched_vs_plain": float(np.max(np.abs(vb - vp) / np.maximum(np.abs(vp), 1e-300))),
            "max_rel_diff_e2e_vs_resident": float(np.max(np.abs(v_e2e.double().numpy() - vb) / np.abs(vb))),
        }
        if dtype == torch.float64:
            # the sums factor into dim * n one-dimensional terms an integral:
            # the argument's multiply, the weight's multiply and the add of
            # each (the term's exp, cos or sin and long rows' Horner steps
            # are not counted)
            rec["terms_per_s"] = terms / t_batch
            ach = 3.0 * terms / t_batch / 1e12
            rec["roofline"] = {"bound": "fp64 and latency", "achieved": ach, "peak": peaks["fp64"],
                               "unit": "TFLOP/s", "frac": ach / peaks["fp64"], "ops_per_term": 3,
                               "terms": terms, "peak_source": "FP64 FMA probe measured in this run"}
        out[name] = rec
    out["cpu_baseline"] = c3_cpu_baseline(specs)
    return out


def measure_grid_cases(tq, dev, L, peaks, flush, reps=20):
    """C1: plain Simpson, dim 3, 101 points per dimension (N = 1,030,301),
    fp64, exp(x0+x1+x2) on [0,1]^3 against (e-1)^3: the API call, the fused
    kernel alone (C-ABI, CUDA events) with its FP64 roofline, and the
    materialised path (any torch callable) with the HBM roofline of its two
    kernels, also at 301^3 nodes.  C4: GaussLegendre, dim 4, 32 nodes per
    dimension, fp64, cos(2 pi u + a.x) with u and the domain bounds
    requiring gradients: forward and forward+backward times, gradients
    against central differences (h = 1e-6), and the batch of 1024 such
    integrals through the batched adjoint."""
    import numpy as np
    import torch

    lib = L.lib()
    hbm, hbm_src = hbm_peak()

    def timed(fn):
        return timed_launches(torch, fn, reps) * 1000.0

    out = {}
    # ---------------------------------------------------------------- C1
    dom = torch.tensor([[0.0, 1.0]] * 3, dtype=torch.float64, device=dev)
    f1 = tq.ExpSum(3)
    v = tq.Simpson().integrate(f1, 3, N=1_030_301, integration_domain=dom)
    ms = timed(lambda: tq.Simpson().integrate(f1, 3, N=1_030_301, integration_domain=dom))
    exact = (math.e - 1.0) ** 3
    t0 = time.perf_counter()
    v_e2e = tq.Simpson().integrate(f1, 3, N=1_030_301,
                                   integration_domain=torch.tensor([[0.0, 1.0]] * 3, dtype=torch.float64)).item()
    t_e2e = time.perf_counter() - t0
    n, nodes = 101, 101**3
    params = f1.device_params(dev)
    res = torch.empty((), dtype=torch.float64, device=dev)
    ws = torch.zeros(lib.tq_grid_fused_workspace_size(L.TQ_RULE_SIMPSON, 3, n), dtype=torch.uint8, device=dev)

    def fused():
        L.check(lib.tq_grid_fused(L.TQ_F64, L.TQ_RULE_SIMPSON, 3, n, dom.data_ptr(), None, None, f1.family,
                                  params.data_ptr(), res.data_ptr(), L.TQ_F64, None, ws.data_ptr(), ws.numel(),
                                  L.stream_handle()), "tq_grid_fused")

    t_k = timed_launches(torch, fused, 200)
    ach = 3.0 * 3 * n / t_k / 1e12
    c1 = {"api_ms": ms, "kernel_us": t_k * 1e6, "nodes_per_s": nodes / t_k, "terms_per_s": 3 * n / t_k,
          "e2e_ms": t_e2e * 1000.0, "rel_err_vs_analytic": abs(v.item() - exact) / exact,
          "e2e_value_matches": v_e2e == v.item(),
          "roofline": {"kernel": "grid_fused_kernel<double,double,SIMPSON,EXP_SUM>", "bound": "latency",
                       "achieved": ach, "peak": peaks["fp64"], "unit": "TFLOP/s", "frac": ach / peaks["fp64"],
                       "ops_per_term": 3, "peak_source": "FP64 FMA probe measured in this run",
                       "note": "the sum factors into 3 x 101 one-dimensional terms (argument and weight "
                               "multiply and an add each): a few warps, so the launch and its reductions "
                               "are latency"}}
    # materialised path: an arbitrary torch callable
    fn = lambda x: torch.exp(x.sum(1))  # noqa: E731
    c1["materialised_api_ms"] = timed(lambda: tq.Simpson().integrate(fn, 3, N=nodes, integration_domain=dom))
    mat = {}
    for tag, nn in (("n101", 101), ("n301", 301)):
        tot = nn**3
        pts = torch.empty((tot, 3), dtype=torch.float64, device=dev)

        def gp():
            L.check(lib.tq_grid_points(L.TQ_F64, L.TQ_RULE_SIMPSON, 3, nn, dom.data_ptr(), None, 0, tot,
                                       pts.data_ptr(), L.stream_handle()), "tq_grid_points")

        t_p = timed_launches(torch, gp, 10, flush)
        fv = torch.exp(pts.sum(1))
        acc = torch.zeros(2, dtype=torch.float64, device=dev)
        wsw = torch.zeros(lib.tq_weighted_sum_workspace_size(tot, 1), dtype=torch.uint8, device=dev)

        def wsum():
            L.check(lib.tq_weighted_sum(L.TQ_F64, L.TQ_RULE_SIMPSON, 3, nn, dom.data_ptr(), None, 0, tot,
                                        fv.data_ptr(), L.TQ_F64, 1, acc.data_ptr(), wsw.data_ptr(), wsw.numel(),
                                        L.stream_handle()), "tq_weighted_sum")

        t_w = timed_launches(torch, wsum, 10, flush)
        bp, bw = tot * 3 * 8, tot * 8
        mat[tag] = {
            "nodes": tot,
            "grid_points": {"us": t_p * 1e6, "bytes": bp, "achieved_gbs": bp / t_p / 1e9, "peak_gbs": hbm,
                            "frac": bp / t_p / 1e9 / hbm, "bytes_per_node": 24},
            "weighted_sum": {"us": t_w * 1e6, "bytes": bw, "achieved_gbs": bw / t_w / 1e9, "peak_gbs": hbm,
                             "frac": bw / t_w / 1e9 / hbm, "bytes_per_node": 8,
                             "arithmetic": "pairs of values added in fp64, the pairs split into two floats "
                                           "by integer operations and summed as double-floats"},
        }
        del pts, fv
    mat["peak_source"] = hbm_src
    mat["l2"] = "flushed (256 MiB write) before every timed launch"
    c1["materialised"] = mat
    out["c1_simpson_d3_fp64"] = c1

    # ---------------------------------------------------------------- C4
    a = [1.2, -2.1, 0.7, 2.6]
    u0 = 0.37

    def fwd(u, d):
        return tq.GaussLegendre().integrate(tq.Oscillatory(4, a=a, b=u), 4, N=32**4, integration_domain=d)

    u = torch.tensor(u0, dtype=torch.float64, device=dev, requires_grad=True)
    d4 = torch.tensor([[0.0, 1.0]] * 4, dtype=torch.float64, device=dev, requires_grad=True)
    with torch.no_grad():
        ms_f = timed(lambda: fwd(torch.tensor(u0, dtype=torch.float64, device=dev),
                                 torch.tensor([[0.0, 1.0]] * 4, dtype=torch.float64, device=dev)))

    def fb():
        u.grad = None
        d4.grad = None
        val = fwd(u, d4)
        val.backward()
        return val

    ms_fb = timed(fb)
    g = np.concatenate([[u.grad.item()], d4.grad.double().cpu().numpy().ravel()])
    h = 1e-6
    fd = []
    with torch.no_grad():
        for k in range(9):
            up, dp = u0, np.array([[0.0, 1.0]] * 4)
            um, dm = u0, dp.copy()
            if k == 0:
                up, um = u0 + h, u0 - h
            else:
                dp = dp.copy()
                dp.ravel()[k - 1] += h
                dm.ravel()[k - 1] -= h
            fp = fwd(torch.tensor(up, dtype=torch.float64, device=dev), torch.tensor(dp, device=dev)).item()
            fm = fwd(torch.tensor(um, dtype=torch.float64, device=dev), torch.tensor(dm, device=dev)).item()
            fd.append((fp - fm) / (2 * h))
    fd = np.array(fd)
    c4 = {"forward_ms": ms_f, "forward_backward_ms": ms_fb, "nodes_per_s": 32**4 / (ms_f / 1000.0),
          "max_abs_grad_diff_vs_central_differences": float(np.max(np.abs(g - fd))),
          "max_abs_grad": float(np.max(np.abs(g)))}
    c4["batch_1024"] = measure_c4_batch(tq, dev, peaks)
    out["c4_gausslegendre_d4_grad_fp64"] = c4
    return out


def measure_c4_batch(tq, dev, peaks, m=1024):
    """1024 differentiation integrals (GL dim 4, 32 nodes, fp64, random a, u)
    with gradients: the batched adjoint (device time, and end to end from
    host parameters through backward) against the per-call form and the
    numpy port on the host."""
    import numpy as np
    import torch
    from torchquad_gb300 import batch as B

    from oracle import grad as OGR

    rng = np.random.default_rng(4)
    a = rng.uniform(-3.0, 3.0, (m, 4))
    us = rng.uniform(0.0, 1.0, m)
    fs = [tq.Oscillatory(4, a=a[i].tolist(), b=float(us[i])) for i in range(m)]
    bg = B.BatchedGrid(dtype=torch.float64)
    plan = bg.plan(fs, ["gausslegendre"] * m, [32**4] * m, [[[0.0, 1.0]] * 4] * m, tile_points=65536)
    t_dev = timed_launches(torch, lambda: bg.adjoint(plan), 5)
    vals, gdom, gpar = bg.adjoint(plan)

    def e2e():
        u = torch.tensor(us, dtype=torch.float64, requires_grad=True)
        d = torch.tensor([[[0.0, 1.0]] * 4] * m, dtype=torch.float64, requires_grad=True)
        ff = [tq.Oscillatory(4, a=a[i].tolist(), b=u[i]) for i in range(m)]
        v = bg.integrate(ff, ["gausslegendre"] * m, [32**4] * m, list(d))
        v.sum().backward()
        return float(v.detach().sum()), u.grad, d.grad

    e2e()
    torch.cuda.synchronize()
    t0 = time.perf_counter()
    e2e()
    t_e2e = time.perf_counter() - t0
    # per-call form: integrate + backward, one integral at a time
    k = 64
    torch.cuda.synchronize()
    t0 = time.perf_counter()
    diffs = []
    for i in range(k):
        ui = torch.tensor(us[i], dtype=torch.float64, device=dev, requires_grad=True)
        di = torch.tensor([[0.0, 1.0]] * 4, dtype=torch.float64, device=dev, requires_grad=True)
        vi = tq.GaussLegendre().integrate(tq.Oscillatory(4, a=a[i].tolist(), b=ui), 4, N=32**4, integration_domain=di)
        vi.backward()
        diffs.append(abs(vi.item() - vals[i].item()) / max(1.0, abs(vi.item())))
    torch.cuda.synchronize()
    t_plain = (time.perf_counter() - t0) / k
    # host port: value and gradient in numpy (one core), bounded sample
    t0 = time.perf_counter()
    j = 0
    while j < m and time.perf_counter() - t0 < 5.0:
        OGR.value_and_grad(3, np.concatenate([[1.0, us[j]], a[j], np.zeros(4)]), OGR.GAUSS, 4, 32, [[0.0, 1.0]] * 4)
        j += 1
    t_cpu = (time.perf_counter() - t0) / j
    terms = m * 4 * 32
    ach = 12.0 * terms / t_dev / 1e12
    return {
        "batched_device_ms": t_dev * 1e3, "batched_fwd_bwd_integrals_per_s": m / t_dev,
        "batched_e2e_ms": t_e2e * 1e3, "batched_e2e_integrals_per_s": m / t_e2e,
        "plain_fwd_bwd_integrals_per_s": 1.0 / t_plain,
        "speedup_batched_vs_plain": t_plain * m / t_dev, "speedup_batched_e2e_vs_plain": t_plain * m / t_e2e,
        "max_rel_diff_batched_vs_plain_sample": float(max(diffs)),
        "roofline": {"kernel": "batch_adjoint_kernel", "bound": "latency",
                     "achieved": ach, "peak": peaks["fp64"], "unit": "TFLOP/s", "frac": ach / peaks["fp64"],
                     "ops_per_term": 12, "peak_source": "FP64 FMA probe measured in this run",
                     "note": "value and gradient factor into six weighted moments of each dimension's 32 "
                             "nodes (a multiply and an add each; the cos and sin are not counted)"},
        "cpu_baseline": {"integrals_per_s": 1.0 / t_cpu, "unit": "integrals/s (value + gradient)",
                         "cores": cpu_cores_used(), "kind": "port",
                         "sample": f"{j} of the integrals, numpy gradient of the discrete rule "
                                   "(oracle/grad.py), one process"},
    }


def vegas_batch_workload(n=1024, seed=5):
    """C5's VEGAS share at the sizes one batch holds: the first n VEGAS
    requests of the serving stream (dims 1-10, Gaussian-peak or oscillatory
    integrands, target relative error 1e-3..1e-5) with N log-uniform in
    1e4..2.56e5 (maps of at most 1024 intervals), fp32."""
    from torchquad_gb300.serving import poisson_stream

    reqs = [r for _, r in poisson_stream(4 * n, 1e5, seed=seed, n_range=(1e4, 2.56e5)) if r.method == "vegas"]
    return reqs[:n]


def measure_vegas_batch(tq, dev, n=1024, reps=5, k_plain=128):
    """Batched VEGAS (torchquad_gb300.vegas_batch) on C5's VEGAS share: every
    integral keeps its own N, target error and seed; the batch replays one
    captured graph (one launch per phase for all integrals).  Against the
    per-call VEGAS().integrate of the same requests (a sample, one after the
    other) and the numpy port on the host."""
    import numpy as np
    import torch
    from torchquad_gb300 import _lib as L
    from torchquad_gb300.vegas_batch import VegasBatch

    from oracle import integrands as OI
    from oracle import philox as OP
    from oracle import vegas as OV

    reqs = vegas_batch_workload(n)
    fns = [r.integrand for r in reqs]
    Ns = [r.N for r in reqs]
    doms = [r.domain for r in reqs]
    seeds = [r.seed for r in reqs]
    eps = [r.eps_rel for r in reqs]
    vb = VegasBatch(fns, Ns, dtype=torch.float32)

    def call():
        return vb.integrate(domains=doms, seeds=seeds, eps_rel=eps)

    call()  # eager
    call()  # captures the graph
    launches0 = L.launches[0]
    torch.cuda.synchronize()
    t0 = time.perf_counter()
    for _ in range(reps):
        res = call()
    t_e2e = (time.perf_counter() - t0) / reps
    launches = (L.launches[0] - launches0) // reps
    # device time of the graph alone (CUDA events on the replaying stream)
    ev = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
    ev[0].record()
    for _ in range(reps):
        vb.graph.replay()
    ev[1].record()
    torch.cuda.synchronize()
    t_dev = ev[0].elapsed_time(ev[1]) / 1e3 / reps
    res = call().cpu().numpy().astype(np.float64)
    evals = int(vb.nr_of_fevals.sum())
    its = vb.it.copy()
    exact = np.array([f.exact(d) for f, d in zip(fns, doms)])
    err = np.abs(res - exact) / np.maximum(np.abs(exact), 1e-300)
    # per-call form on a sample of the same requests
    k = min(k_plain, n)

    def per_call(i):
        v = tq.VEGAS()
        r = v.integrate(fns[i], fns[i].dim, N=Ns[i], integration_domain=torch.tensor(doms[i], dtype=torch.float32,
                                                                                     device=dev),
                        seed=seeds[i], eps_rel=eps[i])
        return float(r), v._nr_of_fevals

    for i in range(min(8, k)):
        per_call(i)
    torch.cuda.synchronize()
    t0 = time.perf_counter()
    plain = [per_call(i) for i in range(k)]
    t_plain = (time.perf_counter() - t0) / k
    diff = max(abs(plain[i][0] - res[i]) / max(abs(plain[i][0]), 1e-300) for i in range(k))
    # numpy port on the host, the requests in order, bounded
    t0 = time.perf_counter()
    j = 0
    while j < n and time.perf_counter() - t0 < 8.0:
        r = reqs[j]
        p = r.integrand.params_numpy()
        OV.Vegas().integrate(lambda x, fam=r.integrand.family, p=p: OI.evaluate(fam, p, x), r.dim, r.N, r.domain,
                             OP.ReplayStream(r.seed), dt=np.float32, eps_rel=r.eps_rel)
        j += 1
    t_cpu = (time.perf_counter() - t0) / max(1, j)
    h2d = n * ctypes.sizeof(L.VegasRun)
    return {
        "workload": f"{n} VEGAS requests of the serving stream (seed 5), dims 1-10, N log-uniform "
                    "1e4..2.56e5, target rel err 1e-3..1e-5, fp32, Gaussian-peak / oscillatory",
        "integrals": n, "evals": evals, "max_iterations_run": int(its.max()),
        "batched_device_ms": t_dev * 1e3, "batched_integrals_per_s": n / t_dev,
        "batched_evals_per_s": evals / t_dev,
        "e2e": {"ms": t_e2e * 1e3, "integrals_per_s": n / t_e2e, "h2d_bytes_per_call": h2d,
                "d2h_bytes_per_call": vb._rb.numel() * 8},
        "gpu_launches_per_call": launches,
        "plain_per_call_integrals_per_s": 1.0 / t_plain, "plain_sample": k,
        "speedup_batched_vs_plain": t_plain * n / t_dev, "speedup_batched_e2e_vs_plain": t_plain * n / t_e2e,
        "max_rel_diff_batched_vs_plain_sample": float(diff),
        "accuracy": {"median_rel_err": float(np.median(err)),
                     "frac_within_target_rel_err": float(np.mean(err <= np.asarray(eps))),
                     "frac_within_1e-3": float(np.mean(err <= 1e-3))},
        "cpu_baseline": {"integrals_per_s": 1.0 / t_cpu, "unit": "integrals/s", "cores": cpu_cores_used(),
                         "kind": "port", "sample": f"the first {j} requests, numpy VEGAS restatement "
                                                  "(oracle/vegas.py), one process"},
    }


def _serving_accuracy(reqs):
    import numpy as np

    ratios, within = [], []
    for r in reqs:
        ex = r.integrand.exact(r.domain)
        err = abs(r.result - ex) / max(abs(ex), 1e-300)
        ratios.append(err / r.eps_rel)
        within.append(err <= r.eps_rel)
    return {"frac_within_target_rel_err": float(np.mean(within)),
            "median_rel_err_over_target": float(np.median(ratios)),
            "p90_rel_err_over_target": float(np.percentile(ratios, 90))}


def measure_serving(tq, dev, n=1000, rates=(1e2, 1e3, 1e4, 1e5)):
    """Poisson request streams (MC / VEGAS / Simpson, dims 1-10, N log-uniform
    1e4..1e8, target relative error 1e-3..1e-5, seed 2) through the serving
    loop: p50/p99 latency, integrals/s, evaluations and accuracy against the
    closed-form integral per arrival rate.  Matched work: Monte Carlo runs to
    its N as MonteCarlo.integrate does (the per-call form has no stopping
    rule); the early-stop variant, which stops Monte Carlo at its target
    error, is reported beside it at the highest rate.  The same requests
    then go through the plain per-call API one after the other."""
    import warnings

    import numpy as np
    import torch
    from torchquad_gb300.serving import IntegrationServer, poisson_stream

    out = {"requests_per_rate": n}

    def serve(rate, early):
        stream = poisson_stream(n, rate, seed=2)
        with IntegrationServer(max_active=64, mc_early_stop=early) as srv:
            t0 = time.perf_counter()
            for t_arr, req in stream:
                delay = t0 + t_arr - time.perf_counter()
                if delay > 0:
                    time.sleep(delay)
                srv.submit(req)
            srv.drain(timeout=900)
            st = srv.stats()
            reqs = list(srv.completed)
        rec = {k: st[k] for k in ("p50_ms", "p99_ms", "integrals_per_s", "peak_active", "evals")}
        rec.update(_serving_accuracy(reqs))
        return rec

    for rate in rates:
        out[f"rate_{int(rate)}"] = serve(rate, False)
    out[f"rate_{int(rates[-1])}_mc_early_stop"] = serve(rates[-1], True)
    # plain per-call path, same requests, back to back
    stream = poisson_stream(n, rates[-1], seed=2)
    cls = {"montecarlo": tq.MonteCarlo, "vegas": tq.VEGAS, "simpson": tq.Simpson}
    lat, evals, done = [], 0, []
    with warnings.catch_warnings():
        warnings.simplefilter("ignore")
        torch.cuda.synchronize()
        t0 = time.perf_counter()
        for _, r in stream:
            t1 = time.perf_counter()
            dom = torch.tensor(r.domain, dtype=r.dtype, device=dev)
            kw = {"seed": r.seed} if r.method != "simpson" else {}
            if r.method == "vegas":
                kw["eps_rel"] = r.eps_rel
            integ = cls[r.method]()
            r.result = integ.integrate(r.integrand, r.dim, N=r.N, integration_domain=dom, **kw).item()
            evals += int(integ._nr_of_fevals)
            lat.append(time.perf_counter() - t1)
            done.append(r)
        t_plain = time.perf_counter() - t0
    out["plain_per_call"] = {"integrals_per_s": n / t_plain, "p50_ms": float(np.percentile(lat, 50) * 1e3),
                             "p99_ms": float(np.percentile(lat, 99) * 1e3), "evals": evals,
                             **_serving_accuracy(done)}
    best = max(v["integrals_per_s"] for k, v in out.items() if k.startswith("rate_") and "early" not in k)
    out["served_vs_plain_integrals_per_s_matched_work"] = best / (n / t_plain)
    out["served_early_stop_vs_plain_integrals_per_s"] = (
        out[f"rate_{int(rates[-1])}_mc_early_stop"]["integrals_per_s"] / (n / t_plain))
    out["cpu_baseline"] = serving_cpu_baseline(n)
    return out


def serving_cpu_baseline(n, budget_s=8.0, max_n=2_000_000):
    """The oracle port on the requests of the stream with N <= max_n, in
    arrival order, until budget_s (Monte Carlo: the same Philox draws;
    VEGAS and Simpson: the numpy restatements)."""
    import numpy as np

    from oracle import grid as OG
    from oracle import integrands as OI
    from oracle import mc as OM
    from oracle import philox as OP
    from oracle import vegas as OV
    from torchquad_gb300.serving import poisson_stream

    t0 = time.perf_counter()
    k = 0
    for _, r in poisson_stream(n, 1e5, seed=2):
        if time.perf_counter() - t0 > budget_s:
            break
        if r.N > max_n:
            continue
        p = r.integrand.params_numpy()
        fn = lambda x, fam=r.integrand.family, p=p: OI.evaluate(fam, p, x)  # noqa: E731
        dt = np.float32
        if r.method == "montecarlo":
            u = OP.uniform(r.seed, 0, 0, r.N * r.dim, dt).reshape(r.N, r.dim)
            OM.integrate(fn, r.dim, r.N, r.domain, u)
        elif r.method == "vegas":
            OV.Vegas().integrate(fn, r.dim, r.N, r.domain, OP.ReplayStream(r.seed), dt=dt, eps_rel=r.eps_rel)
        else:
            OG.integrate(fn, OG.SIMPSON, r.dim, r.N, r.domain, dt=dt)
        k += 1
    t = time.perf_counter() - t0
    return {"integrals_per_s": k / t, "unit": "integrals/s", "cores": cpu_cores_used(), "kind": "port",
            "sample": f"{k} requests of the stream with N <= {max_n}, in arrival order, numpy restatements "
                      "of the reference, one process (the larger requests take minutes each on one core)"}


# ----------------------------------------------------------- CPU (oracle)
def _oracle_one(seed):
    import numpy as np

    from oracle import integrands as OI
    from oracle import philox as OP
    from oracle import vegas as OV

    a = 1.0 / (2.0 * SIGMA * SIGMA)
    c = (1.0 / (SIGMA * math.sqrt(2.0 * math.pi))) ** DIM
    params = np.array([c, 0.0] + [a] * DIM + [0.5] * DIM)
    v = OV.Vegas()
    t0 = time.perf_counter()
    r = v.integrate(lambda x: OI.evaluate(2, params, x), DIM, N_EVALS, [[0.0, 1.0]] * DIM,
                    OP.ReplayStream(seed), dt=np.float32, n_intervals=N_BINS)
    return v.fevals, time.perf_counter() - t0, r


def run_reference(args):
    """CPU arm: the reference algorithm (numpy restatement) on all host cores."""
    ws, rank, _ = _dist_env()
    if rank != 0:
        return 0
    import multiprocessing as mp

    cores = os.cpu_count() or 1
    ctx = mp.get_context("spawn")
    with ctx.Pool(cores) as pool:
        for w in range(args.warmup):
            pool.map(_oracle_one, [1000 + w * cores + i for i in range(cores)])
        times, evals = [], 0
        t_all = time.perf_counter()
        for k in range(args.steps):
            t0 = time.perf_counter()
            res = pool.map(_oracle_one, [k * cores + i for i in range(cores)])
            times.append(time.perf_counter() - t0)
            evals += sum(r[0] for r in res)
        total = time.perf_counter() - t_all
    value = evals / total
    line = {
        "impl": "reference",
        "metric": METRIC,
        "value": value,
        "unit": UNIT,
        "n_gpus": ws,
        "steps": args.steps,
        "warmup": args.warmup,
        "ms_per_step": 1000.0 * total / args.steps,
        "higher_is_better": True,
        "scaling": "weak",
        "vs_baseline": None,
        "dtype": "f32",
        "data": "synthetic",
        "config": CONFIG,
        "cpu_baseline": {
            "value": value,
            "unit": UNIT,
            "cores": cores,
            "kind": "port",
            "sample": f"each step: {cores} full integrations of the workload in parallel processes "
                      "(numpy restatement of the reference, one per host core)",
        },
        "e2e": {"value": value, "unit": UNIT, "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0},
    }
    print(json.dumps(line), flush=True)
    return 0


def cpu_baseline_sample(budget_s=20.0):
    evals, t = 0, 0.0
    n = 0
    while t < budget_s and n < 8:
        e, dt, _ = _oracle_one(500 + n)
        evals += e
        t += dt
        n += 1
    return {
        "value": evals / t,
        "unit": UNIT,
        "cores": 1,
        "kind": "port",
        "sample": f"{n} full integrations of the workload, numpy restatement of the reference, one process",
    }


# --------------------------------------------------------------- clocks
class ClockSampler:
    def __init__(self, path, index):
        self.path, self.index, self.proc = path, index, None

    def __enter__(self):
        q = ("index,clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.active,"
             "clocks_event_reasons.hw_slowdown,clocks_event_reasons.hw_thermal_slowdown,"
             "clocks_event_reasons.sw_thermal_slowdown,clocks_event_reasons.sw_power_cap")
        try:
            self.fh = open(self.path, "w")
            self.proc = subprocess.Popen(
                ["nvidia-smi", f"--id={self.index}", f"--query-gpu={q}", "--format=csv,noheader,nounits",
                 "-lms", "200"], stdout=self.fh, stderr=subprocess.DEVNULL)
        except (OSError, FileNotFoundError):
            self.proc = None
        return self

    def __exit__(self, *exc):
        if self.proc is not None:
            self.proc.terminate()
            try:
                self.proc.wait(timeout=5)
            except subprocess.TimeoutExpired:
                self.proc.kill()
            self.fh.close()

    def summary(self):
        if self.proc is None:
            return {"sm_mhz": None, "sm_max_mhz": None, "reasons": ["nvidia-smi unavailable"]}
        rows = []
        with open(self.path) as fh:
            for line in fh:
                parts = [p.strip() for p in line.split(",")]
                if len(parts) >= 9:
                    rows.append(parts)
        if not rows:
            return {"sm_mhz": None, "sm_max_mhz": None, "reasons": ["no samples"]}
        sm = [float(r[1]) for r in rows if r[1].replace(".", "").isdigit()]
        mx = [float(r[2]) for r in rows if r[2].replace(".", "").isdigit()]
        names = ["hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"]
        reasons = sorted({names[i] for r in rows for i in range(4) if "Active" in r[5 + i] and "Not" not in r[5 + i]})
        return {"sm_mhz": statistics.median(sm) if sm else None, "sm_max_mhz": max(mx) if mx else None,
                "reasons": reasons, "samples": len(rows)}


# --------------------------------------------------------------- GPU arm
def run_gpu(args):
    import torch

    ws, rank, local = _dist_env()
    torch.cuda.set_device(local)
    if ws > 1:
        import torch.distributed as dist

        dist.init_process_group("nccl")
    import torchquad_gb300 as tq
    from torchquad_gb300 import _lib as L
    from torchquad_gb300.integration import vegas as V

    dev = torch.device("cuda", local)
    f = tq.GaussianPeak.normal(DIM, 0.5, SIGMA)
    domain_dev = torch.tensor([[0.0, 1.0]] * DIM, dtype=torch.float32, device=dev)
    flush = torch.empty(256 << 20, dtype=torch.uint8, device=dev)

    def barrier():
        if ws > 1:
            import torch.distributed as dist

            dist.barrier()
        torch.cuda.synchronize()

    def one(seed, domain):
        v = tq.VEGAS()
        r = v.integrate(f, DIM, N=N_EVALS, integration_domain=domain, seed=seed, n_intervals=N_BINS)
        return v, r

    for w in range(args.warmup):
        one(10_000 + w, domain_dev)
    barrier()

    # ---- device-resident inputs
    clocks = ClockSampler(os.environ.get("TQ_CLOCKS_CSV", f"/tmp/tq_clocks_{rank}.csv"), local)
    step_ms, evals, results, errors = [], 0, [], []
    with clocks:
        # keep the GPU under the same load for about a second first, so the
        # 200 ms clock samples cover the load the timed steps run under
        t_soak = time.perf_counter() + 1.0
        k_soak = 0
        while time.perf_counter() < t_soak:
            one(20_000 + k_soak, domain_dev)
            k_soak += 1
        barrier()
        launches0 = L.launches[0]
        v = r = None
        for k in range(args.steps):
            # a user's loop drops the previous integrator before the next
            # (one that keeps it alive gets a second pooled device plan)
            v = r = None
            flush.fill_(k & 0xFF)
            e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            e0.record()
            v, r = one(rank_seed(rank, k), domain_dev)
            e1.record()
            torch.cuda.synchronize()
            step_ms.append(e0.elapsed_time(e1))
            evals += v._nr_of_fevals
            results.append(r.item())
            errors.append(float(v._get_error()))
        barrier()
    launches = L.launches[0] - launches0
    t_local = sum(step_ms) / 1000.0

    # ---- dominant kernel: the same integrations with the captured sequences
    # run as individual launches, CUDA events around every fused sampling
    # launch on the launching (current) stream
    sampler_events, sampler_points = [], []
    other_events = {"update_map": [], "finish": [], "finish_update_map": [], "get_nh": [], "get_nh_split": [],
                    "warmup_fused": []}
    orig_iter = V.VegasDevice.iterate_fused
    originals = {name: getattr(V.VegasDevice, name) for name in other_events}

    def timed_iterate(self, *a, **k):
        if torch.cuda.is_current_stream_capturing():  # a graph being recorded runs nothing
            return orig_iter(self, *a, **k)
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        e0.record()
        orig_iter(self, *a, **k)
        e1.record()
        sampler_events.append((e0, e1))

    def timed(name):
        fn = originals[name]

        def wrapper(self, *a, **k):
            if torch.cuda.is_current_stream_capturing():
                return fn(self, *a, **k)
            e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            e0.record()
            out = fn(self, *a, **k)
            e1.record()
            other_events[name].append((e0, e1))
            return out

        return wrapper

    # a device-side sleep ahead of every block of launches lets the host
    # enqueue the whole block first, so the events time the GPU alone
    orig_block, orig_warm = V._FusedPlan._block_seq, V._FusedPlan._warm_seq

    def slept(fn):
        def wrapper(self):
            if not torch.cuda.is_current_stream_capturing():
                torch.cuda._sleep(4_000_000)
            return fn(self)

        return wrapper

    V._FusedPlan._block_seq, V._FusedPlan._warm_seq = slept(orig_block), slept(orig_warm)
    V.VegasDevice.iterate_fused = timed_iterate
    for name in other_events:
        setattr(V.VegasDevice, name, timed(name))
    V.FORCE_EAGER[0] = True
    try:
        for k in range(args.steps):
            v = None
            flush.fill_(k & 0xFF)
            n0 = len(sampler_events)
            v, _ = one(rank_seed(rank, k), domain_dev)
            torch.cuda.synchronize()
            stats = v._dev.stats[: v.it, 2].cpu()
            sampler_points += [float(stats[j]) for j in range(len(sampler_events) - n0)]
    finally:
        V._FusedPlan._block_seq, V._FusedPlan._warm_seq = orig_block, orig_warm
        V.VegasDevice.iterate_fused = orig_iter
        for name, fn in originals.items():
            setattr(V.VegasDevice, name, fn)
        V.FORCE_EAGER[0] = False
    sampler_ms = [a.elapsed_time(b) for a, b in sampler_events]
    # mean duration per call of each step of an iteration (eager launches,
    # CUDA events on the launching stream)
    step_us = {"iterate_fused": 1e3 * sum(sampler_ms) / max(1, len(sampler_ms))}
    for name, evs in other_events.items():
        if evs:
            step_us[name] = 1e3 * sum(a.elapsed_time(b) for a, b in evs) / len(evs)

    # ---- end to end through the public API with host inputs
    e2e_ms, e2e_evals = [], 0
    # domain bounds, integrand parameters, RNG offset and loop settings travel
    # as the launch arguments of one tq_vegas_begin_run (a tq_vegas_run)
    h2d = ctypes.sizeof(L.VegasRun)
    d2h_per = []
    barrier()
    for k in range(args.steps):
        flush.fill_(k & 0xFF)
        torch.cuda.synchronize()
        t0 = time.perf_counter()
        f_host = tq.GaussianPeak.normal(DIM, 0.5, SIGMA)  # parameters uploaded inside the step
        v = tq.VEGAS()
        r = v.integrate(f_host, DIM, N=N_EVALS, integration_domain=[[0.0, 1.0]] * DIM, seed=rank * 7 + k,
                        n_intervals=N_BINS)
        val = r.item()
        e2e_ms.append((time.perf_counter() - t0) * 1000.0)
        e2e_evals += v._nr_of_fevals
        # one read-back per run (control, flags, RNG offset, statistics rows),
        # then the result
        d2h_per.append(v._dev._rb.numel() * 8 + 4)
        assert math.isfinite(val)
    barrier()

    # ---- FP32 / FP64 FMA peaks (measured in this run)
    peaks = fp_peaks(L, torch)
    fp32_peak = peaks["fp32"]

    # ---- reduce over ranks
    t_max, e2e_t, tot_evals, tot_e2e = reduce_over_ranks(t_local, sum(e2e_ms) / 1000.0, evals, e2e_evals,
                                                         ws, dev)
    if rank != 0:
        if ws > 1:
            import torch.distributed as dist

            dist.destroy_process_group()
        return 0

    # algorithmic FP32 work of one sampled point: d x (stratified y: add,
    # div; map: mul, floor, sub, mul, add; Jacobian mul; domain map mul, add;
    # separable term 4) + outer exp + 3 muls = 16 d + 7
    flops_per_point = 16 * DIM + 7
    pts = sum(sampler_points) / max(1, len(sampler_points))
    avg_ms = sum(sampler_ms) / max(1, len(sampler_ms))
    achieved = flops_per_point * pts / (avg_ms / 1000.0) / 1e12
    line = {
        "metric": METRIC,
        "value": tot_evals / t_max,
        "unit": UNIT,
        "n_gpus": ws,
        "steps": args.steps,
        "warmup": args.warmup,
        "ms_per_step": 1000.0 * t_max / args.steps,
        # rank 0's per-step device times: a single stalled step (the GPU or
        # driver held up for tens of ms) shows here rather than only in the mean
        "step_ms": [round(x, 4) for x in step_ms],
        "step_ms_median": statistics.median(step_ms),
        "higher_is_better": True,
        "scaling": "weak",
        "vs_baseline": None,
        "dtype": "f32",
        "data": "synthetic",
        "config": {**CONFIG, "parallelism": f"replicas x{ws}" if ws > 1 else "single GPU"},
        "e2e": {
            "value": tot_e2e / e2e_t,
            "unit": UNIT,
            "h2d_bytes_per_step": h2d,
            "d2h_bytes_per_step": int(statistics.mean(d2h_per)),
            "ms_per_step": statistics.mean(e2e_ms),
        },
        "roofline": {
            "kernel": "vegas_sample_kernel (fused stratified iteration)",
            "bound": "fp32",
            "achieved": achieved,
            "peak": fp32_peak,
            "unit": "TFLOP/s",
            "frac": achieved / fp32_peak,
            # one ncu capture of the sampler gives the DRAM bytes of a launch;
            # that figure is in the committed profile summary, not measured here
            "traffic": None,
            "peak_source": "FP32 FMA probe kernel measured in this run (MEASURED_PEAKS.json has HBM and bf16 only)",
            "points_per_launch": pts,
            "avg_launch_us": avg_ms * 1000.0,
            "flops_per_point": flops_per_point,
        },
        "accuracy": c2_accuracy(results, errors),
        "iteration_steps_us": step_us,
        "gpu_launches": launches,
        "clocks": clocks.summary(),
        "evals_per_step": tot_evals / (args.steps * ws),
    }
    if not args.no_batched:
        line["grid_cases"] = measure_grid_cases(tq, dev, L, peaks, flush)
        line["batched"] = measure_batched(tq, dev, L, peaks)
        line["vegas_batch"] = measure_vegas_batch(tq, dev)
    if not args.no_serving:
        line["serving"] = measure_serving(tq, dev)
    if not args.no_cpu_baseline:
        line["cpu_baseline"] = cpu_baseline_sample(args.cpu_seconds)
    print(json.dumps(line), flush=True)
    if ws > 1:
        import torch.distributed as dist

        dist.destroy_process_group()
    return 0


def run_case(name):
    """One launch of a named kernel workload after one warm-up launch, for
    profiling a single kernel (ncu -k ... -c 1):
      c1_fused        fused Simpson, dim 3, 101^3 nodes, fp64, exp(x0+x1+x2)
      points_n301     tq_grid_points, Simpson, dim 3, 301^3 nodes, fp64
      wsum_n301       tq_weighted_sum of those 301^3 fp64 values
      c3_fp64         the 4096-integral batch, fp64, one tq_batch_grid launch
      c3_fp32         the same batch in fp32
      c4_batch        1024 differentiation integrals, one tq_batch_grid_adjoint
      c2              one plain VEGAS integration (dim 6, N = 1e7, 50 intervals),
                      its kernels launched eagerly
      vegas_batch     the 1024-integral VEGAS batch of C5's VEGAS share, its
                      phases launched eagerly"""
    import torch

    import torchquad_gb300 as tq
    from torchquad_gb300 import _lib as L
    from torchquad_gb300 import batch as B

    dev = torch.device("cuda", 0)
    lib = L.lib()
    runs = []
    if name == "c1_fused":
        dom = torch.tensor([[0.0, 1.0]] * 3, dtype=torch.float64, device=dev)
        f = tq.ExpSum(3)
        runs = [lambda: tq.Simpson().integrate(f, 3, N=101**3, integration_domain=dom)]
    elif name in ("points_n301", "wsum_n301"):
        dom = torch.tensor([[0.0, 1.0]] * 3, dtype=torch.float64, device=dev)
        tot = 301**3
        pts = torch.empty((tot, 3), dtype=torch.float64, device=dev)
        fv = torch.rand(tot, dtype=torch.float64, device=dev)
        acc = torch.zeros(2, dtype=torch.float64, device=dev)
        ws = torch.zeros(lib.tq_weighted_sum_workspace_size(tot, 1), dtype=torch.uint8, device=dev)
        if name == "points_n301":
            runs = [lambda: L.check(lib.tq_grid_points(L.TQ_F64, L.TQ_RULE_SIMPSON, 3, 301, dom.data_ptr(), None, 0,
                                                       tot, pts.data_ptr(), L.stream_handle()), "pts")]
        else:
            runs = [lambda: L.check(lib.tq_weighted_sum(L.TQ_F64, L.TQ_RULE_SIMPSON, 3, 301, dom.data_ptr(), None, 0,
                                                        tot, fv.data_ptr(), L.TQ_F64, 1, acc.data_ptr(),
                                                        ws.data_ptr(), ws.numel(), L.stream_handle()), "wsum")]
    elif name in ("c3_fp64", "c3_fp32"):
        specs, _ = c3_workload()
        fs = [tq.GaussianPeak(d, a=a.tolist(), u=u.tolist()) for (_, d, _, _, a, u) in specs]
        dt = torch.float64 if name == "c3_fp64" else torch.float32
        bg = B.BatchedGrid(dtype=dt, autotune=False, block=256, strip=16, tile_points=32768)
        plan = bg.plan(fs, [sp[0] for sp in specs], [sp[2] for sp in specs], [sp[3] for sp in specs])
        runs = [lambda: bg.run(plan)]
    elif name == "c4_batch":
        import numpy as np

        rng = np.random.default_rng(4)
        a, us = rng.uniform(-3.0, 3.0, (1024, 4)), rng.uniform(0.0, 1.0, 1024)
        fs = [tq.Oscillatory(4, a=a[i].tolist(), b=float(us[i])) for i in range(1024)]
        bg = B.BatchedGrid(dtype=torch.float64)
        plan = bg.plan(fs, ["gausslegendre"] * 1024, [32**4] * 1024, [[[0.0, 1.0]] * 4] * 1024, tile_points=65536)
        runs = [lambda: bg.adjoint(plan)]
    elif name == "c2":
        from torchquad_gb300.integration import vegas as V

        f = tq.GaussianPeak.normal(DIM, 0.5, SIGMA)
        dom = torch.tensor([[0.0, 1.0]] * DIM, dtype=torch.float32, device=dev)
        V.FORCE_EAGER[0] = True
        runs = [lambda: tq.VEGAS().integrate(f, DIM, N=N_EVALS, integration_domain=dom, seed=0, n_intervals=N_BINS)]
    elif name == "vegas_batch":
        from torchquad_gb300.vegas_batch import VegasBatch

        reqs = vegas_batch_workload(1024)
        vb = VegasBatch([r.integrand for r in reqs], [r.N for r in reqs], dtype=torch.float32)
        runs = [lambda: vb.integrate(domains=[r.domain for r in reqs], seeds=[r.seed for r in reqs],
                                     eps_rel=[r.eps_rel for r in reqs])]
        os.environ["TORCHQUAD_GB300_CUDA_GRAPHS"] = "0"  # eager phases: each launch is seen
    else:
        raise SystemExit(f"unknown case {name}")
    for fn in runs * 2:  # warm-up launch, then the profiled one
        fn()
    torch.cuda.synchronize()
    print(json.dumps({"case": name, "ok": True}))
    return 0


def main():
    p = argparse.ArgumentParser()
    p.add_argument("--gpus", type=int, default=1)
    p.add_argument("--steps", type=int, default=10)
    p.add_argument("--warmup", type=int, default=3)
    p.add_argument("--impl", default="ours", choices=["ours", "reference"])
    p.add_argument("--no-cpu-baseline", action="store_true")
    p.add_argument("--no-batched", action="store_true", help="skip the batched-vs-plain measurement")
    p.add_argument("--no-serving", action="store_true", help="skip the serving measurement")
    p.add_argument("--cpu-seconds", type=float, default=20.0)
    p.add_argument("--case", default=None, help="run one named kernel workload twice (for ncu), see run_case")
    args = p.parse_args()
    if args.case:
        from __graft_entry__ import build

        build()
        return run_case(args.case)
    if args.warmup < 3 and args.impl == "ours":
        args.warmup = 3
    if args.impl == "reference":
        return run_reference(args)
    from __graft_entry__ import build

    build()
    return run_gpu(args)


if __name__ == "__main__":
    sys.exit(main())
