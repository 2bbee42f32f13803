"""Performance cases: the integrations a user of the package runs, through its
public entry points, over the sizes of the benchmark, the tests and the
tutorial of the reference.

    listed()             the fixed cases
    draw(rng)            one more case of the same ranges
    prepare(case, seed)  inputs and kept plans of a case, on the GPU
    run(state)           one pass; returns its outputs
    work(case)           bytes and operations one pass cannot do without
    exact(case, seed)    the same outputs in 64 bits by plain torch

The built-in integrands (``torchquad_gb300.integrands``) are functions of a
separable sum, so a tensor-product rule needs every dimension's nodes once:
``work`` counts those, not the nodes of the product grid.
"""
import functools
import math
import warnings

import numpy as np
import torch

import torchquad_gb300 as tq
from torchquad_gb300.batch import BatchedGrid
from torchquad_gb300.vegas_batch import VegasBatch

RULES = {"trapezoid": tq.Trapezoid, "simpson": tq.Simpson, "boole": tq.Boole, "gausslegendre": tq.GaussLegendre}
DTYPES = {"fp32": torch.float32, "fp64": torch.float64}
FAMILIES = ("exp_sum", "gaussian", "oscillatory", "sum_sin")

# The integrators announce that a later version returns array-like results.
warnings.filterwarnings("ignore", message="DEPRECATION WARNING")


def listed():
    return [
        # the smallest call: a 1-D integral of a torch callable, where launches
        # and host work are everything
        {"name": "callable_d1_small", "kind": "callable", "rule": "trapezoid", "dim": 1, "n": 1001, "dtype": "fp32"},
        # a whole call on an arbitrary torch callable with vector values: the
        # reference's "vectorised integrand" use, 200 parameter values at once
        {"name": "callable_d1_vector200", "kind": "vector", "rule": "simpson", "dim": 1, "n": 10001, "values": 200,
         "dtype": "fp32"},
        # the staged API on a large grid: the rule applied to values the user
        # has computed on calculate_grid's points
        {"name": "result_d3_n301", "kind": "result", "rule": "boole", "dim": 3, "n": 301, "dtype": "fp64"},
        # the plain grid benchmark: exp(x0+x1+x2) on 101^3 nodes in fp64
        {"name": "builtin_d3_n101", "kind": "builtin", "rule": "simpson", "dim": 3, "n": 101, "family": "exp_sum",
         "dtype": "fp64"},
        # the tutorial's 5-D sum of sines on 37^5 nodes in fp32
        {"name": "builtin_d5_n37", "kind": "builtin", "rule": "simpson", "dim": 5, "n": 37, "family": "sum_sin",
         "dtype": "fp32"},
        # the differentiation benchmark: value and gradients of a 32^4
        # Gauss-Legendre integral, forward and backward, with fresh parameters
        # as an optimiser's step has them
        {"name": "gradient_d4_n32", "kind": "gradient", "rule": "gausslegendre", "dim": 4, "n": 32,
         "family": "oscillatory", "dtype": "fp64"},
        # Monte Carlo of a built-in integrand, drawn inside the kernel
        {"name": "mc_builtin_d6_1e7", "kind": "mc", "dim": 6, "N": 10_000_000, "family": "gaussian",
         "callable": False, "dtype": "fp32"},
        # Monte Carlo of a torch callable: points, values, mean
        {"name": "mc_callable_d3_1e6", "kind": "mc", "dim": 3, "N": 1_000_000, "family": "gaussian",
         "callable": True, "dtype": "fp64"},
        # the headline: plain VEGAS, dim 6, N = 1e7, 50 map intervals, fp32
        {"name": "vegas_d6_1e7", "kind": "vegas", "dim": 6, "N": 10_000_000, "intervals": 50, "dtype": "fp32"},
        # many resident VEGAS integrals advanced together, as a server runs
        # them: dims 1 to 10, N from 1e4 to 2.56e5
        {"name": "vegas_batch_256", "kind": "vegas_batch", "count": 256, "dtype": "fp32"},
        # many independent integrals of mixed rule, dimension and size in one
        # packed batch that the program keeps
        {"name": "batch_4096", "kind": "batch", "count": 4096, "dtype": "fp64"},
        # values and gradients of many packed 32^4 integrals
        {"name": "batch_gradient_1024", "kind": "batch_gradient", "count": 1024, "dim": 4, "n": 32,
         "family": "oscillatory", "dtype": "fp64"},
    ]


# ------------------------------------------------------------------ drawing
def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _valid_n(rule, n):
    """n as the rule takes it (Simpson odd, Boole one more than a multiple of four)."""
    if rule == "simpson":
        return max(3, n - 1 + n % 2)
    if rule == "boole":
        return max(5, n - (n - 1) % 4)
    return max(2, n)


def draw(rng):
    kind = rng.choice(["callable", "vector", "result", "builtin", "gradient", "mc", "vegas", "vegas_batch", "batch",
                       "batch_gradient"])
    dtype = rng.choice(["fp32", "fp64"])
    rule = rng.choice(list(RULES))
    case = {"kind": kind, "dtype": dtype}
    if kind in ("callable", "result"):
        dim = rng.randint(1, 4)
        total = _log_int(rng, 300, 2_000_000 if kind == "callable" else 27_000_000)
        n = int(total ** (1.0 / dim) + 1e-8)
        n = min(n, 256) if rule == "gausslegendre" else n
        case.update(rule=rule, dim=dim, n=_valid_n(rule, n))
    elif kind == "vector":
        dim = rng.randint(1, 2)
        n = int(_log_int(rng, 300, 20_000) ** (1.0 / dim) + 1e-8)
        n = min(n, 256) if rule == "gausslegendre" else n
        case.update(rule=rule, dim=dim, n=_valid_n(rule, n), values=_log_int(rng, 2, 256))
    elif kind == "builtin":
        dim = rng.randint(1, 6)
        n = int(_log_int(rng, 1000, 60_000_000 if dim > 1 else 2_000_000) ** (1.0 / dim) + 1e-8)
        n = min(n, 256) if rule == "gausslegendre" else n
        case.update(rule=rule, dim=dim, n=_valid_n(rule, n), family=rng.choice(FAMILIES))
    elif kind == "gradient":
        dim = rng.randint(1, 5)
        n = min(200, int(_log_int(rng, 100, 2_000_000) ** (1.0 / dim) + 1e-8))
        case.update(rule=rule, dim=dim, n=_valid_n(rule, n), family=rng.choice(FAMILIES))
    elif kind == "mc":
        on_points = rng.random() < 0.4
        case.update(dim=rng.randint(1, 10), N=_log_int(rng, 10_000, 3_000_000 if on_points else 30_000_000),
                    family=rng.choice(FAMILIES), callable=on_points)
    elif kind == "vegas":
        case.update(dim=rng.randint(1, 8), N=_log_int(rng, 10_000, 10_000_000 if dtype == "fp32" else 2_000_000),
                    intervals=rng.choice([0, 50]))
    elif kind == "vegas_batch":
        case.update(count=_log_int(rng, 4, 256))
    elif kind == "batch":
        case.update(count=_log_int(rng, 16, 4096))
    else:
        dim = rng.randint(2, 4)
        case.update(count=_log_int(rng, 8, 1024), dim=dim, n=rng.randint(8, (0, 0, 200, 60, 32)[dim]),
                    family=rng.choice(FAMILIES))
    return case


# ------------------------------------------------------------------- inputs
def _family_params(rng, family, dim):
    """Parameter values (a, u, b, c) as the benchmark's integrals have them."""
    if family == "gaussian":
        return rng.uniform(0.5, 5.0, dim), rng.uniform(0.0, 1.0, dim), 0.0, rng.uniform(0.5, 2.0)
    if family == "oscillatory":
        return rng.uniform(-3.0, 3.0, dim), np.zeros(dim), rng.uniform(0.0, 1.0), rng.uniform(0.5, 2.0)
    if family == "exp_sum":
        return rng.uniform(-1.5, 1.5, dim), np.zeros(dim), rng.uniform(-0.5, 0.5), rng.uniform(0.5, 2.0)
    return rng.uniform(0.5, 2.0, dim), np.zeros(dim), 0.0, rng.uniform(0.5, 2.0)


def _builtin(family, dim, a, u, b, c):
    if family == "gaussian":
        return tq.GaussianPeak(dim, a=a, u=u, c=c)
    if family == "oscillatory":
        return tq.Oscillatory(dim, a=a, b=b, c=c)
    if family == "exp_sum":
        return tq.ExpSum(dim, a=a, b=b, c=c)
    return tq.SumSin(dim, a=a, c=c)


def _domain(rng, dim):
    lo = rng.uniform(-1.0, 0.0, dim)
    return np.stack([lo, lo + rng.uniform(0.5, 2.0, dim)], axis=1)


def _numbers(case, seed):
    """Everything drawn for a case, as numpy arrays, from the seed alone."""
    rng = np.random.default_rng([seed, 7919])
    kind = case["kind"]
    if kind in ("callable", "result"):
        return {"a": rng.uniform(0.5, 5.0, case["dim"]), "u": rng.uniform(0.0, 1.0, case["dim"]),
                "domain": _domain(rng, case["dim"])}
    if kind == "vector":
        return {"p": rng.uniform(0.5, 3.0, (case["dim"], case["values"])), "domain": _domain(rng, case["dim"])}
    if kind in ("builtin", "gradient", "mc"):
        a, u, b, c = _family_params(rng, case["family"], case["dim"])
        return {"a": a, "u": u, "b": b, "c": c, "domain": _domain(rng, case["dim"]),
                "seed": int(rng.integers(1, 1 << 40))}
    if kind == "vegas":
        return {"u": float(rng.uniform(0.45, 0.55)), "seed": int(rng.integers(1, 1 << 40))}
    if kind == "vegas_batch":
        items = []
        for _ in range(case["count"]):
            dim = int(rng.integers(1, 11))
            family = ("gaussian", "oscillatory")[int(rng.integers(0, 2))]
            a, u, b, c = _family_params(rng, family, dim)
            items.append({"family": family, "dim": dim, "N": int(10 ** rng.uniform(4.0, 5.4)), "a": a, "u": u, "b": b,
                          "c": c, "domain": _domain(rng, dim), "seed": int(rng.integers(1, 1 << 40)),
                          "eps": float(10 ** rng.uniform(-5.0, -3.0))})
        return {"items": items}
    if kind == "batch":
        items = []
        for _ in range(case["count"]):
            dim = int(rng.integers(1, 5))
            rule = ("trapezoid", "simpson", "boole", "gausslegendre")[int(rng.integers(0, 4))]
            N = int(10 ** rng.uniform(3.0, 6.0))
            if rule == "gausslegendre":
                N = min(N, 256 ** dim)
            a, u, _, c = _family_params(rng, "gaussian", dim)
            items.append({"family": "gaussian", "dim": dim, "rule": rule, "N": N, "a": a, "u": u, "b": 0.0, "c": c,
                          "domain": _domain(rng, dim)})
        return {"items": items}
    items = []
    for _ in range(case["count"]):
        a, u, b, c = _family_params(rng, case["family"], case["dim"])
        items.append({"family": case["family"], "dim": case["dim"], "rule": "gausslegendre",
                      "N": case["n"] ** case["dim"], "a": a, "u": u, "b": b, "c": c,
                      "domain": _domain(rng, case["dim"])})
    return {"items": items}


def _on(device, dtype, v):
    return torch.tensor(v, dtype=dtype, device=device)


# the torch callables a user passes; p holds their constants
def _peak(x, a, u):
    return torch.exp(-(a * (x - u) ** 2).sum(dim=1))


def _waves(x, p):
    return torch.sqrt(torch.cos(torch.sin(x @ p)) + 1.0)


def _grid_values(case, v, dev):
    """Values of a smooth integrand on the case's grid, last dimension fastest."""
    dtype = torch.float64 if case["rule"] == "gausslegendre" else DTYPES[case["dtype"]]
    dom, a, u = (_on(dev, torch.float64, v[k]) for k in ("domain", "a", "u"))
    s = torch.zeros(1, dtype=torch.float64, device=dev)
    for k in range(case["dim"]):
        x = _nodes_weights(case["rule"], case["n"], dom[k, 0], dom[k, 1])[0]
        s = (s[:, None] + (a[k] * (x - u[k]) ** 2)[None, :]).reshape(-1)
    return torch.exp(-s).to(dtype)


def _item_fn(it):
    return _builtin(it["family"], it["dim"], it["a"].tolist(), it["u"].tolist(), float(it["b"]), float(it["c"]))


def prepare(case, seed):
    dev = torch.device("cuda", torch.cuda.current_device())
    dtype = DTYPES[case["dtype"]]
    v = _numbers(case, seed)
    kind = case["kind"]
    s = {"case": case}
    if kind in ("callable", "vector", "result"):
        # a Gauss-Legendre grid has fp64 points whatever the domain's type
        pt = torch.float64 if case["rule"] == "gausslegendre" else dtype
        if kind == "vector":
            p = _on(dev, pt, v["p"])
            s["fn"] = lambda x: _waves(x, p)
        else:
            a, u = _on(dev, pt, v["a"]), _on(dev, pt, v["u"])
            s["fn"] = lambda x: _peak(x, a, u)
        s["N"] = case["n"] ** case["dim"]
        # the smallest calls pass a list, as the reference's examples do
        s["domain"] = v["domain"].tolist() if kind == "callable" and dtype == torch.get_default_dtype() else \
            _on(dev, dtype, v["domain"])
        if kind == "result":
            s["integrator"] = RULES[case["rule"]]()
            s["hs"] = (s["domain"][:, 1] - s["domain"][:, 0]) / (case["n"] - 1)
            s["values"] = _grid_values(case, v, dev)
        return s
    if kind in ("builtin", "mc"):
        fam, b, c = case["family"], float(v["b"]), float(v["c"])
        if case.get("callable"):
            a, u = _on(dev, dtype, v["a"]), _on(dev, dtype, v["u"])
            s["fn"] = lambda x: _family_value(x, fam, a, u, b, c)
        else:
            s["fn"] = _builtin(fam, case["dim"], v["a"].tolist(), v["u"].tolist(), b, c)
        s["domain"] = _on(dev, dtype, v["domain"])
        s["N"] = case["N"] if kind == "mc" else case["n"] ** case["dim"]
        s["seed"] = v["seed"]
        return s
    if kind == "gradient":
        s["domain"] = _on(dev, dtype, v["domain"]).requires_grad_()
        s["a"] = _on(dev, torch.float64, v["a"]).requires_grad_()
        s["u"] = _on(dev, torch.float64, v["u"]).requires_grad_(case["family"] == "gaussian")
        s["b"] = _on(dev, torch.float64, v["b"]).requires_grad_(case["family"] in ("oscillatory", "exp_sum"))
        s["c"] = float(v["c"])
        s["N"] = case["n"] ** case["dim"]
        return s
    if kind == "vegas":
        s["fn"] = tq.GaussianPeak.normal(case["dim"], v["u"], 0.05)
        s["domain"] = [[0.0, 1.0]] * case["dim"] if dtype == torch.get_default_dtype() else \
            _on(dev, dtype, [[0.0, 1.0]] * case["dim"])
        s["seed"] = v["seed"]
        return s
    items = v["items"]
    fns = [_item_fn(it) for it in items]
    if kind == "vegas_batch":
        s["batch"] = VegasBatch(fns, [it["N"] for it in items], dtype=dtype)
        s["domains"] = [it["domain"].tolist() for it in items]
        s["seeds"] = [it["seed"] for it in items]
        s["eps"] = [it["eps"] for it in items]
        return s
    s["grid"] = BatchedGrid(dtype=dtype, autotune=False)
    s["plan"] = s["grid"].plan(fns, [it["rule"] for it in items], [it["N"] for it in items],
                               [it["domain"] for it in items])
    return s


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind in ("callable", "vector", "builtin"):
        return RULES[case["rule"]]().integrate(s["fn"], case["dim"], N=s["N"], integration_domain=s["domain"])
    if kind == "result":
        return s["integrator"].calculate_result(s["values"], case["dim"], case["n"], s["hs"], s["domain"])
    if kind == "mc":
        return tq.MonteCarlo().integrate(s["fn"], case["dim"], N=s["N"], integration_domain=s["domain"],
                                         seed=s["seed"])
    if kind == "gradient":
        wrt = {"domain": s["domain"], "a": s["a"]}
        if s["u"].requires_grad:
            wrt["u"] = s["u"]
        if s["b"].requires_grad:
            wrt["b"] = s["b"]
        f = _builtin(case["family"], case["dim"], s["a"], s["u"], s["b"], s["c"])
        value = RULES[case["rule"]]().integrate(f, case["dim"], N=s["N"], integration_domain=s["domain"])
        grads = torch.autograd.grad(value, list(wrt.values()))
        return {"value": value.detach(), **dict(zip(wrt, grads))}
    if kind == "vegas":
        return tq.VEGAS().integrate(s["fn"], case["dim"], N=case["N"], integration_domain=s["domain"], seed=s["seed"],
                                    n_intervals=case["intervals"] or None)
    if kind == "vegas_batch":
        return s["batch"].integrate(domains=s["domains"], seeds=s["seeds"], eps_rel=s["eps"])
    if kind == "batch":
        return s["grid"].run(s["plan"])
    values, g_domain, g_params = s["grid"].adjoint(s["plan"])
    return {"values": values, "domains": g_domain, "params": g_params}


# --------------------------------------------------------------- the floors
# operations of one node's term of a separable family, an elementary function
# counted as 20
_TERM = 24


def work(case):
    size = 4 if case["dtype"] == "fp32" else 8
    kind = case["kind"]
    d = case.get("dim", 0)
    if kind in ("callable", "vector"):
        # points written for the callable and read by it, values written and
        # read once; the callable's own arithmetic
        size = 8 if case["rule"] == "gausslegendre" else size
        nodes, vals = case["n"] ** d, case.get("values", 1)
        return {"bytes": nodes * size * 2 * (d + vals), "flops": nodes * vals * (2 * d + 22)}
    if kind == "result":
        size = 8 if case["rule"] == "gausslegendre" else size
        return {"bytes": case["n"] ** d * size, "flops": 2 * case["n"] ** d}
    if kind == "builtin":
        return {"bytes": 16 * d + 8, "flops": d * case["n"] * _TERM}
    if kind == "gradient":
        return {"bytes": 48 * d, "flops": d * case["n"] * 2 * _TERM}
    if kind == "mc":
        # every draw's ten Philox rounds (40 integer operations per four
        # words), its map and its term; a callable's points and values pass
        # through memory
        words = 1 if size == 4 else 2
        return {"bytes": case["N"] * size * 2 * (d + 1) if case["callable"] else 16 * d,
                "flops": case["N"] * (d * (10 * words + 6) + 20)}
    if kind == "vegas":
        return {"bytes": 64 * d, "flops": int(0.6 * case["N"]) * (16 * d + 7)}
    if kind == "vegas_batch":
        return {"bytes": 400 * case["count"], "flops": case["count"] * 60_000 * (16 * 5 + 7)}
    if kind == "batch":
        # a quarter of the integrals has one dimension, of 1e3 to 1e6 nodes
        # (a quarter of those Gauss-Legendre, at most 256)
        return {"bytes": 160 * case["count"], "flops": int(case["count"] * 27_000 * 4)}
    return {"bytes": 160 * case["count"], "flops": case["count"] * d * case["n"] * 2 * _TERM}


# ------------------------------------------------- the same in 64 bits, plainly
_leggauss = functools.lru_cache(maxsize=None)(np.polynomial.legendre.leggauss)


def _nodes_weights(rule, n, lo, hi):
    """1-D nodes and weights of a composite rule on [lo, hi], fp64 tensors
    (differentiable in lo and hi)."""
    if rule == "gausslegendre":
        r, w = _leggauss(n)
        r, w = torch.from_numpy(r).to(lo.device), torch.from_numpy(w).to(lo.device)
        return 0.5 * (hi - lo) * r + 0.5 * (hi + lo), 0.5 * (hi - lo) * w
    i = torch.arange(n, device=lo.device)
    end = (i == 0) | (i == n - 1)
    if rule == "trapezoid":
        num, den = torch.where(end, 1.0, 2.0).double(), 2.0
    elif rule == "simpson":
        num, den = torch.where(end, 1.0, torch.where(i % 2 == 1, 4.0, 2.0)).double(), 3.0
    else:
        inner = torch.where(i % 2 == 1, 32.0, torch.where(i % 4 == 2, 12.0, 14.0))
        num, den = torch.where(end, 7.0, inner).double(), 22.5
    t = i.double() / (n - 1)
    return lo + (hi - lo) * t, num * ((hi - lo) / (n - 1) / den)


def _terms(family, x, a, u):
    if family == "gaussian":
        return a * (x - u) ** 2
    return torch.sin(a * x) if family == "sum_sin" else a * x


def _outer(family, s, b, c):
    if family == "gaussian":
        return c * torch.exp(-s)
    if family == "exp_sum":
        return c * torch.exp(s + b)
    if family == "oscillatory":
        return c * torch.cos(2.0 * math.pi * b + s)
    return c * s


def _family_value(x, family, a, u, b, c):
    return _outer(family, _terms(family, x, a, u).sum(dim=1), b, c)


def _separable(family, rule, n, dom, a, u, b, c):
    """The tensor-product sum of a built-in integrand: every node of the grid,
    one slab of the first dimension at a time where the grid is large."""
    dim = dom.shape[0]
    xs, ws = zip(*[_nodes_weights(rule, n, dom[k, 0], dom[k, 1]) for k in range(dim)])
    s, w = torch.zeros(1, dtype=torch.float64, device=dom.device), torch.ones(1, dtype=torch.float64, device=dom.device)
    for k in range(1, dim):
        t = _terms(family, xs[k], a[k], u[k])
        s = (s[:, None] + t[None, :]).reshape(-1)
        w = (w[:, None] * ws[k][None, :]).reshape(-1)
    t0 = _terms(family, xs[0], a[0], u[0])
    step = max(1, (1 << 24) // s.numel())
    parts = []
    for i in range(0, n, step):
        v = _outer(family, t0[i:i + step, None] + s[None, :], b, c)
        parts.append(((v * w[None, :]).sum(dim=1) * ws[0][i:i + step]).sum())
    return torch.stack(parts).sum()


def _philox(block, seed):
    """Philox4x32-10 words of counters `block` under key `seed`, as int64."""
    m = 0xFFFFFFFF
    c = [block & m, (block >> 32) & m, torch.zeros_like(block), torch.zeros_like(block)]
    k0, k1 = seed & m, (seed >> 32) & m
    for _ in range(10):
        p0, p1 = c[0] * 0xD2511F53, c[2] * 0xCD9E8D57
        c = [((p1 >> 32) & m) ^ c[1] ^ k0, p1 & m, ((p0 >> 32) & m) ^ c[3] ^ k1, p0 & m]
        k0, k1 = (k0 + 0x9E3779B9) & m, (k1 + 0xBB67AE85) & m
    return c


def _uniform(first, count, seed, dtype, dev):
    """Elements first .. first + count of the stream (first a multiple of 4)."""
    per = 4 if dtype == torch.float32 else 2
    b = torch.arange(first // per, (first + count + per - 1) // per, dtype=torch.int64, device=dev)
    w = _philox(b, seed)
    if per == 4:
        u = torch.stack([(x >> 8).double() * 2.0 ** -24 for x in w], dim=1)
    else:
        u = torch.stack([((w[2 * i] >> 11) | (w[2 * i + 1] << 21)).double() * 2.0 ** -53 for i in (0, 1)], dim=1)
    return u.reshape(-1)[:count]


def exact(case, seed):
    dev = torch.device("cuda", torch.cuda.current_device())
    dtype = DTYPES[case["dtype"]]
    v = _numbers(case, seed)
    kind = case["kind"]
    f64 = lambda x: torch.tensor(x, dtype=torch.float64, device=dev)  # noqa: E731
    rounded = lambda x, t=dtype: torch.tensor(x, dtype=t).to(dev, torch.float64)  # noqa: E731
    if kind in ("callable", "vector", "result"):
        dom, n, dim = rounded(v["domain"]), case["n"], case["dim"]
        pt = torch.float64 if case["rule"] == "gausslegendre" else dtype
        xs, ws = zip(*[_nodes_weights(case["rule"], n, dom[k, 0], dom[k, 1]) for k in range(dim)])
        if kind == "vector":
            x = torch.stack([g.reshape(-1) for g in torch.meshgrid(*xs, indexing="ij")], dim=1)
            w = math.prod(torch.meshgrid(*ws, indexing="ij")).reshape(-1)
            return (_waves(x, rounded(v["p"], pt)) * w[:, None]).sum(dim=0)
        a, u = rounded(v["a"], pt), rounded(v["u"], pt)
        if kind == "result":
            # the values the rule is applied to are the case's input
            values = _grid_values(case, v, dev).double().reshape([n] * dim)
            for k in reversed(range(dim)):
                values = (values * ws[k]).sum(dim=-1)
            return values
        return _separable("gaussian", case["rule"], n, dom, a, u, 0.0, 1.0)
    if kind == "builtin":
        return _separable(case["family"], case["rule"], case["n"], rounded(v["domain"]), f64(v["a"]), f64(v["u"]),
                          float(v["b"]), float(v["c"]))
    if kind == "mc":
        dom = rounded(v["domain"])
        pt = dtype if case["callable"] else torch.float64
        a, u = rounded(v["a"], pt), rounded(v["u"], pt)
        dim, N = case["dim"], case["N"]
        step, parts = 1 << 20, []
        for i in range(0, N, step):
            k = min(step, N - i)
            x = _uniform(i * dim, k * dim, v["seed"], dtype, dev).reshape(k, dim) * (dom[:, 1] - dom[:, 0]) + dom[:, 0]
            parts.append(_family_value(x, case["family"], a, u, float(v["b"]), float(v["c"])).sum())
        return torch.stack(parts).sum() * torch.prod(dom[:, 1] - dom[:, 0]) / N
    if kind == "gradient":
        dom = rounded(v["domain"]).requires_grad_()
        p = {"domain": dom, "a": f64(v["a"]).requires_grad_()}
        u, b = f64(v["u"]), f64(v["b"])
        if case["family"] == "gaussian":
            p["u"] = u.requires_grad_()
        if case["family"] in ("oscillatory", "exp_sum"):
            p["b"] = b.requires_grad_()
        value = _separable(case["family"], case["rule"], case["n"], dom, p["a"], u, b, float(v["c"]))
        return {"value": value.detach(), **dict(zip(p, torch.autograd.grad(value, list(p.values()))))}
    if kind in ("vegas", "vegas_batch"):
        return None  # an adaptive estimate: its draws and maps depend on every rounding before them
    if kind == "batch":
        return torch.stack([
            _separable("gaussian", it["rule"], _points(it["rule"], it["dim"], it["N"]), rounded(it["domain"]),
                       f64(it["a"]), f64(it["u"]), 0.0, float(it["c"])) for it in v["items"]])
    if case["count"] * case["n"] ** case["dim"] > 1 << 31:
        return None  # every node of every grid through autograd takes too long
    values, g_dom, g_par = [], [], []
    for it in v["items"]:
        dom = rounded(it["domain"]).requires_grad_()
        a, u, b, c = (f64(it[k]).requires_grad_() for k in ("a", "u", "b", "c"))
        value = _separable(it["family"], it["rule"], case["n"], dom, a, u, b, c)
        g = torch.autograd.grad(value, [dom, c, b, a, u], allow_unused=True)
        g = [torch.zeros_like(t) if x is None else x for x, t in zip(g, (dom, c, b, a, u))]
        values.append(value.detach())
        g_dom.append(g[0].reshape(-1))
        g_par.append(torch.cat([g[1].reshape(1), g[2].reshape(1), g[3], g[4]]))
    return {"values": torch.stack(values), "domains": torch.cat(g_dom), "params": torch.cat(g_par)}


def _points(rule, dim, N):
    """Points per dimension after the rule's adjustment of N."""
    n = int(N ** (1.0 / dim) + 1e-8)
    if rule == "simpson":
        return 3 if n < 3 else n - 1 + n % 2
    if rule == "boole":
        return 5 if n < 5 else n - (n - 1) % 4
    return n
