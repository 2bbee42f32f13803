"""GPU: built-in integrands on tensor-product grids by 1-D sums per dimension
(sum factorisation) against the numpy oracle, which evaluates every node of
the grid; and integrals whose factors would leave the floating range, which
the node-by-node path keeps."""
import warnings

import numpy as np
import pytest
import torch

import torchquad_gb300 as tq
from oracle import grid as OG
from oracle import integrands as OI

pytestmark = pytest.mark.gpu

RULES = {"trapezoid": (tq.Trapezoid, OG.TRAPEZOID), "simpson": (tq.Simpson, OG.SIMPSON),
         "boole": (tq.Boole, OG.BOOLE), "gausslegendre": (tq.GaussLegendre, OG.GAUSS)}


def family(name, dim):
    k = np.arange(dim)
    a = [float(x) for x in 0.4 + 0.35 * k]
    return {"exp": tq.ExpSum(dim, a=[(-1.0) ** i * v for i, v in enumerate(a)], b=-0.3, c=1.7),
            "gauss": tq.GaussianPeak(dim, a=[3.0 * v for v in a], u=[float(x) for x in 0.2 + 0.1 * k], c=-0.6),
            "osc": tq.Oscillatory(dim, a=[2.0 * v for v in a], b=0.37, c=2.5),
            "sumsin": tq.SumSin(dim, a=[1.5 * v for v in a], c=0.8)}[name]


def domain(dim):
    return [[-0.5 + 0.1 * k, 0.9 + 0.05 * k] for k in range(dim)]


def valid_n(rule, n):
    return {"simpson": max(3, n - 1 + n % 2), "boole": max(5, n - (n - 1) % 4)}.get(rule, n)


def oracle(f, rid, dim, N, dom, dt):
    """(value, sum of |w f|): the integrand in fp64 on the working type's nodes."""
    ev = lambda x: OI.evaluate(f.family, f.params_numpy(), x.astype(np.float64))  # noqa: E731
    return (float(OG.integrate(ev, rid, dim, N, np.asarray(dom), dt)),
            float(OG.integrate(lambda x: np.abs(ev(x)), rid, dim, N, np.asarray(dom), dt)))


def integrate(rule, f, dim, N, dom, dtype, cuda):
    with warnings.catch_warnings():
        warnings.simplefilter("ignore")
        return RULES[rule][0]().integrate(f, dim, N=N, integration_domain=torch.tensor(dom, dtype=dtype, device=cuda))


# nodes per dimension around a warp's 32 lanes, one and several units, one
# CTA and several, rows up to and beyond the one-dimensional limit
SIZES = [(1, 5), (1, 33), (1, 1001), (1, 4093), (1, 4097), (2, 3), (2, 31), (2, 33), (2, 129), (2, 1101), (3, 17),
         (3, 65), (4, 9), (5, 13), (8, 5), (12, 3)]


@pytest.mark.parametrize("dtype", [torch.float64, torch.float32])
@pytest.mark.parametrize("fam", ["exp", "gauss", "osc", "sumsin"])
@pytest.mark.parametrize("rule", list(RULES))
def test_sizes_match_oracle(rule, fam, dtype, cuda):
    """Within the grid rules' bounds, 1e-12 (fp64) and 1e-6 (fp32) of the
    sum of the terms' magnitudes."""
    for dim, n in SIZES:
        if rule == "boole" and n ** dim < 5 ** dim:
            continue
        if rule == "gausslegendre":
            n = min(n, 200)
        n = valid_n(rule, n)
        N = n ** dim
        f = family(fam, dim)
        dom = domain(dim)
        got = integrate(rule, f, dim, N, dom, dtype, cuda).item()
        f64 = dtype == torch.float64
        want, mag = oracle(f, RULES[rule][1], dim, N, dom, np.float64 if f64 else np.float32)
        assert abs(got - want) <= (1e-12 if f64 else 1e-6) * mag, (dim, n, got, want)


REFUSED = [
    ("exponents beyond 300", tq.ExpSum(2, a=[400.0, -380.0], b=-5.0), [[0.0, 1.0], [0.0, 1.0]]),
    ("peak between coarse nodes", tq.GaussianPeak(2, a=[3.0e6, 2.0], u=[0.513, 0.4]), [[0.0, 1.0], [0.0, 1.0]]),
    ("convex exponent", tq.GaussianPeak(2, a=[-0.5, 1.0], u=[0.2, 0.3]), [[0.0, 1.0], [-1.0, 1.0]]),
    ("zero factor", tq.ExpSum(2, a=[1.0, 2.0], c=0.0), [[0.0, 1.0], [0.0, 1.0]]),
    ("large factor", tq.ExpSum(2, a=[-1.0, 2.0], c=1e70), [[0.0, 1.0], [0.0, 1.0]]),
    ("tiny domain", tq.SumSin(2, a=[1.0, 2.0]), [[0.0, 1e-32], [0.5, 1.0]]),
    ("fast oscillation", tq.Oscillatory(2, a=[1.2e6, 1.0], b=0.1), [[0.0, 1.0], [0.0, 1.0]]),
]


@pytest.mark.parametrize("case", REFUSED, ids=lambda c: c[0])
@pytest.mark.parametrize("rule", ["simpson", "gausslegendre"])
def test_other_ranges_keep_the_node_path(case, rule, cuda):
    _, f, dom = case
    n = 41
    got = integrate(rule, f, 2, n * n, dom, torch.float64, cuda).item()
    want, mag = oracle(f, RULES[rule][1], 2, n * n, dom, np.float64)
    # the angle a x of the fast oscillation is rounded to 2^-53 * 1.2e6
    tol = 1e-9 if f.family == OI.OSCILLATORY else 1e-12
    assert abs(got - want) <= tol * mag + 1e-300, (got, want)


def test_fp32_overflow_stays_an_overflow(cuda):
    """e^89 is infinite in fp32 node by node, although the integral's factors are not."""
    f = tq.ExpSum(2, a=[60.0, 60.0])
    got = integrate("simpson", f, 2, 41 * 41, [[0.0, 1.0], [0.0, 1.0]], torch.float32, cuda)
    assert not torch.isfinite(got)


def _assert_gradients(got, want, tol, what):
    """(value, d domain, d params): each within tol of the largest of its kind."""
    for g, w, kind in zip(got, want, ("value", "domain", "params")):
        g, w = np.asarray(g, dtype=np.float64).reshape(-1), np.asarray(w, dtype=np.float64).reshape(-1)
        scale = max(np.abs(w).max(), abs(float(want[0])))
        assert np.all(np.abs(g - w) <= tol * scale), (what, kind, g, w)


@pytest.mark.parametrize("dtype", [torch.float64, torch.float32])
@pytest.mark.parametrize("fam", ["exp", "gauss", "osc", "sumsin"])
def test_gradients_match_oracle(fam, dtype, cuda):
    """Per call and in one batch, every rule: within 1e-10 (fp64, the bound
    of the gradient tests); fp32 nodes and steps are rounded by 2^-24 of the
    coordinates, n 2^-24 of a step in every dimension."""
    from oracle import grad as OGR
    from torchquad_gb300.batch import BatchedGrid
    from torchquad_gb300.integration import _kernels as K

    specs = [(r, dim, valid_n(r, n)) for r in RULES
             for dim, n in [(1, 33), (1, 1001), (1, 4093), (2, 5), (2, 65), (2, 301), (3, 33), (4, 17), (6, 5), (8, 5)]
             if not (r == "gausslegendre" and n > 256) and n ** dim <= 2_000_000]
    fs = [family(fam, dim) for _, dim, _ in specs]
    doms = [domain(dim) for _, dim, _ in specs]
    bg = BatchedGrid(dtype=dtype, autotune=False)
    plan = bg.plan(fs, [s[0] for s in specs], [n ** dim for _, dim, n in specs], doms, tile_points=2048)
    assert list(plan.desc_np["n"]) == [n for _, _, n in specs]
    vals, gdom, gpar = (x.cpu().numpy() for x in bg.adjoint(plan))
    for i, (rule, dim, n) in enumerate(specs):
        f = fs[i]
        want = OGR.value_and_grad(f.family, f.params_numpy(), RULES[rule][1], dim, n, doms[i])
        tol = 1e-10 if dtype == torch.float64 else 4.0 * 2.0**-24 * max(n, 8) * dim
        integ = RULES[rule][0]()
        r, w = integ._gl_tables(n, cuda)
        one = K.grid_adjoint(integ._rule, dim, n, torch.tensor(doms[i], dtype=dtype, device=cuda), r, w, f)
        _assert_gradients([x.cpu().numpy() for x in one], want, tol, ("per call", rule, dim, n))
        d = plan.desc_np[i]
        in_batch = (vals[i], gdom[d["dom_off"]:d["dom_off"] + 2 * dim], gpar[d["par_off"]:d["par_off"] + 2 + 2 * dim])
        _assert_gradients(in_batch, want, tol, ("batch", rule, dim, n))


@pytest.mark.parametrize("dtype", [torch.float64, torch.float32])
@pytest.mark.parametrize("tile", [37, 64, 4096, 32768])
def test_batch_values_match_oracle(dtype, tile, cuda):
    """Factored and node-by-node integrals of all families and rules in one
    launch, one tile and many an integral, both block sizes."""
    from torchquad_gb300.batch import BatchedGrid

    fs, rules, Ns, doms, want, mag = [], [], [], [], [], []
    nd = np.float64 if dtype == torch.float64 else np.float32
    for rule in RULES:
        for fam in ("exp", "gauss", "osc", "sumsin"):
            for dim, n in [(1, 9), (1, 129), (1, 4093), (1, 40_001), (2, 9), (2, 65), (3, 33), (5, 9)]:
                n = valid_n(rule, min(n, 200) if rule == "gausslegendre" else n)
                fs.append(family(fam, dim))
                rules.append(rule)
                Ns.append(n ** dim)
                doms.append(domain(dim))
    if dtype == torch.float64:
        for _, f, dom in REFUSED[:4]:
            fs.append(f)
            rules.append("simpson")
            Ns.append(41 * 41)
            doms.append(dom)
    for f, rule, N, dom in zip(fs, rules, Ns, doms):
        v, m = oracle(f, RULES[rule][1], f.dim, N, dom, nd)
        want.append(v)
        mag.append(m)
    want, mag = np.array(want), np.array(mag)
    for block in (128, 256):
        bg = BatchedGrid(dtype=dtype, autotune=False, tile_points=tile, block=block, strip=4)
        got = bg.integrate(fs, rules, Ns, doms).double().cpu().numpy()
        tol = 1e-12 if dtype == torch.float64 else 1e-6
        bad = np.abs(got - want) > tol * mag + 1e-300
        assert not bad.any(), [(fs[i], rules[i], Ns[i], got[i], want[i]) for i in np.nonzero(bad)[0][:5]]


@pytest.mark.parametrize("where", ["device", "host", "mixed", "strided"])
@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
def test_backward_from_device_and_host_parameters(where, dtype, cuda):
    """The parameter vector gathered on the device and the one-launch backward
    against the gradient oracle; host parameters take the torch path."""
    from oracle import grad as OGR

    dim, n = 3, 21
    dom_l = domain(dim)
    a, u, c = [0.9, 1.7, 0.6], [0.2, 0.4, 0.1], 1.3
    dev = {"device": cuda, "host": "cpu", "mixed": cuda, "strided": cuda}[where]
    leaf = lambda x, d=dev, t=torch.float64: torch.tensor(x, dtype=t, device=d).requires_grad_()  # noqa: E731
    if where == "strided":
        base = leaf([[v, 0.0] for v in a])
        a_t = base[:, 0]
    else:
        base = a_t = leaf(a)
    u_t = leaf(u, "cpu" if where == "mixed" else dev)
    c_t = leaf(c, dev, torch.float32)
    dom = torch.tensor(dom_l, dtype=dtype, device=cuda).requires_grad_()
    f = tq.GaussianPeak(dim, a=a_t, u=u_t, c=c_t)
    val = tq.Simpson().integrate(f, dim, N=n**dim, integration_domain=dom)
    want = OGR.value_and_grad(f.family, np.concatenate([[np.float32(c), 0.0], a, u]), OGR.SIMPSON, dim, n, dom_l)
    tol = 1e-10 if dtype == torch.float64 else 4.0 * 2.0**-24 * n * dim
    for scale in (1.0, -2.5):
        g = torch.autograd.grad(val, [dom, c_t, base, u_t], grad_outputs=torch.tensor(scale, dtype=val.dtype, device=cuda),
                                retain_graph=True)
        ga = g[2][:, 0] if where == "strided" else g[2]
        assert [x.dtype for x in g] == [dtype, torch.float32, torch.float64, torch.float64]
        assert all(x.device == t.device for x, t in zip(g, (dom, c_t, base, u_t)))
        c_tol = max(tol, 2.0**-23)
        got_par = np.concatenate([[0.0, 0.0], ga.detach().cpu().numpy(), g[3].cpu().numpy()]) / scale
        want_par = np.concatenate([[0.0, 0.0], want[2][2:]])
        _assert_gradients((val.item(), g[0].cpu().numpy() / scale, got_par), (want[0], want[1], want_par),
                          tol, (where, dtype))
        assert abs(g[1].item() / scale - want[2][0]) <= c_tol * abs(want[2][0])


def test_parameters_written_between_calls(cuda):
    """Parameters on the device, written in place or replaced: every call sees
    the values of its time, also from another stream."""
    a = torch.tensor([1.0, 2.0], dtype=torch.float64, device=cuda)
    f = tq.ExpSum(2, a=a)
    dom = [[0.0, 1.0], [0.0, 1.0]]
    exact = lambda v: np.prod([(np.exp(x) - 1.0) / x for x in v])  # noqa: E731
    run = lambda: integrate("gausslegendre", f, 2, 24**2, dom, torch.float64, cuda).item()  # noqa: E731
    for v in ([1.0, 2.0], [0.5, 2.0], [0.5, 2.0], [1.5, 0.25]):
        a.copy_(torch.tensor(v, dtype=torch.float64))
        for _ in range(3):
            assert abs(run() - exact(v)) <= 1e-12 * exact(v)
    s = torch.cuda.Stream()
    s.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(s):
        a.mul_(2.0)
        assert abs(run() - exact([3.0, 0.5])) <= 1e-11
    torch.cuda.current_stream().wait_stream(s)
    f.a = torch.tensor([0.7, 0.9], dtype=torch.float64, device=cuda)
    assert abs(run() - exact([0.7, 0.9])) <= 1e-11
