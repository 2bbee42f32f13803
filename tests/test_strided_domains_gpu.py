"""GPU: domain tensors that are not contiguous (transposed, sliced, lazily
negated) mean what their values say, in results, gradients and point sets."""
import pytest
import torch

import torchquad_gb300 as tq
from torchquad_gb300.integration.integration_grid import IntegrationGrid

pytestmark = pytest.mark.gpu

LO, HI = [0.1, -0.4, 0.3], [1.2, 0.9, 1.1]


def domains(dtype, cuda):
    plain = torch.tensor([LO, HI], dtype=dtype, device=cuda).T.contiguous()
    wide = torch.full((3, 5), 7.0, dtype=dtype, device=cuda)
    wide[:, 1:3] = plain
    cdt = torch.complex128 if dtype == torch.float64 else torch.complex64
    z = torch.complex(torch.zeros_like(plain), -plain).to(cdt)
    return plain, {"transposed": torch.tensor([LO, HI], dtype=dtype, device=cuda).T, "sliced": wide[:, 1:3],
                   "negated": z.conj().imag, "host": torch.tensor([LO, HI], dtype=dtype).T}


def f(x):
    return torch.exp(x[:, 0] - 0.5 * x[:, 1]) + x[:, 2]


def fv(x):
    return torch.stack([x[:, 0], x[:, 1] * x[:, 2]], dim=1)


@pytest.mark.parametrize("form", ["transposed", "sliced", "negated", "host"])
@pytest.mark.parametrize("dtype", [torch.float64, torch.float32])
def test_values(form, dtype, cuda):
    plain, others = domains(dtype, cuda)
    dom = others[form]
    assert not dom.is_contiguous() or form == "host"
    built = tq.ExpSum(3, a=[0.7, -1.3, 0.4])
    for rule in (tq.Trapezoid(), tq.Simpson(), tq.Boole(), tq.GaussLegendre()):
        for fn in (built, f, fv):
            assert torch.equal(rule.integrate(fn, 3, N=9**3, integration_domain=dom),
                               rule.integrate(fn, 3, N=9**3, integration_domain=plain))
        if form != "host":
            points, _, n = rule.calculate_grid(9**3, dom)
            want, hs, _ = rule.calculate_grid(9**3, plain)
            assert torch.equal(points, want)
            assert torch.equal(rule.calculate_result(f(points), 3, n, hs, dom),
                               rule.calculate_result(f(want), 3, n, hs, plain))
    for fn in (built, f, fv):
        assert torch.equal(tq.MonteCarlo().integrate(fn, 3, N=2000, integration_domain=dom, seed=2),
                           tq.MonteCarlo().integrate(fn, 3, N=2000, integration_domain=plain, seed=2))
        if fn is not fv:
            got = tq.VEGAS().integrate(fn, 3, N=20_000, integration_domain=dom, seed=2)
            want = tq.VEGAS().integrate(fn, 3, N=20_000, integration_domain=plain, seed=2)
            assert torch.allclose(got, want, rtol=1e-6)  # sums by atomics
    if form != "host":
        assert torch.equal(IntegrationGrid(5**3, dom).points, IntegrationGrid(5**3, plain).points)
        got = tq.MonteCarlo().calculate_result(f(plain.new_ones(10, 3)), dom)
        assert torch.equal(got, tq.MonteCarlo().calculate_result(f(plain.new_ones(10, 3)), plain))


@pytest.mark.parametrize("dtype", [torch.float64, torch.float32])
def test_gradients(dtype, cuda):
    for fn in (tq.ExpSum(3, a=[0.7, -1.3, 0.4]), f):
        for rule in (tq.Simpson(), tq.GaussLegendre()):
            t = torch.tensor([LO, HI], dtype=dtype, device=cuda, requires_grad=True)
            p = t.detach().T.contiguous().requires_grad_(True)
            got = rule.integrate(fn, 3, N=9**3, integration_domain=t.T)
            want = rule.integrate(fn, 3, N=9**3, integration_domain=p)
            got.backward()
            want.backward()
            assert torch.equal(got, want)
            assert torch.allclose(t.grad.T, p.grad, rtol=1e-5 if dtype == torch.float32 else 1e-12)
