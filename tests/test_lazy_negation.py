"""Tensors whose memory is not their value (lazily negated or conjugated
views, zero tensors without storage): kernels must not read their pointers.
Autograd hands such gradients to a backward in ordinary code."""
import pytest
import torch

import torchquad_gb300 as tq
from torchquad_gb300 import _lib as L
from torchquad_gb300.integration.utils import _split_integrand_values

F64 = torch.float64


def test_plain_tensor_refuses_lazy_values():
    z = torch.tensor([1.0 + 2.0j, 3.0 - 4.0j])
    assert L.plain_tensor(torch.ones(2))
    assert L.plain_tensor(z) and L.plain_tensor(z.imag)
    assert z.conj().imag.is_neg() and not L.plain_tensor(z.conj().imag)
    assert L.plain_tensor(z.conj().imag.resolve_neg())
    assert not L.plain_tensor(z.conj())
    assert not L.plain_tensor(torch._efficientzerotensor(()))


def test_integrand_values_are_resolved():
    z = torch.tensor([[1.0 + 2.0j], [3.0 - 4.0j]])
    v, shape, is_complex = _split_integrand_values(z.conj())
    assert is_complex and shape == (1,) and not v.is_neg()
    assert torch.equal(v, torch.tensor([[1.0, -2.0], [3.0, 4.0]]))
    one = z[:1, 0].conj().imag  # one value: contiguous and lazily negated
    assert one.is_neg() and one.is_contiguous()
    v, _, _ = _split_integrand_values(one)
    assert not v.is_neg() and v.item() == -2.0


def _case(cuda, dtype):
    dom = torch.tensor([[0.1, 1.2], [-0.4, 0.9]], dtype=dtype, device=cuda, requires_grad=True)
    a = torch.tensor([0.7, -1.3], dtype=dtype, device=cuda, requires_grad=True)
    b = torch.tensor(0.3, dtype=dtype, device=cuda, requires_grad=True)
    c = torch.tensor(1.7, dtype=dtype, device=cuda, requires_grad=True)
    value = tq.Simpson().integrate(tq.ExpSum(2, a=a, b=b, c=c), 2, N=31**2, integration_domain=dom)
    return value, (dom, a, b, c)


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [F64, torch.float32])
@pytest.mark.parametrize("part", ["conjugate", "modulus"])
def test_gradient_of_complex_loss(part, dtype, cuda):
    """The integral as the imaginary part of a conjugated number: its
    gradient arrives lazily negated.  Against the same loss in real numbers."""
    w = complex(0.8, -0.6)
    out = []
    for form in ("complex", "real"):
        value, inputs = _case(cuda, dtype)
        x = torch.tensor(0.25, dtype=dtype, device=cuda)
        if form == "complex":
            z = torch.complex(x, value).conj() * w
            loss = z.real if part == "conjugate" else (z + 1.0).abs()
        else:  # (x - i value) w
            re, im = x * w.real + value * w.imag, x * w.imag - value * w.real
            loss = re if part == "conjugate" else torch.sqrt((re + 1.0) ** 2 + im**2)
        out.append(torch.autograd.grad(loss, inputs))
    tol = 1e-12 if dtype == F64 else 1e-5  # the same products, rounded once or twice differently
    for got, want in zip(*out):
        assert torch.allclose(got, want, rtol=tol, atol=tol), (got, want)


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [F64, torch.float32])
def test_lazily_negated_parameters(dtype, cuda):
    """a, b, c and u as imaginary parts of conjugated device tensors (strided
    and lazily negated) mean what their values say."""
    cdt = torch.complex128 if dtype == F64 else torch.complex64
    z = torch.tensor([0.0 - 0.7j, 0.0 - 1.3j], dtype=cdt, device=cuda)
    one = torch.tensor(0.0 - 1.7j, dtype=cdt, device=cuda)
    dom = [[0.1, 1.2], [-0.4, 0.9]]
    a, c = z.conj().imag, one.conj().imag
    assert a.is_neg() and c.is_neg()
    for mk in (lambda a, c: tq.ExpSum(2, a=a, b=c, c=c), lambda a, c: tq.GaussianPeak(2, a=a, u=a, c=c)):
        got = tq.Simpson().integrate(mk(a, c), 2, N=31**2, integration_domain=dom)
        want = tq.Simpson().integrate(mk(a.tolist(), c.item()), 2, N=31**2, integration_domain=dom)
        assert got.item() == want.item()
        got = tq.MonteCarlo().integrate(mk(a, c), 2, N=1000, integration_domain=dom, seed=3)
        want = tq.MonteCarlo().integrate(mk(a.tolist(), c.item()), 2, N=1000, integration_domain=dom, seed=3)
        assert got.item() == want.item()
