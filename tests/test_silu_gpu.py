"""SiLU to third order against torch in float64: wide and scalar accesses, saturated and zero arguments, unaligned views."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype,tol", [(torch.float32, 2e-6), (torch.float64, 1e-14)])      # a dozen round-offs of the largest term
@pytest.mark.parametrize("n,offset", [(0, 0), (1, 0), (7, 0), (1024, 0), (1023, 1), (4096, 1)])
def test_silu_and_its_derivatives(dtype, tol, n, offset):
    from fasteq_b200.ops.silu import silu
    g = torch.Generator().manual_seed(n)
    base = torch.randn(n + offset, generator=g, dtype=torch.float64).mul_(4).to(dtype)
    if n > 5:
        base[offset:offset + 4] = torch.tensor([0.0, -120.0, 120.0, -0.0], dtype=dtype)
    a, b = torch.randn(n, generator=g, dtype=torch.float64).to(dtype), torch.randn(n, generator=g, dtype=torch.float64).to(dtype)

    def orders(f, z, a, b):
        z = z.detach().requires_grad_(True)
        y = f(z)
        (d1,) = torch.autograd.grad((y * a).sum(), z, create_graph=True)
        (d2,) = torch.autograd.grad((d1 * b).sum(), z, create_graph=True)
        (d3,) = torch.autograd.grad(d2.sum(), z)
        a2 = a.detach().requires_grad_(True)
        (e1,) = torch.autograd.grad((f(z) * a2).sum(), z, create_graph=True)
        e2 = torch.autograd.grad((e1 * b).sum(), (a2, z))              # the kernel's second order
        return [y, d1, d2, d3, *e2]

    got = orders(silu, base.cuda()[offset:], a.cuda(), b.cuda())
    want = orders(torch.nn.functional.silu, base[offset:].double(), a.double(), b.double())
    for x, y in zip(got, want):
        assert x.shape == y.shape
        assert torch.all((x.detach().cpu().double() - y).abs() <= tol * (1 + y.abs()))
