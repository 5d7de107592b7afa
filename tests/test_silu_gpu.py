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


def test_no_less_precise_than_torch():
    """Against float64, at most torch's own error in every order (2-norm of the difference over that of the result)."""
    from fasteq_b200.ops.silu import silu
    g = torch.Generator(device="cuda").manual_seed(0)
    z, a, b = (torch.randn(1_000_000, device="cuda", generator=g) for _ in range(3))

    def orders(f, z, a, b):
        z, a = z.detach().requires_grad_(True), a.detach().requires_grad_(True)
        (plain,) = torch.autograd.grad(f(z), z, a.detach())
        y = f(z)
        (d1,) = torch.autograd.grad(y, z, a, create_graph=True)
        return [t.detach() for t in (y, plain, d1, *torch.autograd.grad(d1, (a, z), b))]

    want = orders(torch.nn.functional.silu, z.double(), a.double(), b.double())
    err = lambda got: [float((x.double() - y).norm() / y.norm()) for x, y in zip(got, want)]
    for k, (ours, theirs) in enumerate(zip(err(orders(silu, z, a, b)), err(orders(torch.nn.functional.silu, z, a, b)))):
        assert ours <= 1.003 * theirs, (k, ours, theirs)         # 0.3 %: the statistics of a million roundings
