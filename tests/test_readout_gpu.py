"""Scalar readout against the elementwise expression: warps' remainders, all columns or some, with and without a running sum,
gradients of features and weights to second order."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype,tol", [(torch.float32, 2e-6), (torch.float64, 1e-14)])      # a sum of <= 160 products: ~ 20 round-offs
@pytest.mark.parametrize("n,c,d", [(0, 8, 8), (1, 1, 1), (9, 33, 33), (1000, 128, 512), (17, 160, 200)])
@pytest.mark.parametrize("running", [False, True])
def test_scalar_readout(dtype, tol, n, c, d, running):
    from fasteq_b200.ops.readout import scalar_readout
    g = torch.Generator().manual_seed(n + c)
    mk = lambda *s: torch.randn(*s, generator=g, dtype=torch.float64)
    h, w, e, a, b = mk(n, d), mk(c), mk(n), mk(n), mk(n, d)

    def all_of(f, cast):
        hh, ww, ee = (cast(t).requires_grad_(True) for t in (h, w, e))
        y = f(hh, ww, ee if running else None)
        first = torch.autograd.grad((y ** 2 * cast(a)).sum(), (hh, ww) + ((ee,) if running else ()))
        y = f(hh, ww, ee if running else None)
        (gh,) = torch.autograd.grad((y ** 2).sum(), hh, create_graph=True)
        return [y, *first, *torch.autograd.grad((gh * cast(b)).sum(), (hh, ww))]

    plain = lambda hh, ww, ee: (hh[:, :c] * ww).sum(-1) + (0 if ee is None else ee)
    got = all_of(scalar_readout, lambda t: t.to(dtype).cuda())
    want = all_of(plain, lambda t: t.to(dtype).double())
    for x, y in zip(got, want):
        assert x.shape == y.shape
        scale = max(float(y.abs().max()), 1.0) if y.numel() else 1.0
        assert y.numel() == 0 or float((x.detach().cpu().double() - y).abs().max()) <= 4 * tol * scale
