"""Weight gradient of SO3Linear at the edges of its tiles, of its 16-row steps and of its splits, against float64."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype,tol", [(torch.float32, 2e-6), (torch.float64, 1e-14)])
@pytest.mark.parametrize("u,v", [(4, 4), (64, 64), (64, 68), (68, 64), (132, 260), (33, 64)])       # 33: the general kernel
@pytest.mark.parametrize("batch", [1, 37, 2500])
def test_weight_gradient(dtype, tol, u, v, batch):
    from fasteq_b200 import descriptors
    from fasteq_b200.irreps import Irreps
    from fasteq_b200.ops import fast_equi_linear
    # rows of 1, 3 and 5 per batch entry, two paths into one output irrep; the 16-row steps straddle batch entries
    d = descriptors.linear(Irreps(f"{u}x0e+{u}x1o+{u}x1o+{u}x2e"), Irreps(f"{v}x0e+{v}x1o+{v}x2e"))
    dim_in, dim_out = 12 * u, 9 * v
    g = torch.Generator().manual_seed(batch)
    x = torch.randn(batch, dim_in, generator=g, dtype=torch.float64).to(dtype)
    go = torch.randn(batch, dim_out, generator=g, dtype=torch.float64).to(dtype)
    w = torch.randn(d.num_weights, generator=g, dtype=torch.float64).to(dtype)
    wd = w.cuda().requires_grad_(True)
    (gw,) = torch.autograd.grad(fast_equi_linear(d, wd, x.cuda()), wd, go.cuda())
    xr, gr = x.double().reshape(batch, 12, u), go.double().reshape(batch, 9, v)
    rows = [(0, 0, 1, 1), (1, 1, 3, 2), (4, 1, 3, 2), (7, 4, 5, 1)]      # first rows, rows, paths into the same output irrep
    got = gw.cpu().double().reshape(4, u, v)
    for q, (i, o, n, into) in enumerate(rows):
        want = torch.einsum("btu,btv->uv", xr[:, i:i + n], gr[:, o:o + n]) / (into * u) ** 0.5      # 1 / sqrt(fan-in)
        err = (got[q] - want).norm() / want.norm()
        assert err <= tol, (q, float(err))                            # 2e-6: about 30 round-offs, blocked sums of 32 rows
