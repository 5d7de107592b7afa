"""Weight gradients of more than 65,535 tiles (as many as a grid's second dimension holds): long, thin ones, so that the
matrices stay small."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,k,tile", [(4, 128 * 65_536 + 4, 128), (3, 64 * 65_536 + 1, 64)])       # FP32 ring kernel, general kernel
def test_more_tiles_than_a_second_grid_dimension_holds(n, k, tile):
    from fasteq_b200.ops.dense import _matmul_tn
    assert -(-k // tile) > 65_535
    gen = torch.Generator(device="cuda").manual_seed(0)
    g, x = torch.randn(2, n, device="cuda", generator=gen), torch.randn(2, k, device="cuda", generator=gen)
    got = _matmul_tn(g, x)
    want = torch.einsum("mn,mk->nk", g.double(), x.double())
    assert (got - want).abs().max() <= 2e-7 * 2 * want.abs().max()                      # two products and one sum, rounded


@pytest.mark.parametrize("dtype,tol", [(torch.float32, 2e-6), (torch.float64, 1e-14)])
@pytest.mark.parametrize("m", [1, 15, 128, 129, 257])
@pytest.mark.parametrize("n,k", [(4, 260), (132, 64), (132, 260)])
def test_few_rows(dtype, tol, m, n, k):
    """Up to 128 rows: one share and 64 x 64 tiles; beyond: larger tiles; several shares: the interleaved reduction."""
    from fasteq_b200.ops.dense import _matmul_tn
    gen = torch.Generator().manual_seed(m)
    g, x = torch.randn(m, n, generator=gen, dtype=torch.float64).to(dtype), torch.randn(m, k, generator=gen, dtype=torch.float64).to(dtype)
    want = g.double().t() @ x.double()
    assert (_matmul_tn(g.cuda(), x.cuda()).cpu().double() - want).norm() <= tol * want.norm()      # blocked sums of 32 rows
