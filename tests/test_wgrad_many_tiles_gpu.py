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
