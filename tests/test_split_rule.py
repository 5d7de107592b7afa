"""When the tensor-product kernels cut their shares between edges, and the degrees the decision rests on."""
import pytest
import torch

from fasteq_b200 import _cabi
from fasteq_b200.ops import uniform1d_jit as u1d


def _desc(direction, u=128, out_segs=55, f64=False):
    return _cabi.U1DDesc(dtype=int(f64), u=u, out_segs=out_segs, direction=direction, ctas_per_sm=4)


def test_a_forward_is_cut_only_where_the_longest_receiver_outweighs_the_carries():
    cut = lambda rows, degree, longest, **k: u1d.split_receivers(_desc(0, **k), rows, rows * degree, longest, 592)
    assert not cut(512, 8, 19) and not cut(3000, 8, 20) and not cut(8000, 2, 7)      # more launches for nothing
    assert cut(192, 52, 83) and cut(1, 60, 60) and cut(2000, 30, 50) and cut(64, 8, 103)
    assert not cut(512, 30, 30) and cut(512, 8, 103)                                # the longest, not the mean
    assert not cut(192, 16, 25) and cut(192, 16, 25, u=33)                          # rows of 132 bytes: no bulk copies
    assert not cut(1024, 16, 29) and cut(1024, 16, 29, f64=True, out_segs=106)
    assert not cut(592 * u1d.SPLIT_ROWS_PER_PIPELINE, 50, 80) and not cut(5, 0, 0)
    assert cut(6000, 52, 83) and not cut(9000, 52, 84) and not cut(12_288, 52, 83)  # many receivers per pipeline: nothing to gain
    # equal receivers that fill whole shares of the slowest rows
    even = lambda rows, degree, longest, **k: u1d.split_receivers(_desc(1, **k), rows, rows * degree, longest, 296)
    assert not even(2000, 8, 8, f64=True, out_segs=106) and not even(2000, 30, 30, f64=True, out_segs=106)
    assert even(2000, 8, 19, f64=True, out_segs=106) and even(1024, 30, 30, f64=True, out_segs=106) and even(2000, 8, 8)
    assert even(64, 8, 8, f64=True, out_segs=106)
    assert u1d.split_receivers(_desc(1), 12_288, 12_288 * 52, 83, 592)
    # the backward carries nothing
    assert u1d.split_receivers(_desc(1), 512, 4096, 19, 592) and not u1d.split_receivers(_desc(1), 592 * 32, 592 * 32 * 50, 80, 592)


@pytest.mark.gpu
@pytest.mark.parametrize("kind", ["sorted", "unsorted", "hub", "outside", "one", "none", "long"])
def test_plan_knows_order_and_largest_degree(kind):
    g = torch.Generator().manual_seed(3)
    n = {"one": 1, "long": 300_001}.get(kind, 777)
    dst = torch.randint(0, n, (0 if kind == "none" else 900_017 if kind == "long" else 5003,), generator=g)
    if kind in ("sorted", "long"):
        dst = dst.sort().values
    elif kind == "hub":
        dst[torch.rand(5003, generator=g) < 0.8] = 5
    elif kind == "outside":
        dst[:40], dst[40:90] = -2, n
    plan = u1d.GraphPlan(dst.int().cuda(), n)
    inside = dst[(dst >= 0) & (dst < n)]
    assert plan.max_degree == (int(torch.bincount(inside, minlength=n).max()) if inside.numel() else 0)
    assert plan.sorted == (kind in ("sorted", "long", "one", "none")) == bool((dst[1:] >= dst[:-1]).all())
    assert torch.equal(plan.seg_ptr.cpu().long(), torch.searchsorted(dst.sort().values, torch.arange(n + 1)))


@pytest.mark.gpu
def test_callers_degree_is_kept_and_otherwise_the_smallest_possible_one_stands_in():
    seg = torch.tensor([0, 2, 7], dtype=torch.int32, device="cuda")
    dst = torch.tensor([0, 0, 1, 1, 1, 1, 1], dtype=torch.int32, device="cuda")
    assert u1d.register_sorted_plan(dst, 2, seg, max_degree=5).max_degree == 5
    assert u1d.register_sorted_plan(dst, 2, seg).max_degree == 4
    u1d.invalidate_plan(dst)
