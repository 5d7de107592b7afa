"""FP32 weight gradient on the tensor cores (more than 128 rows): edges of its chunks of 32 batch entries, of its tiles and of its second-level
sums, operands that bf16 parts cannot hold, and its error against the blocked FP32 sums it replaced."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _grad(g, x):
    from fasteq_b200.ops.dense import _matmul_tn, tensorcore_device_status
    out = _matmul_tn(g, x)
    assert tensorcore_device_status() == 0
    return out


def _operands(m, n, k, scale=1.0):
    gen = torch.Generator(device="cuda").manual_seed(m + n + k)
    return [torch.randn(m, c, device="cuda", generator=gen) * scale for c in (n, k)]


@pytest.mark.parametrize("m", [129, 160, 161, 512, 513, 5000, 100_003])
@pytest.mark.parametrize("n,k", [(4, 4), (64, 64), (60, 128), (128, 68), (132, 128), (260, 132)])
def test_against_float64(m, n, k):
    g, x = _operands(m, n, k)
    want = g.double().t() @ x.double()
    # per chunk two truncated steps (2^-24 each) and one rounding, 16 chunks and up to 60 second-level sums in random walks: below
    # 2^-24 * (2 + sqrt(8) + sqrt(30) / 4); the sums in chunks of 32 FP32 products reach 2.2e-7 at 100,000 rows
    assert (_grad(g, x) - want).norm() <= 3e-7 * want.norm()


@pytest.mark.parametrize("batch", [15, 16, 31, 33, 64, 100])
def test_irrep_rows_of_short_batches(batch):
    """Rows are 32 entries of one irrep row each: batches on both sides of a chunk, and of the limit of the tensor-core kernel."""
    from fasteq_b200 import descriptors
    from fasteq_b200.irreps import Irreps
    from fasteq_b200.ops import fast_equi_linear
    d = descriptors.linear(Irreps("64x0e+64x4e"), Irreps("132x4e+132x0e"))
    gen = torch.Generator(device="cuda").manual_seed(batch)
    x, go = (torch.randn(batch, 10 * c, device="cuda", generator=gen) for c in (64, 132))
    w = torch.randn(d.num_weights, device="cuda", generator=gen).requires_grad_(True)
    (gw,) = torch.autograd.grad(fast_equi_linear(d, w, x), w, go)
    xr, gr = x.double().view(batch, 10, 64), go.double().view(batch, 10, 132)
    got = gw.double().view(2, 64, 132)
    for q, (i, o, n) in enumerate([(0, 9, 1), (1, 0, 9)]):
        want = torch.einsum("btu,btv->uv", xr[:, i:i + n], gr[:, o:o + n]) / 8.0
        assert (got[q] - want).norm() <= 3e-7 * want.norm()


@pytest.mark.parametrize("value", [float("inf"), -float("inf"), float("nan"), 3.4e38])
def test_values_beyond_bf16(value):
    """Infinities and NaN reach exactly the sums they reach in FP32; a value bf16 would round to infinity stays finite."""
    g, x = _operands(1000, 64, 132)
    g[517, 3] = value
    x[517] *= 1e-3
    want = g.double().t() @ x.double()
    got = _grad(g, x)
    assert torch.equal(got.isnan(), want.isnan()) and torch.equal(got.isposinf(), want.isposinf()) and torch.equal(got.isneginf(), want.isneginf())
    fine = want.isfinite()
    assert (got.double() - want)[fine].abs().max() <= 1e-6 * want[fine].abs().max()


@pytest.mark.parametrize("value", [float("inf"), float("nan"), 1e35])
@pytest.mark.parametrize("u,v", [(64, 132), (132, 64), (200, 136)])
def test_values_beyond_bf16_in_irrep_rows(value, u, v):
    """The recomputation in FP32 over paths of several rows, either operand the wider one, tiles beyond the extents."""
    from fasteq_b200 import descriptors
    from fasteq_b200.irreps import Irreps
    from fasteq_b200.ops import fast_equi_linear
    d = descriptors.linear(Irreps(f"{u}x0e+{u}x2e"), Irreps(f"{v}x2e+{v}x0e"))
    gen = torch.Generator(device="cuda").manual_seed(u)
    x, go = (torch.randn(301, 6 * c, device="cuda", generator=gen) for c in (u, v))
    x[300, u + 3] = value                 # the first of the l = 2 rows, channel 3, in the last chunk
    w = torch.randn(d.num_weights, device="cuda", generator=gen).requires_grad_(True)
    (gw,) = torch.autograd.grad(fast_equi_linear(d, w, x), w, go)
    xr, gr, got = x.double().view(301, 6, u), go.double().view(301, 6, v), gw.double().view(2, u, v)
    for q, (i, o, n) in enumerate([(0, 5, 1), (1, 0, 5)]):
        want = torch.einsum("btu,btv->uv", xr[:, i:i + n], gr[:, o:o + n]) / u ** 0.5
        assert torch.equal(got[q].isnan(), want.isnan()) and torch.equal(got[q].isposinf(), want.isposinf())
        for rows in (slice(3, 4), slice(0, 3), slice(4, None)):
            fine = want[rows].isfinite()
            assert (got[q][rows] - want[rows])[fine].norm() <= 3e-7 * want[rows][fine].norm()


@pytest.mark.parametrize("scale", [1e-36, 1e-19, 1e18])
def test_small_and_large_operands(scale):
    g, x = _operands(700, 64, 64)
    g, x = g * scale, (x if scale < 1e-30 else x * scale)
    want = g.double().t() @ x.double()
    # 1e-36: products near FP32's smallest normal number, rounded to multiples of 2^-149
    assert (_grad(g, x).double() - want).norm() <= 3e-7 * want.norm() + (2.0 ** -149 * 700 * 64 if scale < 1e-18 else 0.0)


@pytest.mark.parametrize("tiny", [1e-30, 1e-33, 1e-35, 1e-37, 1e-40])
@pytest.mark.parametrize("side", [0, 1])
def test_tiny_operands_against_large_ones(tiny, side):
    """An operand whose third bf16 part is below bf16's numbers, times one that brings the sums back to ordinary size."""
    ops = _operands(700, 64, 132)
    ops[side], ops[1 - side] = ops[side] * tiny, ops[1 - side] * 1e30
    g, x = ops
    want = g.double().t() @ x.double()
    assert (_grad(g, x).double() - want).norm() <= 3e-7 * want.norm()


def test_a_tiny_channel_beside_ordinary_ones():
    """One channel of one operand is tiny, and so small that its sums vanish beside the tile's others."""
    g, x = _operands(700, 64, 132)
    x[:, 5] *= 1e-34
    want = g.double().t() @ x.double()
    got = _grad(g, x).double()
    for cols in (slice(5, 6), slice(0, 5), slice(6, None)):
        assert (got[:, cols] - want[:, cols]).norm() <= 3e-7 * want[:, cols].norm()


@pytest.mark.parametrize("m", [160, 5000, 100_003])
def test_operands_of_one_sign(m):
    """The tensor core truncates, always towards zero here, and no cancellation hides it: per chunk two truncated steps of at most 2^-23,
    half of that on average, of which the reduction gives three quarters of 2^-24 back, beside the roundings of the sums."""
    g, x = (t.abs() for t in _operands(m, 68, 128))
    want = g.double().t() @ x.double()
    assert (_grad(g, x).double() - want).norm() <= 1e-7 * want.norm()


def test_zero_and_repeat():
    g, x = _operands(4000, 128, 128)
    assert torch.equal(_grad(g, x), _grad(g, x))                     # fixed order of the sums
    assert torch.count_nonzero(_grad(torch.zeros_like(g), x)) == 0
