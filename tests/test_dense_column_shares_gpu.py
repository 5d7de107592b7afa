"""Dense layers whose work is divided otherwise than tile by tile: wide shallow ones of few row blocks (a block's weight tiles are shared out
over CTAs), long narrow ones (two row tiles to a CTA)."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m", [1, 129, 79 * 128 - 3, 149 * 128, 300 * 128 + 1])
@pytest.mark.parametrize("n,k", [(256, 32), (1284, 64)])
def test_against_float64_and_against_more_rows(m, n, k):
    from fasteq_b200.ops.dense import dense, tensorcore_device_status
    gen = torch.Generator(device="cuda").manual_seed(m + n)
    x = torch.randn(700 * 128, k, device="cuda", generator=gen)
    w = torch.randn(n, k, device="cuda", generator=gen) / k ** 0.5
    out = dense(x[:m], w)
    want = x[:m].double() @ w.double().t()
    assert float((out - want).norm()) <= 2e-6 * float(want.norm())           # 3xTF32 at K <= 64: 5e-7 measured
    assert torch.equal(out, dense(x, w)[:m])                                  # 700 blocks are not shared out; the sums are the same
    assert tensorcore_device_status() == 0


@pytest.mark.parametrize("m", [2 * 148 * 128 - 128, 2 * 148 * 128, 2 * 148 * 128 + 1, 3 * 148 * 128 - 5, 4 * 148 * 128 + 300])     # pairs, then single tiles
@pytest.mark.parametrize("n,k", [(64, 256), (64, 260), (20, 1284)])
def test_long_and_narrow(m, n, k):
    from fasteq_b200.ops.dense import dense, tensorcore_device_status
    gen = torch.Generator(device="cuda").manual_seed(m + k)
    x = torch.randn(m, k, device="cuda", generator=gen)
    w = torch.randn(n, k, device="cuda", generator=gen) / k ** 0.5
    out = dense(x, w)
    want = x.double() @ w.double().t()
    # the tensor core truncates once per 8 columns: 2e-8 of the sum each time
    assert float((out - want).norm()) <= (1e-6 + 2.5e-9 * k) * float(want.norm())
    assert float((out - want).abs().max()) <= 1e-5 * float(want.abs().max())        # a misplaced tile would hide in a norm
    assert tensorcore_device_status() == 0
