"""Second-order tensor-product kernels (a tangent row beside each operand) against the sum of first-order launches they stand for."""
import itertools

import pytest
import torch

from fasteq_b200 import descriptors
from fasteq_b200.irreps import Irreps

pytestmark = pytest.mark.gpu
# 128 channels: packed, gradient row in tensor memory; 33: channel tail, element copies; 64 in FP64: one channel per thread; 55
# output segments of 64 channels: one-warp pipelines; l = 3 senders: the ring of one pipeline shortened to what an SM holds
SIGNATURES = [("128x0e+128x1o", 3, "natural", torch.float32), ("128x0e", 3, "natural", torch.float32), ("33x0e+33x1o", 2, None, torch.float32),
              ("64x0e+64x1o", 2, None, torch.float64), ("64x0e+64x1o", 3, None, torch.float32),
              ("128x0e+128x1o+128x2e+128x3o", 3, None, torch.float32)]


def _case(sig, n, e, ordered, shift=0):
    from fasteq_b200.ops import uniform1d_jit as u1d
    in1, lmax, parity, dtype = sig
    sh = Irreps.spherical_harmonics(lmax)
    io, ins = descriptors.full_channelwise_instructions(in1, sh, lmax, parity_filter=parity)
    d = descriptors.channelwise_tensor_product(in1, sh, io, ins)
    g = torch.Generator(device="cuda").manual_seed(n + e)

    def rand(rows, cols):
        flat = torch.randn(rows * cols + shift, generator=g, device="cuda", dtype=dtype)
        return flat[shift:].view(rows, cols)
    src = torch.randint(0, n, (e,), generator=g, device="cuda", dtype=torch.int32)
    dst = torch.randint(0, max(n - 2, 1), (e,), generator=g, device="cuda", dtype=torch.int32)      # the last rows stay empty
    if ordered:
        dst = torch.sort(dst).values
    shapes = ((e, d.w_seg_num * d.u_dim), (n, d.x_seg_num * d.u_dim), (e, d.y_seg_num))
    operands, tangents = [rand(*s) for s in shapes], [rand(*s) for s in shapes]
    call = u1d._Call(*operands, {1: src}, {0: dst}, d.meta(dtype, "cuda"))
    return u1d, call, rand(n, d.out_seg_num * d.u_dim), operands, tangents, dtype


def _compare(u1d, call, go, operands, tangents, dtype, wants=(True,) * 4):
    got = u1d._second_order(call, go, *operands, tuple(tangents), wants)
    want = u1d._second_order_composed(call, go, *operands, tuple(tangents), wants)
    # sums of up to a few hundred products in another order: sqrt(300) round-offs of the largest element
    tol = 2e-6 if dtype == torch.float32 else 4e-15
    for name, a, b in zip(("go", "w", "x", "y"), got, want):
        assert (a is None) == (b is None), name
        if a is not None:
            assert a.shape == b.shape and float((a - b).abs().max()) <= tol * float(b.abs().max()), name


@pytest.mark.parametrize("sig", SIGNATURES, ids=[f"{s[0]}-{s[1]}-{str(s[3])[-2:]}" for s in SIGNATURES])
@pytest.mark.parametrize("n,e,ordered", [(40, 700, True), (513, 6000, False), (3, 2, True)])
def test_all_tangents(sig, n, e, ordered):
    _compare(*_case(sig, n, e, ordered))


@pytest.mark.parametrize("has", [h for h in itertools.product([False, True], repeat=3) if any(h)])
@pytest.mark.parametrize("wants", [(True,) * 4, (True, True, True, False), (False, True, False, True)])
def test_missing_tangents_and_gradients(has, wants):
    """A force pass has no tangent of the first layer's features; a loss on weights asks for no gradient of the harmonics."""
    u1d, call, go, operands, tangents, dtype = _case(("32x0e+32x1o", 2, None, torch.float32), 57, 900, True)
    _compare(u1d, call, go, operands, [t if h else None for t, h in zip(tangents, has)], dtype, wants)


def test_odd_addresses_and_no_edges():
    _compare(*_case(SIGNATURES[0], 30, 200, True, shift=1))
    u1d, call, go, operands, tangents, _ = _case(SIGNATURES[0], 30, 0, True)
    d_go, d_w, d_x, d_y = u1d._second_order(call, go, *operands, tuple(tangents), (True,) * 4)
    assert d_w.numel() == d_y.numel() == 0 and torch.count_nonzero(d_go) == 0 and torch.count_nonzero(d_x) == 0


def test_forms_without_second_order_modules_are_composed():
    from fasteq_b200.ops import uniform1d_jit as u1d
    import dataclasses
    spec = _case(("32x0e+32x1o", 2, None, torch.float32), 8, 20, True)[1].spec
    assert u1d._dual_spec(spec, (True, True, True)) is not None
    for change in (dict(w_shared=True), dict(y_vec=True), dict(x_indexed=False), dict(y_indexed=True), dict(scattered=False)):
        assert u1d._dual_spec(dataclasses.replace(spec, **change), (True, True, True)) is None
