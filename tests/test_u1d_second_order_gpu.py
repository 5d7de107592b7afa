"""Second-order tensor-product kernels (a tangent row beside each operand), through the public operator and ``torch.autograd.grad``, against
a float64 restatement that torch differentiates itself."""
import itertools

import pytest
import torch

from fasteq_b200 import descriptors
from fasteq_b200.irreps import Irreps
from oracle.mace_style_ref import u1d_scatter

pytestmark = pytest.mark.gpu
# 128 channels: packed, gradient row in tensor memory; 33: channel tail, element copies; 64 in FP64: one channel per thread; 55
# output segments of 64 channels: one-warp pipelines; l = 3 senders: the ring of one pipeline shortened to what an SM holds
SIGNATURES = [("128x0e+128x1o", 3, "natural", torch.float32), ("128x0e", 3, "natural", torch.float32), ("33x0e+33x1o", 2, None, torch.float32),
              ("64x0e+64x1o", 2, None, torch.float64), ("64x0e+64x1o", 3, None, torch.float32)]
WIDE = ("128x0e+128x1o+128x2e+128x3o", 3, None, torch.float32)
SMALL = ("32x0e+32x1o", 2, None, torch.float32)


def _case(sig, n, e, ordered, shift=0):
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
    return d, src, dst, rand(n, d.out_seg_num * d.u_dim), [rand(*s) for s in shapes], [rand(*s) for s in shapes]


def _second(op, go, operands, tangents, wants):
    """Gradients of the first-order gradients' products with those tangents that are given, of go, w, x, y as wanted."""
    leaves = [t.detach().requires_grad_(True) for t in [go] + operands]
    first = torch.autograd.grad(op(*leaves[1:]), leaves[1:], leaves[0], create_graph=True)
    pairs = [(f, t) for f, t in zip(first, tangents) if t is not None]
    return torch.autograd.grad([f for f, _ in pairs], [t for t, on in zip(leaves, wants) if on], [t for _, t in pairs], allow_unused=True)


def _compare(sig, n, e, ordered, shift=0, has=(True,) * 3, wants=(True,) * 4):
    from fasteq_b200.ops import fast_uniform1d_jit
    d, src, dst, go, operands, tangents = _case(sig, n, e, ordered, shift)
    tangents = [t if h else None for t, h in zip(tangents, has)]
    meta = d.meta(sig[3], "cuda")
    got = _second(lambda w, x, y: fast_uniform1d_jit(w, x, y, {1: src}, {0: dst}, meta), go, operands, tangents, wants)
    cpu = lambda t: None if t is None else t.cpu().double()
    want = _second(lambda w, x, y: u1d_scatter(w, x, y, d, src.cpu().long(), dst.cpu().long(), n), cpu(go), [cpu(t) for t in operands],
                   [cpu(t) for t in tangents], wants)
    # sums of up to a few hundred products of four factors, each rounded: sqrt(300) round-offs of the largest element
    tol = 2e-6 if sig[3] == torch.float32 else 4e-15
    for name, a, b in zip([k for k, on in zip(("go", "w", "x", "y"), wants) if on], got, want):
        if a is None or b is None:                # no tangent on another operand: nothing, or zeros
            assert all(t is None or not torch.count_nonzero(t) for t in (a, b)), name
        else:
            assert a.shape == b.shape and float((a.cpu().double() - b).abs().max()) <= tol * float(b.abs().max()), name


@pytest.mark.parametrize("sig", SIGNATURES, ids=[f"{s[0]}-{s[1]}-{str(s[3])[-2:]}" for s in SIGNATURES])
@pytest.mark.parametrize("n,e,ordered", [(40, 700, True), (513, 6000, False), (3, 2, True)])
def test_all_tangents(sig, n, e, ordered):
    _compare(sig, n, e, ordered)


@pytest.mark.parametrize("has", [h for h in itertools.product([False, True], repeat=3) if any(h)])
@pytest.mark.parametrize("wants", [(True,) * 4, (True, True, True, False), (False, True, False, True)])
def test_missing_tangents_and_gradients(has, wants):
    """A force pass has no tangent of the first layer's features; a loss on weights asks for no gradient of the harmonics."""
    _compare(SMALL, 57, 900, True, has=has, wants=wants)


def test_wide_rows():
    """Two rows of 34 weight and 16 sender segments a stage: five stages would be 252 KB, an SM has 227."""
    _compare(WIDE, 40, 300, True)


@pytest.mark.parametrize("has", [(True, True, True), (False, True, False)])
def test_rows_too_wide_for_modules_are_composed(has, monkeypatch):
    from fasteq_b200.codegen import u1d as gen
    from fasteq_b200.ops import uniform1d_jit as u1d
    monkeypatch.setattr(gen, "second_order_fits", lambda spec: False)
    monkeypatch.setattr(u1d, "_DUAL_SPECS", {})
    monkeypatch.setattr(u1d, "_SIGNATURES", {})
    loaded, inner = [], u1d.get_module
    monkeypatch.setattr(u1d, "get_module", lambda spec, *a, **k: (loaded.append(spec), inner(spec, *a, **k))[1])
    _compare(SMALL, 57, 900, True, has=has)
    assert loaded and not any(s.dual for s in loaded)


def test_odd_addresses_and_no_edges():
    _compare(SIGNATURES[0], 30, 200, True, shift=1)
    from fasteq_b200.ops import fast_uniform1d_jit
    d, src, dst, go, operands, tangents = _case(SIGNATURES[0], 30, 0, True)
    meta = d.meta(torch.float32, "cuda")
    d_go, d_w, d_x, d_y = _second(lambda w, x, y: fast_uniform1d_jit(w, x, y, {1: src}, {0: dst}, meta), go, operands, tangents, (True,) * 4)
    assert d_w.numel() == d_y.numel() == 0 and torch.count_nonzero(d_go) == 0 and torch.count_nonzero(d_x) == 0


def test_forms_without_second_order_modules_are_composed():
    from fasteq_b200.ops import uniform1d_jit as u1d
    import dataclasses
    from fasteq_b200.prebuild import cwtp_spec
    spec = cwtp_spec(SMALL[0], SMALL[1], SMALL[1], "f32")
    assert u1d._dual_spec(spec, (True, True, True)) is not None
    for change in (dict(w_shared=True), dict(y_vec=True), dict(x_indexed=False), dict(y_indexed=True), dict(scattered=False)):
        assert u1d._dual_spec(dataclasses.replace(spec, **change), (True, True, True)) is None
