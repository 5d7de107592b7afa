"""The force pass of a training step computes no weight gradients (nobody asks for them there); every way of asking still
gets them, to second order."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _weight_gradient_launches(call):
    """``(result, launches of weight-gradient kernels)`` of a call."""
    from torch.profiler import ProfilerActivity, profile
    torch.cuda.synchronize()
    with profile(activities=[ProfilerActivity.CPU, ProfilerActivity.CUDA]) as prof:
        out = call()
        torch.cuda.synchronize()
    kernels = [e.name for e in prof.events() if e.device_type == torch.autograd.DeviceType.CUDA]
    assert kernels                                 # the profiler saw the launches
    return out, sum("wgrad" in k and "reduce" not in k for k in kernels)


def test_force_pass_skips_weight_gradients_and_loses_none():
    from fasteq_b200.ops import dense as dense_mod
    g = torch.Generator(device="cuda").manual_seed(0)
    x = torch.randn(40, 16, device="cuda", generator=g, requires_grad=True)
    w = torch.randn(8, 16, device="cuda", generator=g, requires_grad=True)
    y = (dense_mod.dense(x, w) ** 3).sum()
    (f,), launched = _weight_gradient_launches(lambda: torch.autograd.grad(y, x, create_graph=True))
    assert launched == 0
    _, launched = _weight_gradient_launches(lambda: torch.autograd.grad((dense_mod.dense(x, w) ** 3).sum(), (x, w), create_graph=True))
    assert launched == 1
    (gw,) = torch.autograd.grad((f ** 2).sum(), w)
    xd, wd = x.detach().double().requires_grad_(True), w.detach().double().requires_grad_(True)
    y = xd @ wd.t()
    (fd,) = torch.autograd.grad((y ** 3).sum(), xd, create_graph=True)
    (gwd,) = torch.autograd.grad((fd ** 2).sum(), wd)
    assert (gw.double() - gwd).norm() <= 1e-5 * gwd.norm()
    # asked for together with the inputs, as a leaf, through another tensor, and by backward()
    want = torch.autograd.grad(((xd @ wd.t()) ** 3).sum(), wd)[0]
    both = torch.autograd.grad((dense_mod.dense(x, w) ** 3).sum(), (x, w), create_graph=True)[1]
    through = torch.autograd.grad((dense_mod.dense(x, w * 1.0) ** 3).sum(), w, create_graph=True)[0]
    (dense_mod.dense(x, w) ** 3).sum().backward(create_graph=True)
    for got in (both, through, w.grad):
        assert (got.detach().double() - want).norm() <= 1e-5 * want.norm()
    w.grad = x.grad = None


def _linear(g):
    from fasteq_b200 import descriptors
    from fasteq_b200.irreps import Irreps
    from fasteq_b200.ops import eqlinear, fast_equi_linear
    d = descriptors.linear(Irreps("8x0e+8x1o"), Irreps("8x0e+8x1o"))
    x, w = torch.randn(21, 32, device="cuda", generator=g), torch.randn(d.num_weights, device="cuda", generator=g)

    def plain(x, w):
        xs, ws = x.reshape(21, 4, 8), w.reshape(2, 8, 8) / 8 ** 0.5
        return torch.cat([xs[:, :1] @ ws[0], xs[:, 1:] @ ws[1]], 1).reshape(21, 32)
    return x, w, lambda x, w: fast_equi_linear(d, w, x), plain, (eqlinear._Plan, "wgrad")


def _contraction(g):
    from fasteq_b200.descriptors import symmetric_contraction
    from fasteq_b200.ops import fast_stc_uniform1d_jit, stc_uniform1d_jit as stc
    from tests.test_stc_gpu import _torch_stc
    d = symmetric_contraction("16x0e+16x1o", "16x0e+16x1o")
    x = 0.5 * torch.randn(21, d.x1_segs, 16, device="cuda", generator=g)
    w = 0.3 * torch.randn(2, d.x0_segs, 16, device="cuda", generator=g)
    i0, tables = torch.arange(21, device="cuda") % 2, d.tensors(torch.float32, "cuda")
    # what a pass that wants the weight gradient loads, and one that does not never does
    counted = (stc, "get_module", lambda spec, direction, need_gx0=False, operands=(): direction in ("bwd", "bwdsum") and need_gx0)
    return x, w, lambda x, w: fast_stc_uniform1d_jit(x, w, i0, *tables, d.out_segs), lambda x, w: _torch_stc(x, w, i0, d.paths, d.coeffs, d.out_segs), counted


@pytest.mark.parametrize("layer", [_linear, _contraction])
def test_other_layers_skip_and_keep_theirs(layer, monkeypatch):
    g = torch.Generator(device="cuda").manual_seed(1)
    x, w, ours, plain, (owner, name, *which) = layer(g)
    calls, inner = [], getattr(owner, name)

    def counting(*a, **k):
        if not which or which[0](*a, **k):
            calls.append(1)
        return inner(*a, **k)
    monkeypatch.setattr(owner, name, counting)

    def step(f, x, w):
        x, w = x.requires_grad_(True), w.requires_grad_(True)
        (force,) = torch.autograd.grad((f(x, w) ** 3).sum(), x, create_graph=True)
        skipped = len(calls)
        first = torch.autograd.grad((f(x, w) ** 3).sum(), (x, w), create_graph=True)[1]
        return skipped, torch.autograd.grad((force ** 2).sum(), w)[0], first, torch.autograd.grad((f(x, w) ** 3).sum(), w)[0]

    skipped, *got = step(ours, x.clone(), w.clone())
    assert skipped == 0 and calls
    for a, b in zip(got, step(plain, x.double(), w.double())[1:]):
        assert (a.detach().double() - b.detach()).norm() <= 2e-5 * b.norm()      # products of three FP32 results


def test_readout_skips_and_keeps_its_weight_gradient():
    from fasteq_b200.ops import readout
    g = torch.Generator(device="cuda").manual_seed(2)
    h, w = torch.randn(9, 40, device="cuda", generator=g), torch.randn(33, device="cuda", generator=g)
    seen, inner = [], readout.wanted

    def recording(ctx, i):
        seen.append(inner(ctx, i))
        return seen[-1]
    readout.wanted, keep = recording, readout.wanted
    try:
        h.requires_grad_(True), w.requires_grad_(True)
        (f,) = torch.autograd.grad((readout.scalar_readout(h, w) ** 3).sum(), h, create_graph=True)
        assert seen == [False]
        (got,) = torch.autograd.grad((f ** 2).sum(), w)
    finally:
        readout.wanted = keep
    hd, wd = h.detach().double().requires_grad_(True), w.detach().double().requires_grad_(True)
    (fd,) = torch.autograd.grad(((hd[:, :33] * wd).sum(-1) ** 3).sum(), hd, create_graph=True)
    (want,) = torch.autograd.grad((fd ** 2).sum(), wd)
    assert (got.double() - want).norm() <= 1e-5 * want.norm()
