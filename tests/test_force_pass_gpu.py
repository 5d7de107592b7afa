"""The force pass of a training step computes no weight gradients (nobody asks for them there); every way of asking still
gets them, to second order."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def test_force_pass_skips_weight_gradients_and_loses_none(monkeypatch):
    from fasteq_b200.ops import dense as dense_mod
    calls = []
    inner = dense_mod._matmul_tn
    monkeypatch.setattr(dense_mod, "_matmul_tn", lambda g, x: (calls.append(1), inner(g, x))[1])
    g = torch.Generator(device="cuda").manual_seed(0)
    x = torch.randn(40, 16, device="cuda", generator=g, requires_grad=True)
    w = torch.randn(8, 16, device="cuda", generator=g, requires_grad=True)
    (f,) = torch.autograd.grad((dense_mod.dense(x, w) ** 3).sum(), x, create_graph=True)
    assert not calls
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
