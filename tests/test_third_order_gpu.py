"""Derivatives of the gradients' gradients: the multilinear operators give them, against float64 torch."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _dense(g):
    from fasteq_b200.ops.dense import dense
    return dense, lambda x, w: x @ w.t(), [torch.randn(40, 16, device="cuda", generator=g), torch.randn(8, 16, device="cuda", generator=g)]


def _linear(g):
    from fasteq_b200 import descriptors
    from fasteq_b200.irreps import Irreps
    from fasteq_b200.ops import fast_equi_linear
    d = descriptors.linear(Irreps("8x0e+8x1o"), Irreps("8x0e+8x1o"))

    def plain(x, w):
        xs, ws = x.reshape(21, 4, 8), w.reshape(2, 8, 8) / 8 ** 0.5
        return torch.cat([xs[:, :1] @ ws[0], xs[:, 1:] @ ws[1]], 1).reshape(21, 32)
    return (lambda x, w: fast_equi_linear(d, w, x)), plain, [torch.randn(21, 32, device="cuda", generator=g),
                                                             torch.randn(d.num_weights, device="cuda", generator=g)]


def _tensor_product(g, general=False):
    """``general``: shared weights, no gather, no scatter, which the native host path does not take."""
    from fasteq_b200 import descriptors
    from fasteq_b200.irreps import Irreps
    from fasteq_b200.ops import fast_uniform1d_jit
    from oracle.mace_style_ref import u1d_scatter
    sh = Irreps.spherical_harmonics(2)
    io, ins = descriptors.full_channelwise_instructions("32x0e+32x1o", sh, 2)
    d = descriptors.channelwise_tensor_product("32x0e+32x1o", sh, io, ins)
    n, e = (9, 9) if general else (9, 50)
    shapes = ((1 if general else e, d.w_seg_num * 32), (n, d.x_seg_num * 32), (e, d.y_seg_num))
    meta, ops = d.meta(torch.float32, "cuda"), [torch.randn(*s, device="cuda", generator=g) * 0.3 for s in shapes]
    if general:
        rows = torch.arange(n)
        return (lambda w, x, y: fast_uniform1d_jit(w, x, y, {}, {}, meta)), (lambda w, x, y: u1d_scatter(w.expand(n, -1), x, y, d, rows, rows, n)), ops
    src, dst = torch.randint(0, n, (2, e), generator=g, device="cuda", dtype=torch.int32)
    return ((lambda w, x, y: fast_uniform1d_jit(w, x, y, {1: src}, {0: dst}, meta)),
            (lambda w, x, y: u1d_scatter(w, x, y, d, src.cpu().long(), dst.cpu().long(), n)), ops)


def _general_form(g):
    return _tensor_product(g, True)


@pytest.mark.parametrize("make", [_dense, _linear, _tensor_product, _general_form])
def test_third_order(make):
    ours, plain, operands = make(torch.Generator(device="cuda").manual_seed(3))

    def third(f, operands):
        ops = [t.detach().requires_grad_(True) for t in operands]
        grads = torch.autograd.grad((f(*ops) ** 3).sum(), ops, create_graph=True)
        again = torch.autograd.grad(sum((a ** 2).sum() for a in grads), ops, create_graph=True)
        return torch.autograd.grad(sum((a ** 2).sum() for a in again), ops)

    for a, b in zip(third(ours, operands), third(plain, [t.cpu().double() for t in operands])):
        assert (a.cpu().double() - b).norm() <= 2e-5 * b.norm()          # up to eight chained FP32 (3xTF32) products
