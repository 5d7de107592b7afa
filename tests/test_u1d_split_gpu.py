"""Shares of the tensor-product kernels cut between edges: receivers that several pipelines sum (one receiver with all edges,
a few, ragged ones with empty rows), sorted and unsorted, whole and tailed channel tiles, against the numpy oracle."""
import numpy as np
import pytest
import torch

from fasteq_b200.descriptors import channelwise_tensor_product, full_channelwise_instructions
from fasteq_b200.irreps import Irreps
from oracle import uniform1d_ref

pytestmark = pytest.mark.gpu


def _degrees(kind, rng):
    if kind == "one":
        return np.array([700])
    if kind == "few":
        return np.array([0, 913, 1, 0, 0, 350, 2, 0])
    return rng.integers(0, 60, size=150) * (rng.random(150) < 0.8)


@pytest.mark.parametrize("dtype,tol", [("f32", 1e-5), ("f64", 1e-11)])
@pytest.mark.parametrize("kind", ["one", "few", "ragged"])
@pytest.mark.parametrize("u,lmax,presorted", [(64, 2, True), (33, 2, False), (64, 3, False)])     # 64, 3: 55 output segments
def test_split_receivers_match_oracle(dtype, tol, kind, u, lmax, presorted):
    from fasteq_b200.ops import fast_uniform1d_jit
    from fasteq_b200.ops import uniform1d_jit as u1d
    sh = Irreps.spherical_harmonics(lmax)
    io, ins = full_channelwise_instructions(f"{u}x0e+{u}x1o", sh, lmax)
    d = channelwise_tensor_product(f"{u}x0e+{u}x1o", sh, io, ins)
    rng = np.random.default_rng(u)
    deg = _degrees(kind, rng)
    N, E = deg.size, int(deg.sum())
    dst = np.repeat(np.arange(N), deg)
    if not presorted:
        rng.shuffle(dst)
    src = rng.integers(0, N, size=E)
    t = torch.float32 if dtype == "f32" else torch.float64
    w, x, y, r = (torch.from_numpy(rng.normal(size=s)).to(t).cuda() for s in
                  ((E, d.w_seg_num * u), (N, d.x_seg_num * u), (E, d.y_seg_num), (N, d.out_seg_num * u)))
    for a in (w, x, y):
        a.requires_grad_(True)
    dst_t = torch.from_numpy(dst).int().cuda()
    out = fast_uniform1d_jit(w, x, y, {1: torch.from_numpy(src).int().cuda()}, {0: dst_t}, d.meta(t, "cuda"))
    assert any(split for _, split in u1d.graph_plan(dst_t, N)._parts), "this graph is meant to take the split shares"
    grads = torch.autograd.grad(out, (w, x, y), r)
    paths = list(zip(d.i_list.tolist(), d.j_list.tolist(), d.k_list.tolist(), d.v_list.tolist()))
    a = lambda q, s: q.detach().cpu().double().numpy().reshape(-1, s, q.shape[1] // s)
    args = (a(w, d.w_seg_num), a(x, d.x_seg_num), a(y, d.y_seg_num), paths, d.coeff_list)
    ref = [uniform1d_ref.uniform1d_forward(*args, d.out_seg_num, src_x=src, dst=dst, num_out_rows=N)]
    ref += list(uniform1d_ref.uniform1d_backward(a(r, d.out_seg_num), *args, src_x=src, dst=dst))
    for name, got, want in zip(("out", "gw", "gx", "gy"), (out,) + grads, ref):
        err = np.abs(got.detach().cpu().double().numpy().reshape(want.shape) - want).max() / np.abs(want).max()
        assert err <= tol, (name, err)


@pytest.mark.parametrize("presorted", [True, False])
def test_operands_at_odd_addresses_of_a_tensor_memory_layout(presorted):
    """55 segments of 64 channels park their gradient rows in tensor memory; at odd 4-byte addresses with one channel per thread."""
    from fasteq_b200.codegen import u1d as gen
    from fasteq_b200.ops import fast_uniform1d_jit
    from fasteq_b200.ops import uniform1d_jit as u1d
    sh = Irreps.spherical_harmonics(3)
    io, ins = full_channelwise_instructions("64x0e+64x1o", sh, 3)
    d = channelwise_tensor_product("64x0e+64x1o", sh, io, ins)
    g = torch.Generator(device="cuda").manual_seed(9)
    N, E = 37, 901
    rand = lambda *s: torch.randn(*s, device="cuda", generator=g)
    operands = rand(E, d.w_seg_num * 64), rand(N, d.x_seg_num * 64), rand(E, d.y_seg_num), rand(N, d.out_seg_num * 64)
    dst = torch.randint(0, N, (E,), device="cuda", generator=g, dtype=torch.int32)
    dst = dst.sort().values if presorted else dst
    src = torch.randint(0, N, (E,), device="cuda", generator=g, dtype=torch.int32)
    odd = lambda t: torch.empty(t.numel() + 1, device="cuda")[1:].view(t.shape).copy_(t)

    def run(w, x, y, r):
        w, x, y = (t.requires_grad_(True) for t in (w, x, y))
        out = fast_uniform1d_jit(w, x, y, {1: src}, {0: dst}, d.meta(torch.float32, "cuda"))
        return (out.detach(),) + torch.autograd.grad(out, (w, x, y), r)

    aligned = run(*(t.clone() for t in operands))
    spec = next(s for s, direction, *_ in u1d._MODULES if direction == "bwd" and (s.u, s.out_segs) == (64, 55) and s.dtype == "f32")
    assert gen.untuned(spec, "bwd").go_tmem
    for a, b in zip(run(*(odd(t) for t in operands)), aligned):
        assert (a - b).abs().max() <= 1e-5 * b.abs().max()           # two orders of the same FP32 sums
