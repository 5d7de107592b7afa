"""The symmetric contraction's first-order backward sums the weight gradient by species in the kernel: shares of one node,
shares that span several species, species without nodes, a channel tail, and the same bits on every call."""
import numpy as np
import pytest
import torch

from fasteq_b200.descriptors import symmetric_contraction
from oracle import stc_ref

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype,tol", [(torch.float32, 1e-5), (torch.float64, 1e-11)])
@pytest.mark.parametrize("u,B,S,used", [(33, 1, 1, [0]), (33, 2, 3, [2]), (33, 700, 89, [0, 5, 88]), (160, 1500, 12, list(range(1, 12)))])
def test_summed_weight_gradient(dtype, tol, u, B, S, used):
    from fasteq_b200.ops import fast_stc_uniform1d_jit
    d = symmetric_contraction(f"{u}x0e+{u}x1o", f"{u}x0e+{u}x1o")
    g = torch.Generator().manual_seed(B)
    x1 = (torch.randn(B, d.x1_segs, u, generator=g, dtype=torch.float64) * 0.3).to(dtype)
    x0 = (torch.randn(S, d.x0_segs, u, generator=g, dtype=torch.float64) * 0.1).to(dtype)
    r = torch.randn(B, d.out_segs * u, generator=g, dtype=torch.float64).to(dtype)
    i0 = torch.tensor(used)[torch.randint(0, len(used), (B,), generator=g)]
    tables = d.tensors(dtype, "cuda")
    x1d, x0d = x1.cuda().requires_grad_(True), x0.cuda().requires_grad_(True)

    def grads():
        out = fast_stc_uniform1d_jit(x1d, x0d, i0.cuda(), *tables, d.out_segs)
        return torch.autograd.grad(out, (x1d, x0d), r.cuda())

    gx1, gx0 = grads()
    want = stc_ref.stc_backward(r.double().numpy().reshape(B, d.out_segs, u), x1.double().numpy(), x0.double().numpy(), i0.numpy(),
                                d.paths, d.coeffs)
    for got, ref in zip((gx1, gx0), want):
        err = np.abs(got.cpu().double().numpy() - ref).max() / np.abs(ref).max()
        assert err <= tol, err
    idle = [s for s in range(S) if s not in used]
    assert not gx0[idle].any()
    assert torch.equal(gx0, grads()[1])


@pytest.mark.parametrize("n", [0, 1, 31, 33, 128, 1000, 8191, 8192, 8193])      # edges of a warp, of a CTA and of the counting form
@pytest.mark.parametrize("S", [1, 7, 5000])
def test_nodes_by_species(n, S):
    from fasteq_b200.ops.stc_uniform1d_jit import _by_species
    g = torch.Generator().manual_seed(n)
    species = torch.randint(0, S, (n,), generator=g, dtype=torch.int32)
    species[: n // 9] = torch.tensor([-5, 2**31 - 1, 0], dtype=torch.int32)[torch.arange(n // 9) % 3]
    species = species[torch.randperm(n, generator=g)].cuda()
    ascending, order = _by_species(species)
    want, nodes = torch.sort(species, stable=True)
    assert torch.equal(ascending, want) and torch.equal(order, nodes)


# two channels per thread (multiples of 64; 320: a CTA walks its channels in two turns), shares of several nodes and species, idle species
@pytest.mark.parametrize("u,B,S,used,offset", [(64, 5000, 4, [0, 1, 3], 0), (128, 9001, 12, list(range(1, 12)), 0), (320, 2500, 89, [0, 5, 7, 88], 0),
                                               (64, 700, 3, [0, 2], 1), (128, 3000, 3, [0, 1, 2], 1)])
def test_two_channels_per_thread(u, B, S, used, offset):
    """``offset`` 1: operands at an odd 4-byte address take the one-channel modules."""
    from fasteq_b200.ops import fast_stc_uniform1d_jit
    d = symmetric_contraction(f"{u}x0e+{u}x1o", f"{u}x0e+{u}x1o")
    g = torch.Generator().manual_seed(B)
    n = 150 if u == 320 else 400                                  # distinct nodes; the batch repeats them, which the oracle need not
    x1 = torch.randn(n, d.x1_segs, u, generator=g) * 0.3
    x0 = torch.randn(S, d.x0_segs, u, generator=g) * 0.1
    r = torch.randn(n, d.out_segs * u, generator=g)
    kind = torch.tensor(used)[torch.randint(0, len(used), (n,), generator=g)]
    pick = torch.randint(0, n, (B,), generator=g)

    def at(t):
        if not offset:
            return t.cuda()
        flat = torch.empty(t.numel() + 1, device="cuda")
        return flat[1:].view(t.shape).copy_(t)

    x1d, x0d, rd, i0 = at(x1[pick]).requires_grad_(True), at(x0).requires_grad_(True), at(r[pick]), kind[pick].cuda()
    assert x1d.data_ptr() % 8 == 4 * offset
    out = fast_stc_uniform1d_jit(x1d, x0d, i0, *d.tensors(torch.float32, "cuda"), d.out_segs)
    summed = torch.autograd.grad(out, (x1d, x0d), rd, retain_graph=True)
    per_node = torch.autograd.grad(out, (x1d, x0d), rd, create_graph=True)
    times = torch.bincount(pick, minlength=n).double().numpy()
    x1n, x0n, rn = x1.double().numpy(), x0.double().numpy(), r.double().numpy().reshape(n, d.out_segs, u)
    gx1, _ = stc_ref.stc_backward(rn, x1n, x0n, kind.numpy(), d.paths, d.coeffs)
    _, gx0 = stc_ref.stc_backward(rn * times[:, None, None], x1n, x0n, kind.numpy(), d.paths, d.coeffs)
    want = stc_ref.stc_forward(x1n, x0n, kind.numpy(), d.paths, d.coeffs, d.out_segs)
    close = lambda a, b: np.abs(a.detach().cpu().double().numpy().reshape(b.shape) - b).max() <= 1e-5 * np.abs(b).max()
    assert close(out, want[pick.numpy()])
    for got in (summed, per_node):
        assert close(got[0], gx1[pick.numpy()]) and close(got[1], gx0)
    assert not summed[1][[s for s in range(S) if s not in used]].any()
