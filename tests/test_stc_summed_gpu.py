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
