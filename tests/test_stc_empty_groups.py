"""Symmetric-contraction tables in which a (weight, output) pair is left without a term: its only coefficient is zero, or the
coefficients of one monomial cancel.  Such a pair contributes nothing, in every generated kernel."""
import re

import numpy as np
import pytest
import torch

from fasteq_b200.codegen import stc as gen
from oracle import stc_ref

# weight 0 feeds outputs 0 and 1 (output 1 through terms that cancel), weight 1 feeds output 1 with a zero coefficient only,
# weight 2 feeds output 2 with cancelling cubic terms beside a live quadratic one, output 3 has no live term at all
PATHS = np.array([[0, 0, 0, -1, -1], [0, 1, 0, 1, -1], [1, 0, 0, 1, -1], [1, 1, 1, -1, -1],
                  [0, 1, 2, 2, 2], [2, 1, 0, 2, 2], [1, 2, 2, 2, -1], [2, 2, 2, 3, -1]])
COEFFS = np.array([1.0, 0.5, -0.5, 0.0, 0.25, -0.25, 0.75, 0.0])


def _spec(u, dtype="f32"):
    return gen.make_stc_spec(PATHS, COEFFS, x1_segs=3, x0_segs=3, out_segs=4, u=u, dtype=dtype)


@pytest.mark.parametrize("direction", ["fwd", "bwd", "bwdsum", "dbwd"])
@pytest.mark.parametrize("packed", [False, True])
def test_no_group_is_empty_and_every_sum_is_assigned_before_use(direction, packed):
    spec = _spec(64)
    if packed and not gen.packed_ok(spec, direction):
        pytest.skip("no packed form")
    assert set(gen._groups(spec)) == {(0, 0), (2, 2)} and all(gen._groups(spec).values())
    src = gen.emit_stc(spec, direction, direction in ("bwd", "bwdsum"), packed)
    for name, nxt in re.findall(r"\bV (r|s);\s*(\w+)", src):
        assert nxt == name, f"{name} is read before it is set"
    none = gen.make_stc_spec(PATHS[:1], [0.0], x1_segs=3, x0_segs=3, out_segs=4, u=64, dtype="f32")
    assert gen._groups(none) == {} and "V r;" not in gen.emit_stc(none, "fwd", packed=packed and direction == "fwd")


@pytest.mark.gpu
@pytest.mark.parametrize("dtype,tol", [(torch.float32, 1e-5), (torch.float64, 1e-11)])
@pytest.mark.parametrize("u", [16, 64])
def test_pairs_without_a_term_add_nothing(dtype, tol, u):
    from fasteq_b200.ops import fast_stc_uniform1d_jit
    g = torch.Generator().manual_seed(u)
    B, S = 70, 3
    x1 = torch.randn(B, 3, u, generator=g, dtype=torch.float64).to(dtype)
    x0 = torch.randn(S, 3, u, generator=g, dtype=torch.float64).to(dtype)
    r = torch.randn(B, 4 * u, generator=g, dtype=torch.float64).to(dtype)
    i0 = torch.randint(0, S, (B,), generator=g)
    paths = torch.from_numpy(PATHS).cuda()
    tables = (torch.from_numpy(COEFFS).to(dtype).cuda(), paths, paths.t().contiguous())
    x1d, x0d = x1.cuda().requires_grad_(True), x0.cuda().requires_grad_(True)
    out = fast_stc_uniform1d_jit(x1d, x0d, i0.cuda(), *tables, 4)
    a, b, n = x1.double().numpy(), x0.double().numpy(), i0.numpy()
    want = [stc_ref.stc_forward(a, b, n, PATHS, COEFFS, 4)]
    want += list(stc_ref.stc_backward(r.double().numpy().reshape(want[0].shape), a, b, n, PATHS, COEFFS))
    first = torch.autograd.grad(out, (x1d, x0d), r.cuda(), retain_graph=True)
    for got, ref in zip((out,) + first, want):
        assert np.abs(got.detach().cpu().double().numpy().reshape(ref.shape) - ref).max() <= tol * np.abs(ref).max()
    kept = torch.autograd.grad(out, (x1d, x0d), r.cuda(), create_graph=True)          # the per-node weight gradients
    for got, ref in zip(kept, want[1:]):
        assert np.abs(got.detach().cpu().double().numpy() - ref).max() <= tol * np.abs(ref).max()
    assert not out.detach().view(B, 4, u)[:, 3].any() and not first[1][:, 1].any()
