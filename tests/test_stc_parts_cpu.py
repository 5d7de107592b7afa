"""The summed backward of the symmetric contraction refuses more shares than nodes: an empty share writes no partial sums,
and the second pass would add what happens to be in its slot."""
import ctypes as C

from fasteq_b200.descriptors import symmetric_contraction
from fasteq_b200.codegen.stc import make_stc_spec
from fasteq_b200.ops import stc_uniform1d_jit as stc


def test_more_shares_than_nodes_are_refused():
    d = symmetric_contraction("32x0e", "32x0e")
    spec = make_stc_spec(d.paths, d.coeffs, x1_segs=d.x1_segs, x0_segs=d.x0_segs, out_segs=d.out_segs, u=32, dtype="f32")
    lib = stc.get_module(spec, "bwdsum", True).lib
    p = C.create_string_buffer(64)                              # never read: the call is refused before any launch
    a = C.addressof(p) // 8 * 8 + 8
    for batch, parts in ((4, 5), (1, 2), (1, 1000), (4, 0)):
        assert lib.fasteq_stc_backward_summed(a, a, a, a, a, batch, 1, parts, a, a, a, None) == 2
