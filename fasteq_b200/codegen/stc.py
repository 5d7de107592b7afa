"""CUDA source emitter for the symmetric tensor contraction (STC Uniform1D) kernels, sm_100a.

    out[b, v, u] = sum_p c_p * prod_t x1[b, a_{p,t}, u] * x0[i0[b], d_p, u]

One thread per node and channel -- per pair of adjacent channels in packed FP32 arithmetic where the channel count is a multiple
of 64 -- with the coefficients as literals, so the kernels are bound by FP32 issue and the emitter's job is to need few
instructions.  Forward: paths are grouped by (weight segment d, output segment v) and a cubic group is
``sum_c x_c * (sum c_p * (x_a x_b))`` with the singled-out factors chosen to cover many paths and the pair products shared by all
groups of an output segment.  The backward goes monomial by monomial instead (``_emit_grad_body``); it produces grad_x1 and, on
request, the weight gradient, either per node (second-order graphs) or summed over nodes of equal species.  The species gather
``x0[i0[b]]`` happens in the kernel (the reference materialises it with a torch gather first,
fasteq/ops/stc_uniform1d_jit.py:1016).  Counterpart of the reference's emitters
fasteq/ops/auto_schedule/stc_forward.py:158-340 and stc_backward.py:103-524.
"""
from __future__ import annotations

import hashlib
from dataclasses import dataclass
from typing import Dict, List, Tuple

import numpy as np

from .u1d_common import lit


@dataclass(frozen=True)
class STCSpec:
    paths: Tuple[Tuple[Tuple[int, ...], int, int, float], ...]   # (x1 indices, d, v, c)
    x1_segs: int
    x0_segs: int
    out_segs: int
    u: int
    dtype: str = "f32"

    def __hash__(self) -> int:
        # hashed once per object: the specification keys the module cache on every call and holds hundreds of paths
        h = self.__dict__.get("_hash")
        if h is None:
            h = hash((self.paths, self.x1_segs, self.x0_segs, self.out_segs, self.u, self.dtype))
            object.__setattr__(self, "_hash", h)
        return h

    def __getstate__(self):
        # another process hashes texts differently: a pickled copy computes its own
        return {k: v for k, v in self.__dict__.items() if k != "_hash"}

    @property
    def ctype(self) -> str:
        return "float" if self.dtype == "f32" else "double"

    def key(self, extra: str = "") -> str:
        h = hashlib.sha256()
        h.update(repr((self.paths, self.x1_segs, self.x0_segs, self.out_segs, self.u, self.dtype, extra)).encode())
        return h.hexdigest()[:16]


def make_stc_spec(paths, coeffs, *, x1_segs, x0_segs, out_segs, u, dtype, pad_value=-1) -> STCSpec:
    cs = np.asarray(coeffs, dtype=np.float64)
    if dtype == "f32":
        cs = cs.astype(np.float32).astype(np.float64)
    rows = []
    for row, c in zip(np.asarray(paths), cs):
        vals = [int(t) for t in row if int(t) != pad_value]
        if not 3 <= len(vals) <= 5:
            raise ValueError(f"bad STC path length {len(vals)}; expected 3..5")
        a, d, v = tuple(sorted(vals[:-2])), vals[-2], vals[-1]
        if not (all(0 <= t < x1_segs for t in a) and 0 <= d < x0_segs and 0 <= v < out_segs):
            raise ValueError("STC path index outside its operand's segment count")
        rows.append((a, d, v, float(c)))
    return STCSpec(tuple(rows), int(x1_segs), int(x0_segs), int(out_segs), int(u), dtype)


def _groups(spec: STCSpec):
    """{(d, v): {sorted index tuple: coefficient}} with duplicates merged.  Terms that cancel or have a zero coefficient are dropped,
    and with its last term the pair itself: the emitters start a pair's sum from its first term."""
    g: Dict[Tuple[int, int], Dict[Tuple[int, ...], float]] = {}
    for a, d, v, c in spec.paths:
        m = g.setdefault((d, v), {})
        m[a] = m.get(a, 0.0) + c
    live = {k: {a: c for a, c in m.items() if c != 0.0} for k, m in sorted(g.items())}
    return {k: m for k, m in live.items() if m}


def _cover(cubics, k: int, prefer=()):
    """Greedy cover of index triples by sub-multisets of ``k`` (1 or 2) of their factors: ``{factor(s): [triples]}``.  The
    fewest distinct sub-multisets means the fewest shared partial results; ties go to one in ``prefer``, then to the first."""
    subs = (lambda m: {(m[0],), (m[1],), (m[2],)}) if k == 1 else (lambda m: {(m[0], m[1]), (m[0], m[2]), (m[1], m[2])})
    left, out = sorted(cubics), {}
    while left:
        n: Dict[Tuple[int, ...], int] = {}
        for m in left:
            for t in subs(m):
                n[t] = n.get(t, 0) + 1
        best = min(n, key=lambda t: (-n[t], t not in prefer, t))
        out[best] = [m for m in left if best in subs(m)]
        left = [m for m in left if best not in subs(m)]
    return out


def _rest(mono: Tuple[int, ...], part: Tuple[int, ...]) -> Tuple[int, ...]:
    """The factors of a sorted monomial that ``part`` leaves."""
    r = list(mono)
    for t in part:
        r.remove(t)
    return tuple(r)


def _axpy(ind: str, acc: str, c: str, v: str, first: bool, decl: str = "") -> str:
    return f"{ind}{decl}{acc} = {c} * {v};" if first else f"{ind}{acc} = fma({c}, {v}, {acc});"


def _segment_scope(ind: str, v: int) -> str:
    """Opens the code of output segment ``v`` under a condition that always holds (there is at least one species) but is not
    known to: the compiler then forgets one segment's pair products before the next instead of keeping them for it, which
    took 164 registers instead of 64 forward (128-channel product basis) and kilobytes of spills in FP64."""
    return f"{ind}if (n_species > {-v}) {{"


def _emit_forward_body(groups, dt: str, ind: str) -> List[str]:
    """``o{v} += w[d] * P_dv(x)`` for every group.  Instructions: one per path, one per singled-out factor, one per pair
    product and output segment (1,006 multiplies and FMAs instead of 1,147 for the 550 paths of the 128-channel product basis as
    a nest over sorted index tuples, which shared prefixes only; about 950 after the compiler's common subexpressions).  Small
    terms and short sums come first: in index order the FP32 results were 0.5 % further from FP64 than the nest's (9.26e-8 and 9.22e-8
    of their norm), so they are 0.4 % nearer (9.18e-8), in the same time."""
    L: List[str] = []
    for v in sorted({v for _, v in groups}):
        plan, pairs = [], {}
        for d in (d for d, v2 in groups if v2 == v):
            mono = groups[(d, v)]
            singles = _cover([a for a in mono if len(a) == 3], 1)
            plan.append((d, mono, singles))
            for (c,), ms in singles.items():
                for m in ms:
                    pairs[_rest(m, (c,))] = None
            for a in mono:
                if len(a) == 2:
                    pairs[a] = None
        L.append(_segment_scope(ind, v))
        L += [f"{ind}  const V p{a}_{b} = x{a} * x{b};" for a, b in sorted(pairs)]
        for d, mono, singles in plan:
            L.append(f"{ind}  {{ V r;")
            first = True
            for a, c in sorted(mono.items(), key=lambda t: (abs(t[1]), t[0])):
                if len(a) < 3:
                    L.append(_axpy(ind + "    ", "r", lit(c, dt), f"x{a[0]}" if len(a) == 1 else f"p{a[0]}_{a[1]}", first))
                    first = False
            for (c1,), ms in sorted(singles.items(), key=lambda t: (len(t[1]), t[0])):
                L.append(f"{ind}    {{ V s;")
                for n, m in enumerate(sorted(ms, key=lambda m: (abs(mono[m]), m))):
                    a, b = _rest(m, (c1,))
                    L.append(_axpy(ind + "      ", "s", lit(mono[m], dt), f"p{a}_{b}", n == 0))
                L.append(_axpy(ind + "      ", "r", f"x{c1}", "s", first) + " }")
                first = False
            L.append(f"{ind}    o{v} = fma(LD(wp + {d} * U), r, o{v}); }}")
        L.append(f"{ind}}}")
    return L


def _emit_grad_body(groups, dt: str, ind: str, need_gw: bool) -> List[str]:
    """``ga{a} += d/dx_a`` and (``need_gw``) ``gw{d} += d/dw_d`` of ``sum go{v} w_d P_dv(x)``, monomial by monomial.

    The weights meet the cotangent first: ``C = sum_d c (w_d go_v)`` is a monomial's one coefficient whatever number of paths
    it stands in (410 distinct monomials for the 550 paths of the 128-channel product basis), a cubic one is
    ``C (x_a x_b) x_c`` and the pairs are chosen to cover many: ``S_ab += C x_c``, ``ga_c += C p_ab`` per monomial and
    ``ga_a += S_ab x_b``, ``ga_b += S_ab x_a`` once per pair.  The weight gradient needs the values ``P_dv`` on top: one
    product per monomial, one FMA per path.  1.8 k instructions per thread instead of 3.1 k for the nest run in reverse,
    2.7 k instead of 4.3 k with the weight gradient."""
    L: List[str] = []
    for v in sorted({v for _, v in groups}):
        mono: Dict[Tuple[int, ...], List[Tuple[int, float]]] = {}
        ds = [d for d, v2 in groups if v2 == v]
        for d in ds:
            for a, c in groups[(d, v)].items():
                mono.setdefault(a, []).append((d, c))
        quads = [a for a in sorted(mono) if len(a) == 2]
        pairs = _cover([a for a in mono if len(a) == 3], 2, prefer=quads)
        for a in quads:
            pairs.setdefault(a, [])
        L.append(_segment_scope(ind, v))
        L += [f"{ind}  const V g{d} = LD(wp + {d} * U) * go{v};" for d in ds]
        if need_gw:
            L += [f"{ind}  V P{d} = ZERO;" for d in ds]

        def coefficient(a, ind2):
            return [_axpy(ind2, "C", lit(c, dt), f"g{d}", n == 0, "V " if n == 0 else "") for n, (d, c) in enumerate(mono[a])]

        def value(a, name, ind2):
            return [f"{ind2}P{d} = fma({lit(c, dt)}, {name}, P{d});" for d, c in mono[a]] if need_gw else []

        for a in (a for a in sorted(mono) if len(a) == 1):
            L.append(f"{ind}  {{")
            L += coefficient(a, ind + "    ") + value(a, f"x{a[0]}", ind + "    ")
            L.append(f"{ind}    ga{a[0]} += C; }}")
        for (a, b), ms in sorted(pairs.items()):
            L.append(f"{ind}  {{ const V p = x{a} * x{b}; V S;")
            first = True
            if (a, b) in mono:
                L += [f"{ind}    {{"] + coefficient((a, b), ind + "      ") + value((a, b), "p", ind + "      ")
                L.append(f"{ind}      S = C; }}")
                first = False
            for m in ms:
                (c1,) = _rest(m, (a, b))
                L += [f"{ind}    {{"] + coefficient(m, ind + "      ")
                if need_gw:
                    L.append(f"{ind}      const V m = p * x{c1};")
                    L += value(m, "m", ind + "      ")
                L.append(_axpy(ind + "      ", "S", "C", f"x{c1}", first))
                L.append(f"{ind}      ga{c1} = fma(C, p, ga{c1}); }}")
                first = False
            L.append(f"{ind}    ga{a} = fma(S, x{b}, ga{a}); ga{b} = fma(S, x{a}, ga{b}); }}")
        if need_gw:
            L += [f"{ind}  gw{d} = fma(go{v}, P{d}, gw{d});" for d in ds]
        L.append(f"{ind}}}")
    return L


_COMMON = r"""
__device__ int g_status_word;
static thread_local char g_err[256];
static int cuda_fail(cudaError_t e) { snprintf(g_err, sizeof(g_err), "%s", cudaGetErrorString(e)); return FASTEQ_CUDA_ERROR; }
extern "C" const char* fasteq_last_cuda_error(void) { return g_err; }
extern "C" int fasteq_stc_device_status(int32_t* code) {
  if (!code) return FASTEQ_INVALID;
  int v = 0, zero = 0;
  cudaError_t e = cudaMemcpyFromSymbol(&v, g_status_word, sizeof(int));
  if (e != cudaSuccess) return cuda_fail(e);
  e = cudaMemcpyToSymbol(g_status_word, &zero, sizeof(int));
  if (e != cudaSuccess) return cuda_fail(e);
  *code = v;
  return FASTEQ_OK;
}
"""


def _emit_double_backward(spec: STCSpec, groups, dt: str) -> List[str]:
    """Second-order kernel: with ``t = ggx1`` and ``tw = ggx0`` (per node) the cotangents of the first
    backward's outputs, and ``m = prod x[a_i] * w`` one monomial,

        D     = d/d eps  m(x + eps t, w + eps tw)            d_go[v] += c D
        d_w  += c go[v] * dP                                 (dP = sum_i t[a_i] prod_{j != i} x[a_j])
        d_x[a_k] += c go[v] * (w * d(dP)/dx[a_k] + tw * dP/dx[a_k])

    Factors are handled by position, so repeated indices need no special case.  Straight-line code per
    monomial (no nesting): this kernel serves force-loss training, not the benchmarked inference path.
    Counterpart of fasteq/ops/stc_uniform1d_jit.py:964-968 (double-backward ``run(go, x1, x0, i0, ggx0, ggx1, V)``)."""
    L: List[str] = [f"""
__global__ void __launch_bounds__(NT) fasteq_stc_dbwd_kernel(const T* __restrict__ go, const T* __restrict__ x1,
    const T* __restrict__ x0, const int* __restrict__ i0, const T* __restrict__ ggx1, const T* __restrict__ ggx0n,
    long long batch, long long n_species, T* __restrict__ d_go, T* __restrict__ d_x1, T* __restrict__ d_x0n, int* status) {{
  for (long long b = blockIdx.x; b < batch; b += gridDim.x) {{
    int sp = i0[b];
    if (sp < 0 || sp >= n_species) {{ atomicExch(status, 2); sp = 0; }}
    for (int u = threadIdx.x; u < U; u += NT) {{
      const T* xp = x1 + (size_t)b * A * U + u;
      const T* tp = ggx1 + (size_t)b * A * U + u;
      const T* wp = x0 + (size_t)sp * D * U + u;
      const T* twp = ggx0n + (size_t)b * D * U + u;
      const T* gp = go + (size_t)b * OSEG * U + u;"""]
    L += [f"      const T x{a} = xp[{a} * U], t{a} = tp[{a} * U];" for a in range(spec.x1_segs)]
    L += [f"      const T go{v} = gp[{v} * U];" for v in range(spec.out_segs)]
    L += [f"      T dx{a} = T(0);" for a in range(spec.x1_segs)]
    L += [f"      T dg{v} = T(0);" for v in range(spec.out_segs)]
    by_d: Dict[int, List[int]] = {}
    for (d, v) in groups:
        by_d.setdefault(d, []).append(v)
    for d, vs in by_d.items():
        L.append(f"      {{ const T w = wp[{d} * U], tw = twp[{d} * U]; T dw = T(0);")
        for v in vs:
            for a, c in sorted(groups[(d, v)].items()):
                cl = lit(c, dt)
                n = len(a)
                L.append(f"        {{ const T cg = {cl} * go{v};")
                if n == 1:
                    (p,) = a
                    L.append(f"          dg{v} = fma({cl}, fma(t{p}, w, x{p} * tw), dg{v}); dw = fma(cg, t{p}, dw); dx{p} = fma(cg, tw, dx{p}); }}")
                elif n == 2:
                    p, q = a
                    L.append(f"          const T P = x{p} * x{q}, dP = fma(t{p}, x{q}, x{p} * t{q});")
                    L.append(f"          dg{v} = fma({cl}, fma(dP, w, P * tw), dg{v}); dw = fma(cg, dP, dw);")
                    L.append(f"          dx{p} = fma(cg, fma(w, t{q}, tw * x{q}), dx{p}); dx{q} = fma(cg, fma(w, t{p}, tw * x{p}), dx{q}); }}")
                else:
                    p, q, r = a
                    L.append(f"          const T pq = x{p} * x{q}, pr = x{p} * x{r}, qr = x{q} * x{r};")
                    L.append(f"          const T P = pq * x{r}, dP = fma(t{p}, qr, fma(t{q}, pr, t{r} * pq));")
                    L.append(f"          dg{v} = fma({cl}, fma(dP, w, P * tw), dg{v}); dw = fma(cg, dP, dw);")
                    L.append(f"          dx{p} = fma(cg, fma(w, fma(t{q}, x{r}, x{q} * t{r}), tw * qr), dx{p});")
                    L.append(f"          dx{q} = fma(cg, fma(w, fma(t{p}, x{r}, x{p} * t{r}), tw * pr), dx{q});")
                    L.append(f"          dx{r} = fma(cg, fma(w, fma(t{p}, x{q}, x{p} * t{q}), tw * pq), dx{r}); }}")
        L.append(f"        d_x0n[((size_t)b * D + {d}) * U + u] = dw; }}")
    for d in range(spec.x0_segs):
        if d not in by_d:
            L.append(f"      d_x0n[((size_t)b * D + {d}) * U + u] = T(0);")
    L.append("      T* dxp = d_x1 + (size_t)b * A * U + u;")
    L += [f"      dxp[{a} * U] = dx{a};" for a in range(spec.x1_segs)]
    L.append("      T* dgp = d_go + (size_t)b * OSEG * U + u;")
    L += [f"      dgp[{v} * U] = dg{v};" for v in range(spec.out_segs)]
    L.append("    }\n  }\n}")
    L.append("""
extern "C" int fasteq_stc_forward(const void*, const void*, const int32_t*, int64_t, int64_t, void*, fasteq_stream_t) {
  return FASTEQ_UNSUPPORTED;  // double-backward module
}
extern "C" int fasteq_stc_backward(const void*, const void*, const void*, const int32_t*, int64_t, int64_t, void*, void*, fasteq_stream_t) {
  return FASTEQ_UNSUPPORTED;  // double-backward module
}
extern "C" int fasteq_stc_double_backward(const void* go, const void* x1, const void* x0, const int32_t* i0, const void* ggx1,
                                          const void* ggx0_per_node, int64_t batch, int64_t n_species, void* d_go, void* d_x1,
                                          void* d_x0_per_node, fasteq_stream_t stream) {
  if (batch < 0 || n_species < 0) return FASTEQ_INVALID;
  if (batch == 0) return FASTEQ_OK;
  if (!go || !x1 || !x0 || !i0 || !ggx1 || !ggx0_per_node || !d_go || !d_x1 || !d_x0_per_node) return FASTEQ_INVALID;
  int* st = nullptr;
  cudaError_t e = cudaGetSymbolAddress((void**)&st, g_status_word);
  if (e != cudaSuccess) return cuda_fail(e);
  const long long grid = batch < (1LL << 30) ? batch : (1LL << 30);
  fasteq_stc_dbwd_kernel<<<(unsigned)grid, NT, 0, (cudaStream_t)stream>>>((const T*)go, (const T*)x1, (const T*)x0, i0, (const T*)ggx1,
      (const T*)ggx0_per_node, batch, n_species, (T*)d_go, (T*)d_x1, (T*)d_x0_per_node, st);
  e = cudaGetLastError();
  return e == cudaSuccess ? FASTEQ_OK : cuda_fail(e);
}""")
    return L


def _emit_summed_backward(spec: STCSpec, groups, dt: str) -> List[str]:
    """Backward with the weight gradient already summed over nodes of equal species.

    Bound: FP32 issue (``_emit_grad_body``).  Writing ``[batch, D, U]`` per-node weight gradients and adding them up by
    species afterwards cost twice the arithmetic: 3 GB out, 3 GB back in and one atomic per value at 200 k nodes.  Here the
    nodes come in species order (``order``, a stable sort), a CTA walks one contiguous share of it and keeps the D sums of its
    channel in registers; they go out once per (CTA, species) pair.  Along the order either the CTA or the species grows from
    one pair to the next, so ``CTA + species`` is a slot of its own and ``n_parts + n_species`` rows of partial sums do.  A
    second kernel adds each species' slots in a fixed order: the result does not depend on scheduling."""
    L: List[str] = [f"""
__global__ void __launch_bounds__(NT) fasteq_stc_bwd_sum_kernel(const T* __restrict__ go, const T* __restrict__ x1,
    const T* __restrict__ x0, const long long* __restrict__ order, const int* __restrict__ species, long long batch,
    long long n_species, T* __restrict__ gx1, T* __restrict__ partial, int* status) {{
  const long long lo = batch * blockIdx.x / gridDim.x, hi = batch * (blockIdx.x + 1) / gridDim.x;
  for (int u = threadIdx.x * VEC; u < U; u += NT * VEC) {{
    int cur = -1;                                      // species whose sums are in the registers"""]
    L += [f"    V gw{d} = ZERO;" for d in range(spec.x0_segs)]
    L.append("    for (long long i = lo; i <= hi; ++i) {")
    L.append("      const int sp = i < hi ? species[i] : -1;")
    L.append("      if (sp != cur) {")
    L.append("        if (cur >= 0 && cur < n_species) {")
    L.append("          T* pp = partial + ((size_t)blockIdx.x + cur) * D * U + u;")
    L += [f"          ST(pp + {d} * U, gw{d});" for d in range(spec.x0_segs)]
    L.append("        }")
    L += [f"        gw{d} = ZERO;" for d in range(spec.x0_segs)]
    L.append("        cur = sp;")
    L.append("      }")
    L.append("      if (i == hi) break;")
    L.append("      // a species out of range is reported, differentiates as species 0 and adds to no weight gradient")
    L.append("      if (sp < 0 || sp >= n_species) atomicExch(status, 2);")
    L.append("      const size_t b = (size_t)order[i];")
    L.append("      const T* xp = x1 + b * A * U + u;")
    L.append("      const T* wp = x0 + (size_t)(sp < 0 || sp >= n_species ? 0 : sp) * D * U + u;")
    L.append("      const T* gp = go + b * OSEG * U + u;")
    L += [f"      const V x{a} = LD(xp + {a} * U);" for a in range(spec.x1_segs)]
    L += [f"      const V go{v} = LD(gp + {v} * U);" for v in range(spec.out_segs)]
    L += [f"      V ga{a} = ZERO;" for a in range(spec.x1_segs)]
    L += _emit_grad_body(groups, dt, "      ", True)
    L.append("      T* gxp = gx1 + b * A * U + u;")
    L += [f"      ST(gxp + {a} * U, ga{a});" for a in range(spec.x1_segs)]
    L.append("    }\n  }\n}")
    L.append(r"""
// gx0[s][d][u] = sum of the partial sums of species s, for 32 channels and DS weights per CTA.  Bound by latency: the CTA looks the
// species' nodes up together (256 positions at a time; two binary searches were twenty loads one after the other, 35 us of
// a 67 us backward with 89 species), and few sums go one after the other in a thread per (channel, weight) while many go in eight
// interleaved shares, with the same additions in the same order where both apply (the launch takes eight weights per CTA where a
// species has about eight sums at most).
template <int DS>
__global__ void __launch_bounds__(256) fasteq_stc_sum_parts_kernel(const int* __restrict__ species, const T* __restrict__ partial,
    long long batch, int n_parts, T* __restrict__ gx0) {
  __shared__ T share[8][33];
  constexpr int GROUPS = (D + DS - 1) / DS;
  const int s = blockIdx.x / GROUPS, d0 = blockIdx.x % GROUPS * DS, u = blockIdx.y * 32 + threadIdx.x;
  const int tid = threadIdx.y * 32 + threadIdx.x;
  long long bound[2];                                  // first positions of species s and s + 1 in the order
  for (int e = 0; e < 2; ++e) {
    long long a = e ? bound[0] : 0, n = batch - a;     // the answer is one of a .. a + n
    while (n > 0) {
      const long long step = (n + 255) / 256, at = tid * step;
      const int below = __syncthreads_count(at < n && species[at < n ? a + at : a] < s + e);      // a prefix of the probes
      if (below == 0) break;
      const long long next = (long long)(below - 1) * step + 1, left = n - next;
      a += next; n = left < step - 1 ? left : step - 1;
    }
    bound[e] = a;
  }
  const bool any = bound[0] < bound[1];
  // the CTA of position i is the largest c with floor(batch * c / n_parts) <= i
  const long long first = any ? ((bound[0] + 1) * n_parts - 1) / batch : 0, last = any ? (bound[1] * n_parts - 1) / batch : -1;
  if (DS == 8 && last - first < 8) {
    const int d = d0 + threadIdx.y;
    if (d >= D || u >= U) return;
    T sum = T(0);
#pragma unroll 8
    for (long long c = first; c <= last; ++c) sum += partial[((size_t)(c + s) * D + d) * U + u];
    gx0[((size_t)s * D + d) * U + u] = sum;
    return;
  }
  for (int d = d0; d < D && d < d0 + DS; ++d) {
    T sum = T(0);
    if (u < U)
      for (long long c = first + threadIdx.y; c <= last; c += 8) sum += partial[((size_t)(c + s) * D + d) * U + u];
    share[threadIdx.y][threadIdx.x] = sum;
    __syncthreads();
    if (threadIdx.y == 0 && u < U) {
#pragma unroll
      for (int k = 1; k < 8; ++k) sum += share[k][threadIdx.x];
      gx0[((size_t)s * D + d) * U + u] = sum;
    }
    if (DS > 1) __syncthreads();
  }
}

extern "C" int fasteq_stc_forward(const void*, const void*, const int32_t*, int64_t, int64_t, void*, fasteq_stream_t) {
  return FASTEQ_UNSUPPORTED;  // summed-backward module
}
extern "C" int fasteq_stc_backward(const void*, const void*, const void*, const int32_t*, int64_t, int64_t, void*, void*, fasteq_stream_t) {
  return FASTEQ_UNSUPPORTED;  // summed-backward module
}
extern "C" int fasteq_stc_double_backward(const void*, const void*, const void*, const int32_t*, const void*, const void*, int64_t,
                                          int64_t, void*, void*, void*, fasteq_stream_t) {
  return FASTEQ_UNSUPPORTED;  // this module holds another direction
}
// the CTAs one wave holds: every share of the order then runs at once
extern "C" int fasteq_stc_backward_summed_parts(int64_t batch, int32_t* n_parts) {
  if (batch < 0 || !n_parts) return FASTEQ_INVALID;
  int dev = 0, sms = 0, per = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, fasteq_stc_bwd_sum_kernel, NT, 0);
  if (e != cudaSuccess) return cuda_fail(e);
  const int64_t wave = (int64_t)sms * (per > 0 ? per : 1);
  *n_parts = (int32_t)(batch < wave ? (batch < 1 ? 1 : batch) : wave);
  return FASTEQ_OK;
}
extern "C" int fasteq_stc_backward_summed(const void* go, const void* x1, const void* x0, const int64_t* order,
                                          const int32_t* species_sorted, int64_t batch, int64_t n_species, int32_t n_parts,
                                          void* partial, void* gx1, void* gx0, fasteq_stream_t stream) {
  if (batch < 0 || n_species < 0 || n_parts < 1 || n_species > 0x7fffffffLL / D) return FASTEQ_INVALID;
  cudaStream_t s = (cudaStream_t)stream;
  if (batch == 0) {
    if (n_species > 0 && !gx0) return FASTEQ_INVALID;
    cudaError_t e = n_species > 0 ? cudaMemsetAsync(gx0, 0, (size_t)n_species * D * U * sizeof(T), s) : cudaSuccess;
    return e == cudaSuccess ? FASTEQ_OK : cuda_fail(e);
  }
  if (n_species == 0 || !go || !x1 || !x0 || !order || !species_sorted || !partial || !gx1 || !gx0) return FASTEQ_INVALID;
  if (n_parts > batch) return FASTEQ_INVALID;        // an empty share writes no slot, but the second kernel would add it
  if (misaligned(go, x1, x0, partial, gx1)) return FASTEQ_INVALID;
  int* st = nullptr;
  cudaError_t e = cudaGetSymbolAddress((void**)&st, g_status_word);
  if (e != cudaSuccess) return cuda_fail(e);
  fasteq_stc_bwd_sum_kernel<<<(unsigned)n_parts, NT, 0, s>>>((const T*)go, (const T*)x1, (const T*)x0, (const long long*)order,
                                                             species_sorted, batch, n_species, (T*)gx1, (T*)partial, st);
  if (n_parts + n_species <= 8 * n_species)
    fasteq_stc_sum_parts_kernel<8><<<dim3((unsigned)(n_species * ((D + 7) / 8)), (U + 31) / 32), dim3(32, 8), 0, s>>>(
        species_sorted, (const T*)partial, batch, n_parts, (T*)gx0);
  else
    fasteq_stc_sum_parts_kernel<1><<<dim3((unsigned)(n_species * D), (U + 31) / 32), dim3(32, 8), 0, s>>>(
        species_sorted, (const T*)partial, batch, n_parts, (T*)gx0);
  e = cudaGetLastError();
  return e == cudaSuccess ? FASTEQ_OK : cuda_fail(e);
}
""")
    return L


def packed_ok(spec: STCSpec, direction: str) -> bool:
    """Whether a thread may carry two channels in packed FP32 arithmetic (full warps of pairs; operands 8-byte aligned).  The
    scalar kernels issued in 84 % (forward) and 67 % (backward with the weight gradient, whose 42 KB of straight-line code also
    waits for instructions) of their cycles; packed ones need half the slots and half the code per channel: 128-channel product
    basis on 200,000 nodes, forward 0.96 -> 0.81 ms, backward 2.79 -> 2.49 ms."""
    return spec.dtype == "f32" and spec.u % 64 == 0 and direction != "dbwd"


_SCALAR = """typedef T V;             // what a thread carries per segment
constexpr int VEC = 1;
#define LD(p) (*(p))
#define ST(p, v) (*(p) = (v))
#define ZERO T(0)
template <typename... P> static bool misaligned(P...) { return false; }
"""

_PACKED = """typedef float2 V;        // what a thread carries per segment: two channels
constexpr int VEC = 2;
#define LD(p) (*reinterpret_cast<const float2*>(p))
#define ST(p, v) (*reinterpret_cast<float2*>(p) = (v))
#define ZERO make_float2(0.f, 0.f)
__device__ __forceinline__ V operator*(V a, V b) { return fasteq::vmul(a, b); }
__device__ __forceinline__ V operator*(float c, V b) { return fasteq::vmul(make_float2(c, c), b); }
__device__ __forceinline__ V fma(V a, V b, V c) { return fasteq::vfma(a, b, c); }
__device__ __forceinline__ V fma(float a, V b, V c) { return fasteq::vfma(make_float2(a, a), b, c); }
__device__ __forceinline__ void operator+=(V& a, V b) { a = fasteq::vadd(a, b); }
template <typename... P> static bool misaligned(P... p) { return ((reinterpret_cast<uintptr_t>(p) | ...) & 7u) != 0; }
"""

_NOT_SUMMED = r"""
extern "C" int fasteq_stc_backward_summed_parts(int64_t, int32_t*) { return FASTEQ_UNSUPPORTED; }
extern "C" int fasteq_stc_backward_summed(const void*, const void*, const void*, const int64_t*, const int32_t*, int64_t, int64_t, int32_t,
                                          void*, void*, void*, fasteq_stream_t) {
  return FASTEQ_UNSUPPORTED;  // the module of direction 3 holds these
}
"""


def emit_stc(spec: STCSpec, direction: str, need_gx0: bool = False, packed: bool = False) -> str:
    dt = spec.dtype
    groups = _groups(spec)
    if packed and not packed_ok(spec, direction):
        raise ValueError("packed arithmetic needs FP32, a multiple of 64 channels and a first-order kernel")
    threads = min(((spec.u // 2 if packed else spec.u) + 31) // 32 * 32, 128)
    head = f"""// Generated by fasteq_b200.codegen.stc -- do not edit.
#include <cstdio>
#include <cstdint>
#include <cuda_runtime.h>
#include "fasteq_b200.h"
#include "fasteq_device.cuh"
typedef {spec.ctype} T;
constexpr int U = {spec.u}, A = {spec.x1_segs}, D = {spec.x0_segs}, OSEG = {spec.out_segs}, NT = {threads};
{_PACKED if packed else _SCALAR}{_COMMON}
extern "C" int fasteq_stc_describe(fasteq_stc_desc* d) {{
  if (!d) return FASTEQ_INVALID;
  d->abi_version = FASTEQ_ABI_VERSION; d->dtype = {0 if dt == 'f32' else 1}; d->u = U; d->x1_segs = A; d->x0_segs = D;
  d->out_segs = OSEG; d->num_paths = {len(spec.paths)}; d->direction = {dict(fwd=0, bwd=1, dbwd=2, bwdsum=3)[direction]}; d->need_gx0 = {int(need_gx0)};
  return FASTEQ_OK;
}}
"""
    body: List[str] = []
    if direction == "fwd":
        body.append(f"""
__global__ void __launch_bounds__(NT) fasteq_stc_fwd_kernel(const T* __restrict__ x1, const T* __restrict__ x0,
    const int* __restrict__ i0, long long batch, long long n_species, T* __restrict__ out, int* status) {{
  fasteq::let_next_kernel_begin();
  for (long long b = blockIdx.x; b < batch; b += gridDim.x) {{
    int sp = i0[b];
    if (sp < 0 || sp >= n_species) {{ atomicExch(status, 2); sp = 0; }}
    for (int u = threadIdx.x * VEC; u < U; u += NT * VEC) {{
      const T* xp = x1 + (size_t)b * A * U + u;
      const T* wp = x0 + (size_t)sp * D * U + u;""")
        body += [f"      const V x{a} = LD(xp + {a} * U);" for a in range(spec.x1_segs)]
        body += [f"      V o{v} = ZERO;" for v in range(spec.out_segs)]
        body += _emit_forward_body(groups, dt, "      ")
        body.append("      T* op = out + (size_t)b * OSEG * U + u;")
        body += [f"      ST(op + {v} * U, o{v});" for v in range(spec.out_segs)]
        body.append("    }\n  }\n}")
        body.append("""
extern "C" int fasteq_stc_forward(const void* x1, const void* x0, const int32_t* i0, int64_t batch, int64_t n_species,
                                  void* out, fasteq_stream_t stream) {
  if (batch < 0 || n_species < 0) return FASTEQ_INVALID;
  if (batch == 0) return FASTEQ_OK;
  if (!x1 || !x0 || !i0 || !out || misaligned(x1, x0, out)) return FASTEQ_INVALID;
  int* st = nullptr;
  cudaError_t e = cudaGetSymbolAddress((void**)&st, g_status_word);
  if (e != cudaSuccess) return cuda_fail(e);
  const long long grid = batch < (1LL << 30) ? batch : (1LL << 30);
  fasteq_stc_fwd_kernel<<<(unsigned)grid, NT, 0, (cudaStream_t)stream>>>((const T*)x1, (const T*)x0, i0, batch, n_species, (T*)out, st);
  e = cudaGetLastError();
  return e == cudaSuccess ? FASTEQ_OK : cuda_fail(e);
}
extern "C" int fasteq_stc_backward(const void*, const void*, const void*, const int32_t*, int64_t, int64_t, void*, void*, fasteq_stream_t) {
  return FASTEQ_UNSUPPORTED;  // forward module
}
extern "C" int fasteq_stc_double_backward(const void*, const void*, const void*, const int32_t*, const void*, const void*, int64_t,
                                          int64_t, void*, void*, void*, fasteq_stream_t) {
  return FASTEQ_UNSUPPORTED;  // this module holds another direction
}
""")
    elif direction == "dbwd":
        body += _emit_double_backward(spec, groups, dt)
    elif direction == "bwdsum":
        body += _emit_summed_backward(spec, groups, dt)
    else:
        body.append(f"""
constexpr bool NEED_GX0 = {str(need_gx0).lower()};
__global__ void __launch_bounds__(NT) fasteq_stc_bwd_kernel(const T* __restrict__ go, const T* __restrict__ x1,
    const T* __restrict__ x0, const int* __restrict__ i0, long long batch, long long n_species, T* __restrict__ gx1,
    T* __restrict__ gx0n, int* status) {{
  fasteq::let_next_kernel_begin();
  for (long long b = blockIdx.x; b < batch; b += gridDim.x) {{
    int sp = i0[b];
    if (sp < 0 || sp >= n_species) {{ atomicExch(status, 2); sp = 0; }}
    for (int u = threadIdx.x * VEC; u < U; u += NT * VEC) {{
      const T* xp = x1 + (size_t)b * A * U + u;
      const T* wp = x0 + (size_t)sp * D * U + u;
      const T* gp = go + (size_t)b * OSEG * U + u;""")
        body += [f"      const V x{a} = LD(xp + {a} * U);" for a in range(spec.x1_segs)]
        body += [f"      const V go{v} = LD(gp + {v} * U);" for v in range(spec.out_segs)]
        body += [f"      V ga{a} = ZERO;" for a in range(spec.x1_segs)]
        if need_gx0:
            body += [f"      V gw{d} = ZERO;" for d in range(spec.x0_segs)]
        body += _emit_grad_body(groups, dt, "      ", need_gx0)
        if need_gx0:
            body += [f"      ST(gx0n + ((size_t)b * D + {d}) * U + u, gw{d});" for d in range(spec.x0_segs)]
        body.append("      T* gxp = gx1 + (size_t)b * A * U + u;")
        body += [f"      ST(gxp + {a} * U, ga{a});" for a in range(spec.x1_segs)]
        body.append("    }\n  }\n}")
        body.append("""
extern "C" int fasteq_stc_forward(const void*, const void*, const int32_t*, int64_t, int64_t, void*, fasteq_stream_t) {
  return FASTEQ_UNSUPPORTED;  // backward module
}
extern "C" int fasteq_stc_backward(const void* go, const void* x1, const void* x0, const int32_t* i0, int64_t batch,
                                   int64_t n_species, void* gx1, void* gx0_per_node, fasteq_stream_t stream) {
  if (batch < 0 || n_species < 0) return FASTEQ_INVALID;
  if (batch == 0) return FASTEQ_OK;
  if (!go || !x1 || !x0 || !i0 || !gx1 || (NEED_GX0 && !gx0_per_node)) return FASTEQ_INVALID;
  if (misaligned(go, x1, x0, gx1, gx0_per_node)) return FASTEQ_INVALID;
  int* st = nullptr;
  cudaError_t e = cudaGetSymbolAddress((void**)&st, g_status_word);
  if (e != cudaSuccess) return cuda_fail(e);
  const long long grid = batch < (1LL << 30) ? batch : (1LL << 30);
  fasteq_stc_bwd_kernel<<<(unsigned)grid, NT, 0, (cudaStream_t)stream>>>((const T*)go, (const T*)x1, (const T*)x0, i0, batch,
                                                                        n_species, (T*)gx1, (T*)gx0_per_node, st);
  e = cudaGetLastError();
  return e == cudaSuccess ? FASTEQ_OK : cuda_fail(e);
}
extern "C" int fasteq_stc_double_backward(const void*, const void*, const void*, const int32_t*, const void*, const void*, int64_t,
                                          int64_t, void*, void*, void*, fasteq_stream_t) {
  return FASTEQ_UNSUPPORTED;  // this module holds another direction
}
""")
    return head + "\n".join(body) + "\n" + (_NOT_SUMMED if direction != "bwdsum" else "")


def arith_ops(spec: STCSpec, direction: str, need_gx0: bool = False) -> Dict[str, int]:
    """Floating-point instructions one (node, channel) thread executes in the generated kernel, counted in its
    source text: ``fma(...)`` calls and explicit multiplications (the kernel body is straight-line code, so the
    count is the executed count).  Used to state the kernels' FP32-issue utilisation."""
    import re
    src = emit_stc(spec, direction, need_gx0)
    body = src[src.index("__global__"):]
    end = body.find('extern "C"')
    body = body[:end if end > 0 else len(body)]
    body = re.sub(r"//[^\n]*", "", body)
    body = re.sub(r"\b(LD|ST)\([^,;]*?\* U", r"\1(", body)                     # address arithmetic
    body = re.sub(r"\[[^\]]*\]", "[]", body)                                   # subscripts hold index arithmetic only
    body = "\n".join(ln for ln in body.splitlines() if "size_t" not in ln and "const T*" not in ln)
    fma = len(re.findall(r"\bfma\(", body))
    mul = len(re.findall(r"\s\*\s", body)) - len(re.findall(r"\b1\.0f? \* ", body))   # x * 1.0 is folded away by the compiler
    return {"fma": fma, "mul": mul}
