"""Operators on a side stream: every launch goes to torch's current stream, and cached state built on one
stream (prepared weight forms, graph plans) is ordered before its first use on another."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _model_inputs(dtype=torch.float32):
    from fasteq_b200.graph import make_boxes
    b = make_boxes(2, [20, 14], [7.0, 6.5], 3.5, 3, seed=5)
    t = lambda a, dt=None: torch.from_numpy(a).cuda() if dt is None else torch.from_numpy(a).to(dt).cuda()
    return t(b.positions, dtype), (t(b.species), t(b.edge_src), t(b.edge_dst), t(b.edge_shift, dtype), t(b.node_graph), b.n_graphs)


def _same(e, f, e_ref, f_ref):
    # the position gradient is accumulated with floating-point atomics, so forces agree to rounding, not bit for bit
    return bool((e - e_ref).abs().max() <= 1e-6 * e_ref.abs().max()) and bool((f - f_ref).abs().max() <= 1e-5 * f_ref.abs().max())


def test_model_on_a_side_stream_matches_the_default_stream():
    from fasteq_b200.nn.mace_style import MACEStyleModel
    from fasteq_b200.ops import _prepared
    torch.manual_seed(0)
    model = MACEStyleModel(num_species=3, channels=32, r_max=3.5, avg_num_neighbors=12.0).cuda()
    for p in model.parameters():
        p.requires_grad_(False)
    pos, args = _model_inputs()
    ref = model(pos, *args)
    e_ref, f_ref = ref["energy"].clone(), ref["forces"].clone()
    torch.cuda.synchronize()
    side = torch.cuda.Stream()
    # (a) caches warm from the default stream, first use on the side stream
    with torch.cuda.stream(side):
        out = model(pos, *args)
        e1, f1 = out["energy"].clone(), out["forces"].clone()
    side.synchronize()
    assert _same(e1, f1, e_ref, f_ref)
    # (b) caches built on the side stream, next use on the default stream without a host sync in between
    _prepared.clear()
    from fasteq_b200.ops import uniform1d_jit
    uniform1d_jit._PLANS.clear()
    with torch.cuda.stream(side):
        out = model(pos, *args)
        e2, f2 = out["energy"].clone(), out["forces"].clone()
    out = model(pos, *args)
    e3, f3 = out["energy"].clone(), out["forces"].clone()
    torch.cuda.synchronize()
    assert _same(e2, f2, e_ref, f_ref)
    assert _same(e3, f3, e_ref, f_ref)


def test_operators_launch_on_the_current_stream():
    """A long kernel queued on the side stream first: an operator launched there afterwards must not have run
    ahead of it (it would if it went to the default stream), which shows in the value it reads."""
    from fasteq_b200.ops.dense import dense
    side = torch.cuda.Stream()
    x = torch.zeros(4096, 64, device="cuda")
    w = torch.eye(64, device="cuda")
    big = torch.randn(8192, 8192, device="cuda")
    torch.cuda.synchronize()
    with torch.cuda.stream(side):
        for _ in range(4):
            big = big @ big * 1e-4       # keeps the side stream busy
        x.fill_(3.0)                     # ordered behind the matmuls on the side stream
        y = dense(x, w)                  # must see the filled values
    side.synchronize()
    assert float(y.min()) == 3.0 and float(y.max()) == 3.0


def _operator(n=600, e=5000, seed=0):
    from fasteq_b200 import descriptors
    from fasteq_b200.irreps import Irreps
    sh = Irreps.spherical_harmonics(2)
    io, ins = descriptors.full_channelwise_instructions("32x0e+32x1o", sh, 2)
    d = descriptors.channelwise_tensor_product("32x0e+32x1o", sh, io, ins)
    g = torch.Generator(device="cuda").manual_seed(seed)
    src, dst = (torch.randint(0, n, (e,), generator=g, device="cuda", dtype=torch.int32) for _ in range(2))
    w, x, y = (torch.randn(*s, generator=g, device="cuda") for s in ((e, d.w_seg_num * 32), (n, d.x_seg_num * 32), (e, d.y_seg_num)))
    return src, dst, w, x, y, d.meta(torch.float32, "cuda")


def test_threads_share_a_plan_on_their_own_streams():
    """The partitions of a graph are built by whichever thread comes first and used by all: each stream waits for what others built."""
    import threading
    from fasteq_b200.ops import fast_uniform1d_jit, uniform1d_jit as u1d
    src, dst, w, x, y, meta = _operator()

    def step(index):
        ops = [t.detach().requires_grad_(True) for t in (w, x, y)]
        out = fast_uniform1d_jit(*ops, {1: src}, {0: index}, meta)
        return [out.detach(), *torch.autograd.grad(out, ops, torch.ones_like(out))]
    want = step(dst)
    for _ in range(10):
        index, got = dst.clone(), {}              # a plan of its own, whose partitions nobody has built
        u1d.graph_plan(index, x.shape[0])
        start = threading.Barrier(4)

        def work(k):
            with torch.cuda.stream(torch.cuda.Stream()) as _:
                torch.cuda.current_stream().wait_stream(torch.cuda.default_stream())
                start.wait()
                got[k] = step(index)
                torch.cuda.current_stream().synchronize()
        threads = [threading.Thread(target=work, args=(k,)) for k in range(4)]
        for t in threads:
            t.start()
        for t in threads:
            t.join()
        for k in range(4):
            for a, b in zip(got[k], want):         # the features' gradient is summed by atomics
                assert (a - b).norm() <= 1e-6 * b.norm()


def test_a_partition_first_needed_under_capture_stays_with_the_capture():
    """Its kernel is recorded, not run: a call outside, before any replay, must not find it."""
    from fasteq_b200.ops import fast_uniform1d_jit, uniform1d_jit as u1d
    src, dst, w, x, y, meta = _operator(e=1500)       # few edges a row: forwards keep whole receivers, backwards cut them
    ops = [t.requires_grad_(True) for t in (w, x, y)]
    go = torch.randn_like(fast_uniform1d_jit(*ops, {1: src}, {0: dst}, meta))

    def step(index):
        return torch.autograd.grad(fast_uniform1d_jit(*ops, {1: src}, {0: index}, meta), ops, go)
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        want = step(dst)                               # modules loaded, first-use allocations made
    index = dst.clone()
    with torch.no_grad():
        fast_uniform1d_jit(*ops, {1: src}, {0: index}, meta)
    plan = u1d.graph_plan(index, x.shape[0])
    kept = dict(plan._parts)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with u1d.record_plans() as plans, torch.cuda.graph(graph, stream=side):
        captured = step(index)
    assert plans == [plan] and plan._parts.keys() == kept.keys()
    for _ in range(2):
        for a, b in zip(step(index), want):
            assert (a - b).norm() <= 1e-6 * b.norm()   # the features' gradient is summed by atomics
        assert len(plan._parts) > len(kept)
        graph.replay()
        torch.cuda.synchronize()
        for a, b in zip(captured, want):
            assert (a - b).norm() <= 1e-6 * b.norm()


def test_prepared_weights_are_evicted_beside_threads_that_hold_the_gil():
    """A cached form that Python has seen takes the GIL when it goes, on autograd's thread too; other threads wait for the cache with the
    GIL in hand."""
    import threading
    from fasteq_b200.ops import _prepared
    from fasteq_b200.ops.dense import dense
    _prepared.set_budget(6 * 64 * 64 * 4)                 # three weights' forms
    done = []

    def work(seed):
        g = torch.Generator(device="cuda").manual_seed(seed)
        x = torch.randn(40, 64, device="cuda", generator=g, requires_grad=True)
        for _ in range(60):
            w = torch.randn(64, 64, device="cuda", generator=g)
            out = dense(x, w)
            _prepared.snapshot()
            (gx,) = torch.autograd.grad(out, x, torch.ones_like(out))     # prepares the transposed form: evicts
        want = w.double().sum(0)
        done.append(bool((gx.double() - want).abs().max() <= 2e-6 * want.abs().max() * 8))
    try:
        threads = [threading.Thread(target=work, args=(k,), daemon=True) for k in range(4)]
        for t in threads:
            t.start()
        for t in threads:
            t.join(60)
        assert done == [True] * 4
    finally:
        _prepared.set_budget(None)
        _prepared.clear()
