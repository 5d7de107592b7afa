"""A thread that has done no CUDA work launches a tensor-core kernel first, all its memory taken from torch's cache (autograd's own thread
when a weight gradient opens the backward pass)."""
import threading

import pytest
import torch

pytestmark = pytest.mark.gpu


def _weight_gradient():
    from fasteq_b200.ops.dense import _matmul_tn
    g, x = (torch.randn(1000, 64, device="cuda") for _ in range(2))
    return lambda: _matmul_tn(g, x)


def _wide_layer():
    from fasteq_b200.ops.dense import dense
    x, w = torch.randn(1000, 64, device="cuda"), torch.randn(640, 64, device="cuda")
    return lambda: dense(x, w)


def _radial_layers():
    from fasteq_b200.ops.radial_chain import radial_chain
    b, ws = torch.randn(1000, 8, device="cuda"), [torch.randn(64, 8, device="cuda"), torch.randn(64, 64, device="cuda")]
    return lambda: radial_chain(b, ws)


@pytest.mark.parametrize("make", [_weight_gradient, _wide_layer, _radial_layers])
def test_first_cuda_work_of_a_thread(make):
    call, got = make(), []
    with torch.no_grad():
        want = call()
        for _ in range(3):          # outputs and scratch of the thread's call come from the cache
            call()
    torch.cuda.synchronize()

    def work():
        try:
            with torch.no_grad():
                got.append(call())
            torch.cuda.current_stream().synchronize()
        except Exception as e:
            got.append(e)

    t = threading.Thread(target=work)
    t.start()
    t.join()
    assert isinstance(got[0], torch.Tensor), got[0]
    assert torch.equal(got[0], want)
