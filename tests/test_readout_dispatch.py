"""Which operands the one-launch readout takes; the others keep the elementwise expression's broadcast or its error."""
import pytest
import torch

from fasteq_b200.ops import readout


def test_operands_the_kernel_takes():
    h, w, e = torch.zeros(5, 8), torch.zeros(3), torch.zeros(5)
    assert readout._one_launch(h, w, None) and readout._one_launch(h, w, e)
    for bad in ((h, w.to("meta"), None), (h, w, e.to("meta")), (h, w, e[:1]), (h, w, e[:4]), (h, w, e.unsqueeze(1)),
                (h, w.unsqueeze(0), None), (h, w.double(), None), (h, w, e.double()), (h, torch.zeros(9), None),
                (h.t(), w, None), (h, torch.zeros(6)[::2], None), (h.half(), w.half(), None)):
        assert not readout._one_launch(*bad)


@pytest.mark.gpu
def test_other_operands_broadcast_or_raise():
    h, w, e = torch.randn(5, 8, device="cuda"), torch.randn(3, device="cuda"), torch.randn(1, device="cuda")
    want = (h[:, :3] * w).sum(-1) + e
    assert torch.equal(readout.scalar_readout(h, w, e), want)
    for bad in ((w.cpu(), None), (w, torch.randn(5)), (w, torch.randn(4, device="cuda"))):
        with pytest.raises(RuntimeError):
            readout.scalar_readout(h, *bad)
