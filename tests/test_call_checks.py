"""What the kernels rely on and a caller may get wrong, or an autograd hook change: tensors on one device, upstream
gradients and saved tensors on a 16-byte boundary.  CPU, under the host emulation, which aborts where the GPU would fault."""
import pytest
import torch

from emu.emu import EmuLauncher
from flex_rnn_b200 import workloads as W
from flex_rnn_b200.twopass import build_twopass


def off(t):
    """The values of ``t``, contiguous, one element off a 16-byte boundary."""
    return torch.empty(t.numel() + 1, dtype=t.dtype)[1:].view(t.shape).copy_(t)


# fp32: the recurrent kernels; bf16 and 36 steps: the chunked ones (checkpoints and row sums are fp32 in both)
@pytest.mark.parametrize("op,dt,T", [("delta_rule", torch.float32, 9), ("mamba2", torch.float32, 9), ("delta_rule", torch.bfloat16, 36)])
def test_misaligned_upstream_gradients_and_saved_tensors(op, dt, T):
    *ins, s = W.synthetic(op, 1, T, 1, 32, 32, dt)[0]
    fwd, bwd, _, _ = build_twopass(W.STEPS[op], tuple(ins), (s,), _launcher=EmuLauncher)
    y, sT, ck, aux = fwd(tuple(ins), (s,))
    dy, dS = torch.randn(y.shape).to(y.dtype), torch.randn(sT.shape).to(sT.dtype)
    want = bwd((dy,), (dS,), tuple(ins), (ck,), (aux,))
    got = bwd((off(dy),), (off(dS),), tuple(ins), (off(ck),), (off(aux),))
    for a, b in zip([*got[0], *got[1]], [*want[0], *want[1]]):
        assert torch.allclose(a, b, rtol=1e-5, atol=0.0)      # equal, but for Mamba-2's A: nine terms added in any order
    with pytest.raises(RuntimeError, match="saved"):
        bwd((dy,), (dS,), tuple(ins), (ck[:, :, :, :1],), (aux,))


def test_tensors_on_another_device_are_refused():
    *ins, s = W.synthetic("delta_rule", 1, 9, 1, 32, 32, torch.float32)[0]
    fwd, bwd, _, _ = build_twopass(W.delta_rule, tuple(ins), (s,), _launcher=EmuLauncher)
    y, sT, ck, aux = fwd(tuple(ins), (s,))
    elsewhere = lambda ts, i: tuple(t.to("meta") if k == i else t for k, t in enumerate(ts))
    for bad in (lambda: fwd(elsewhere(ins, 1), (s,)), lambda: fwd.infer(elsewhere(ins, 3), (s,)), lambda: fwd(tuple(ins), (s.to("meta"),)),
                lambda: bwd((y.to("meta"),), (sT,), tuple(ins), (ck,), (aux,)), lambda: bwd((y,), (sT,), elsewhere(ins, 2), (ck,), (aux,)),
                lambda: bwd((y,), (sT,), tuple(ins), (ck.to("meta"),), (aux,))):
        with pytest.raises(RuntimeError, match="device"):
            bad()
