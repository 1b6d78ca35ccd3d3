"""What the kernels rely on and a caller may get wrong, or an autograd hook change: tensors on one device.  CPU, under the
host emulation, which aborts where the GPU would fault."""
import pytest
import torch

from emu.emu import EmuLauncher
from flex_rnn_b200 import workloads as W
from flex_rnn_b200.twopass import build_twopass


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
