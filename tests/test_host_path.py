"""The native host path of an eager call (csrc/frnn_host.cpp) and the kernels of calls without gradients: same
results as the custom op, whatever the call looks like."""
import contextlib
import threading
import time

import pytest
import torch

import flex_rnn_b200
from flex_rnn_b200 import examples as X
from flex_rnn_b200 import workloads as W
from flex_rnn_b200.twopass import Tuning, build_twopass


@pytest.mark.parametrize("op", ["delta_rule", "mamba2", "gla"])
@pytest.mark.parametrize("T", [1, 7, 19])
def test_emulated_forward_without_gradients(op, T):
    """The kernel that saves nothing gives the outputs and final states of the one that does."""
    from emu.emu import EmuLauncher
    if op in W.STEPS:
        *ins, s0 = W.synthetic(op, 1, T, 2, 16, 16, torch.float32)[0]
        ins, sts, step = ins, [s0], W.STEPS[op]
    else:
        (ins, sts), step = X.zoo_case(op, 1, T, 2, 16, 16), X.ZOO[op]
    tu = Tuning(fw_r=2, fw_c=4, fw_mb=16, fw_stage=min(4, T), bw_r=2, bw_c=4, seg=min(2, T), nslots=2 if T > 3 else 1)
    fwd, _, _, _ = build_twopass(step, tuple(ins), tuple(sts), tuning=tu, _launcher=EmuLauncher)
    full, short = fwd(tuple(ins), tuple(sts)), fwd.infer(tuple(ins), tuple(sts))
    assert len(short) == 2 and all(torch.equal(a, b) for a, b in zip(short, full))


@pytest.mark.gpu
@pytest.mark.parametrize("op,B,T,M,N,dt", [("delta_rule", 2, 33, 64, 64, torch.float32), ("mamba2", 2, 17, 32, 64, torch.bfloat16),
                                           ("gated_delta_rule", 3, 1, 64, 128, torch.bfloat16), ("rwkv7", 1, 40, 24, 40, torch.float16)])
def test_native_path_equals_custom_op(op, B, T, M, N, dt):
    xs, dy, dS = W.synthetic(op, B, T, 2, M, N, dt, device="cuda")
    f = flex_rnn_b200.jit(W.STEPS[op])
    leaves = [x.detach().requires_grad_() for x in xs]

    def both(call):
        y, S = call(*leaves)
        return [y, S, *torch.autograd.grad((y, S), leaves, (dy, dS))]
    want = both(f.apply)
    for _ in range(3):              # the first call of a kind runs through the Python closures, later ones do not
        for a, b in zip(both(f), want):
            assert a.shape == b.shape and a.dtype == b.dtype and a.stride() == b.stride()
            assert torch.equal(a, b) or float((a.float() - b.float()).norm()) <= 1e-5 * float(b.float().norm())   # atomics
    for _ in range(3):
        with torch.no_grad():
            assert all(torch.equal(a, b) for a, b in zip(f(*xs), want))
    # an output left out of the loss, an input that needs no gradient, and a change of layout
    y, S = f(leaves[0].detach(), *leaves[1:])
    (g,) = torch.autograd.grad(y, [leaves[1]], dy.transpose(0, 1).contiguous().transpose(0, 1))
    y2, S2 = f.apply(*leaves)
    (g2,) = torch.autograd.grad(y2, [leaves[1]], dy)
    assert torch.equal(g, g2)
    strided = [torch.stack([x, x], -1)[..., 0].detach().requires_grad_() for x in xs]
    assert all(torch.equal(a, b) for a, b in zip(f(*strided), f.apply(*strided)))


@pytest.mark.gpu
def test_native_path_graph_semantics():
    """Second use of a freed graph raises, create_graph gives the custom op's graph, other streams and a changed
    input are honoured."""
    xs, dy, dS = W.synthetic("delta_rule", 1, 20, 2, 64, 64, torch.float32, device="cuda")
    f = flex_rnn_b200.jit(W.delta_rule)
    leaves = [x.detach().requires_grad_() for x in xs]
    y, S = f(*leaves)
    first = torch.autograd.grad(y, leaves, dy, retain_graph=True)
    again = torch.autograd.grad(y, leaves, dy)
    assert all(torch.equal(a, b) for a, b in zip(first, again))
    with pytest.raises(RuntimeError, match="second time"):
        torch.autograd.grad(y, leaves, dy)
    y, S = f(*leaves)
    g = torch.autograd.grad(y, leaves, dy, create_graph=True)
    assert torch.equal(g[0], first[0])
    with pytest.raises(RuntimeError, match="autograd"):
        torch.autograd.grad(g[0].sum(), leaves)
    y, S = f(*leaves)
    with torch.no_grad():
        leaves[0].add_(1.0)
    with pytest.raises(RuntimeError, match="modified by an inplace operation"):
        torch.autograd.grad(y, leaves, dy)
    st = torch.cuda.Stream()
    st.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(st), torch.no_grad():
        y2, _ = f(*leaves)
    torch.cuda.current_stream().wait_stream(st)
    assert torch.equal(y2, f.apply(*leaves)[0])


LAYOUTS = {"transposed": lambda g: g(2, 4, 3, 1, 8).transpose(1, 2), "sliced": lambda g: g(2, 3, 4, 1, 24)[..., 8:16],
           "expanded": lambda g: g(2, 3, 1, 1, 8).expand(2, 3, 4, 1, 8), "windows": lambda g: g(64).as_strided((2, 3, 4, 1, 8), (24, 6, 2, 1, 1)),
           "odd": lambda g: g(193)[1:].view(2, 3, 4, 1, 8), "reversed_dims": lambda g: g(8, 1, 4, 3, 2).permute(4, 3, 2, 1, 0)}


@pytest.mark.parametrize("layout", list(LAYOUTS))
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_saved_tensors_come_back_as_they_were(layout, dtype):
    """Whatever layout a saved-tensor hook returns, the backward reads the one that was saved, on its alignment."""
    from flex_rnn_b200 import runtime
    as_saved = runtime.host().as_saved
    x = LAYOUTS[layout](lambda *n: torch.randn(n).to(dtype))
    meta = (list(x.shape), list(x.stride()), x.dtype)
    lead = torch.empty(x.numel() + 1, dtype=dtype)[1:].view(x.shape).copy_(x)       # contiguous, off a 16-byte boundary
    for back in (x, x.contiguous(), x.transpose(0, 2).contiguous().transpose(0, 2), lead):
        got = as_saved(back, meta, x, True)
        assert got.data_ptr() % 16 == 0 and torch.equal(got, x)
        assert [s for s, n in zip(got.stride(), got.shape) if n > 1] == [s for s, n in zip(x.stride(), x.shape) if n > 1]
    assert as_saved(x, meta, x, False).data_ptr() == x.data_ptr()
    for bad in (x[:1], x.double(), x.to("meta"), x.reshape(-1)):
        with pytest.raises(RuntimeError, match="saved-tensor hook"):
            as_saved(bad, meta, x, True)


@pytest.mark.gpu
@pytest.mark.parametrize("dt,T", [(torch.float32, 20), (torch.bfloat16, 70)])       # recurrent and chunked kernels
def test_saved_tensor_hooks(dt, T):
    """Gradients do not depend on what saved-tensor hooks do to the layout of the inputs and the checkpoints."""
    xs, dy, dS = W.synthetic("delta_rule", 2, T, 3, 64, 64, dt, device="cuda")
    f = flex_rnn_b200.jit(W.delta_rule)
    xs[0] = xs[0].transpose(1, 2).contiguous().transpose(1, 2)          # dense, but not in the order of its dimensions
    xs[2] = torch.stack([xs[2], xs[2]], -1)[..., 0]
    leaves = [x.detach().requires_grad_() for x in xs]

    def off(t):                    # contiguous and off a 16-byte boundary
        return torch.empty(t.numel() + 1, dtype=t.dtype, device=t.device)[1:].view(t.shape).copy_(t)

    def grads(ctx):
        with ctx:
            y, S = f(*leaves)
        return torch.autograd.grad((y, S), leaves, (dy, dS))
    hooks = torch.autograd.graph.saved_tensors_hooks
    for _ in range(2):             # the first call compiles (a step function cannot be traced under hooks)
        want = grads(contextlib.nullcontext())
    for ctx in (torch.autograd.graph.save_on_cpu(pin_memory=True), hooks(off, lambda t: t),
                hooks(lambda t: t.transpose(0, -1).contiguous(), lambda t: t.transpose(0, -1))):
        assert all(torch.equal(a, b) for a, b in zip(grads(ctx), want))
    with pytest.raises(RuntimeError, match="saved-tensor hook"):
        grads(hooks(lambda t: t.cpu(), lambda t: t))


@pytest.mark.gpu
def test_transformed_backward():
    """Batched upstream gradients and a dispatch mode around the backward find the custom op."""
    from torch.utils._python_dispatch import TorchDispatchMode
    xs, dy, dS = W.synthetic("delta_rule", 1, 20, 2, 64, 64, torch.float32, device="cuda")
    f = flex_rnn_b200.jit(W.delta_rule)
    leaves = [x.detach().requires_grad_() for x in xs]
    want = [torch.autograd.grad(f(*leaves)[0], leaves, dy) for _ in range(2)][1]
    up = torch.stack([dy, 0.5 * dy])
    for a, b in zip(torch.autograd.grad(f(*leaves)[0], leaves, up, is_grads_batched=True), want):
        assert torch.equal(a[0], b) and torch.equal(a[1], 0.5 * b)
    seen = []

    class Log(TorchDispatchMode):
        def __torch_dispatch__(self, fn, types, args=(), kwargs=None):
            seen.append(str(fn))
            return fn(*args, **(kwargs or {}))
    y = f(*leaves)[0]
    with Log():
        got = torch.autograd.grad(y, leaves, dy)
    assert any("flex_rnn_b200" in s for s in seen)
    assert all(torch.equal(a, b) for a, b in zip(got, want))


@pytest.mark.gpu
@pytest.mark.filterwarnings("ignore")
def test_trace_records_the_op():
    """A traced function computes from its arguments, not from those of the tracing call."""
    xs, _, _ = W.synthetic("delta_rule", 1, 20, 2, 64, 64, torch.float32, device="cuda")
    f = flex_rnn_b200.jit(W.delta_rule)
    other = [0.5 * x for x in xs]
    with torch.no_grad():
        for _ in range(2):
            want = f(*other)
        traced = torch.jit.trace(lambda *a: f(*a), tuple(xs), check_trace=False)
        assert all(torch.equal(a, b) for a, b in zip(traced(*other), want))


@pytest.mark.gpu
@pytest.mark.parametrize("grad", [False, True])
def test_full_launch_queue_does_not_stop_other_threads(grad):
    """A launch that waits for room in the queue does so without the interpreter lock."""
    xs, _, _ = W.synthetic("delta_rule", 1, 4, 1, 32, 32, torch.float32, device="cuda")
    f = flex_rnn_b200.jit(W.delta_rule)
    xs = [x.detach().requires_grad_(grad) for x in xs]
    for _ in range(3):
        f(*xs)
    torch.cuda.synchronize()
    gaps, done = [0.0], threading.Event()

    def tick():
        last = time.perf_counter()
        while not done.is_set():
            time.sleep(0.001)
            now = time.perf_counter()
            gaps.append(now - last)
            last = now
    other = threading.Thread(target=tick)
    other.start()
    start = time.perf_counter()
    torch.cuda._sleep(1_500_000_000)            # about 0.8 s of GPU time in front of the queue
    for _ in range(3000):                       # more launches than the queue holds
        f(*xs)
    took = time.perf_counter() - start
    done.set()
    other.join()
    torch.cuda.synchronize()
    assert took > 0.4, "the queue never filled up"
    assert max(gaps) < 0.2, (max(gaps), took)


@pytest.mark.gpu
@pytest.mark.parametrize("native", [True, False])
def test_checkpointed_region(native):
    """Non-reentrant checkpointing, which recomputes through saved-tensor hooks and unpacks each tensor once."""
    from torch.utils.checkpoint import checkpoint
    xs, dy, _ = W.synthetic("delta_rule", 1, 20, 2, 64, 64, torch.float32, device="cuda")
    f = flex_rnn_b200.jit(W.delta_rule)
    leaves = [x.detach().requires_grad_() for x in xs]
    want = torch.autograd.grad(torch.tanh(f(*leaves)[0]), leaves, dy)
    call = f if native else f.apply
    for _ in range(2):
        y = checkpoint(lambda *a: torch.tanh(call(*a)[0]), *leaves, use_reentrant=False)
        assert all(torch.equal(a, b) for a, b in zip(torch.autograd.grad(y, leaves, dy), want))
