"""The chunked form (chunk.py): which step functions have it, and its kernels against the naive scan in fp64 at the
edges of chunks, columns and rows, with decays that vanish inside a chunk.  CPU: under the host emulation; GPU: the
public API."""
import dataclasses

import pytest
import torch

import flex_rnn_b200
from flex_rnn_b200 import chunk
from flex_rnn_b200 import examples as X
from flex_rnn_b200 import workloads as W
from flex_rnn_b200.twopass import build_twopass, default_tuning, make_plan
from oracle import naive_oracle as O


def case(op, B, T, H, M, N, dt, reset=False):
    """16-bit inputs and an fp32 state, so that outputs and final states show the kernels' own accuracy."""
    if op in W.STEPS:
        *ins, s = W.synthetic(op, B, T, H, M, N, dt)[0]
        step = W.STEPS[op]
    else:
        (ins, (s,)), step = X.zoo_case(op, B, T, H, M, N, dt), X.ZOO[op]
    if reset:
        g = torch.Generator().manual_seed(3)
        k = {"gated_delta_rule": 3, "rwkv7": 1, "gla": 3}[op]
        hit = torch.rand(ins[k].shape, generator=g) < 0.05
        ins[k] = torch.where(hit, torch.full_like(ins[k], -200.0 if op == "gla" else 0.0), ins[k])
    g = torch.Generator().manual_seed(1)
    s = 0.1 * torch.randn(s.shape, generator=g)
    dy, dS = torch.randn(B, T, H, M, generator=g), torch.randn(s.shape, generator=g)
    return step, ins, s, dy, dS


def check(got, step, ins, s, dy, dS, dt):
    # fp64 leaves holding the same values: a 16-bit leaf would collect the contributions of all timesteps in 16 bits
    ry, rS, rgx, rgs = O.fwd_bwd(step, [x.double() for x in ins], [s.double()], [dy.double()], [dS.double()], dtype=torch.float64)
    tol = {torch.bfloat16: 1e-2, torch.float16: 2e-3}[dt]
    for a, b in zip(got, [*ry, *rS, *rgx, *rgs]):
        assert a.shape == b.shape
        assert O.rel_err(a.cpu(), b) < (2e-6 if a.dtype == torch.float32 else tol), (a.dtype, O.rel_err(a.cpu(), b))


CASES = [("delta_rule", 1, 32, 1, 32, 16, torch.bfloat16, False), ("gated_delta_rule", 2, 37, 1, 8, 40, torch.float16, True),
         ("rwkv7", 1, 33, 1, 24, 24, torch.bfloat16, True), ("mamba2", 1, 49, 2, 16, 128, torch.bfloat16, False),
         ("gla", 1, 50, 1, 128, 80, torch.float16, True), ("retention", 1, 70, 2, 40, 32, torch.bfloat16, False),
         ("gated_delta_rule", 1, 70, 1, 64, 128, torch.bfloat16, True)]


def test_which_steps_have_the_form():
    for op, want in [("delta_rule", True), ("gated_delta_rule", True), ("rwkv7", True), ("mamba2", True), ("gla", True),
                     ("retention", True), ("longhorn", False), ("hgrn", False), ("mamba", False)]:
        step, ins, s, _, _ = case(op, 1, 64, 2, 32, 1 if op == "hgrn" else 32, torch.bfloat16)
        cp = chunk.chunk_plan(make_plan(step, ins, [s])[0])
        assert (cp is not None and cp.bp is not None) == want, op
    step, ins, s, _, _ = case("delta_rule", 1, 64, 1, 256, 64, torch.bfloat16)
    cp = chunk.chunk_plan(make_plan(step, ins, [s])[0])
    assert cp is not None and cp.short and cp.bp is None            # rows over several CTAs: calls without gradients only
    for H, M, N, short, train in [(64, 64, 64, True, True), (400, 64, 64, False, False), (400, 64, 128, False, True),
                                  (400, 128, 64, True, True), (400, 256, 128, True, False), (4, 64, 256, False, False)]:
        args = [torch.empty(1, 64, H, *x, dtype=torch.bfloat16, device="meta") for x in ((1, N), (1, N), (M, 1), (1, 1))]
        plan = make_plan(W.delta_rule, args, [torch.empty(1, H, M, N, dtype=torch.bfloat16, device="meta")])[0]
        cp = chunk.chunk_plan(plan)
        assert (cp is not None and cp.short, cp is not None and cp.bp is not None) == (short, train), (H, M, N)


@pytest.mark.parametrize("op,B,T,H,M,N,dt,reset", CASES)
def test_emulated(op, B, T, H, M, N, dt, reset):
    from emu.emu import EmuLauncher
    step, ins, s, dy, dS = case(op, B, T, H, M, N, dt, reset)
    fwd, bwd, fm, bm = build_twopass(step, tuple(ins), (s,), _launcher=EmuLauncher)
    assert [ks.name for ks in fwd.sources] == ["frnn_cfw", "frnn_cbw"]
    assert build_twopass(step, tuple(ins), (s,), dryrun=True) == (fm, bm)
    y, sT, ck, aux = fwd(tuple(ins), (s,))
    assert [tuple(m[0]) for m in fm] == [tuple(t.shape) for t in (y, sT, ck, aux)]
    dx, ds = bwd((dy.to(y.dtype),), (dS,), tuple(ins), (ck,), (aux,))
    check([y, sT, *dx, *ds], step, ins, s, dy, dS, dt)
    check([*fwd.infer(tuple(ins), (s,))], step, ins, s, dy, dS, dt)


def run_member(op, k, to, launcher=None):
    """A pinned member of the chunked scans, with recurrent members pinned beside it: fw, bw and infer against the oracle."""
    step, ins, s, dy, dS = case(op, 1, 40, 2, 32, 32, torch.bfloat16)
    tu = dataclasses.replace(default_tuning(1, 40, 2, 32, 32, 1), chunk_variant=k, fw_variant=1, bw_variant=1)
    gi, gs = [x.to(to) for x in ins], s.to(to)
    fwd, bwd, _, _ = build_twopass(step, tuple(gi), (gs,), tuning=tu, _launcher=launcher)
    assert [ks.name for ks in fwd.sources] == ["frnn_cfw", "frnn_cbw"] and fwd.tuned["fw_choice"] == fwd.tuned["bw_choice"] == k
    y, sT, ck, aux = fwd(tuple(gi), (gs,))
    dx, ds = bwd((dy.to(y),), (dS.to(sT),), tuple(gi), (ck,), (aux,))
    check([y, sT, *dx, *ds], step, ins, s, dy, dS, torch.bfloat16)
    check([*fwd.infer(tuple(gi), (gs,))], step, ins, s, dy, dS, torch.bfloat16)
    return [ks.source for ks in (*fwd.sources, fwd.tuned["infer_src"])]


def test_pinned_members():
    """Pinning keeps the chunked form; a forward or backward member alone still asks for the recurrent kernels."""
    from emu.emu import EmuLauncher
    seen = [run_member("gated_delta_rule", k, "cpu", EmuLauncher) for k in range(3)]
    assert all(len({src[i] for src in seen}) == 3 for i in range(3))
    step, ins, s, _, _ = case("delta_rule", 1, 40, 2, 32, 32, torch.bfloat16)
    for kw, name in [(dict(fw_variant=0), "frnn_fw"), (dict(bw_variant=0), "frnn_fw"), (dict(), "frnn_cfw"), (dict(chunk=0, chunk_variant=1), "frnn_fw")]:
        tu = dataclasses.replace(default_tuning(1, 40, 2, 32, 32, 1), **kw)
        fwd = build_twopass(step, tuple(ins), (s,), tuning=tu, _launcher=lambda ks: None)[0]
        assert fwd.sources[0].name == name, kw


@pytest.mark.gpu
@pytest.mark.parametrize("op,k", [("delta_rule", 1), ("delta_rule", 2), ("rwkv7", 1), ("rwkv7", 2), ("mamba2", 1), ("gla", 2)])
def test_pinned_members_gpu(op, k):
    run_member(op, k, "cuda:0")


@pytest.mark.gpu
@pytest.mark.parametrize("op,B,T,H,M,N,dt,reset", CASES + [
    ("delta_rule", 3, 200, 2, 128, 128, torch.bfloat16, False), ("gated_delta_rule", 2, 64, 3, 64, 128, torch.bfloat16, True),
    ("rwkv7", 1, 100, 2, 128, 128, torch.bfloat16, True), ("mamba2", 2, 300, 2, 64, 64, torch.float16, False),
    ("gla", 2, 130, 2, 96, 128, torch.bfloat16, True)])
def test_gpu(op, B, T, H, M, N, dt, reset):
    step, ins, s, dy, dS = case(op, B, T, H, M, N, dt, reset)
    f = flex_rnn_b200.jit(step)
    leaves = [x.cuda().requires_grad_() for x in [*ins, s]]
    for _ in range(2):
        y, sT = f(*leaves)
        grads = torch.autograd.grad((y, sT), leaves, (dy.cuda().to(y.dtype), dS.cuda()))
        assert f.forward_func.kernel_status("cuda:0") == 0
        check([y.detach(), sT.detach(), *grads], step, ins, s, dy, dS, dt)
    with torch.no_grad():
        short = f(*leaves)
    check(short, step, ins, s, dy, dS, dt)


def off(x):
    """One element off a 16-byte boundary."""
    return torch.empty(x.numel() + 1, dtype=x.dtype, device=x.device)[1:].view(x.shape).copy_(x)


LAYOUTS = {
    "packed": lambda x: torch.cat([x, x], dim=-1)[..., :x.shape[-1]],                 # sliced out of a wider tensor
    "permuted": lambda x: x.transpose(1, 2).contiguous().transpose(1, 2),             # [B, H, T, ..] in memory
    "heads": lambda x: x[:, :, :1].expand_as(x),                                      # the same for all heads, not copied
    "times": lambda x: x[:, :1].expand_as(x),
    "off": off,
    "spread": lambda x: torch.stack([x, x], -1)[..., 0],                              # elements two apart
    "plain": lambda x: x,
}
# which layout each input has, in turn; state: transposed in memory where "t", off a boundary where "o"
LAYOUT_CASES = [
    ("delta_rule", 2, 34, 2, 24, 40, ["packed", "off", "permuted", "spread"], "t"), ("gated_delta_rule", 1, 37, 3, 32, 32, ["heads", "times"], "o"),
    ("rwkv7", 1, 33, 2, 24, 24, ["off", "packed", "heads", "spread", "permuted", "times"], ""), ("mamba2", 2, 49, 2, 16, 48, ["spread", "off"], "to"),
    ("gla", 1, 70, 1, 128, 128, ["plain", "off", "packed", "permuted"], "t"), ("gated_delta_rule", 1, 65, 1, 128, 128, ["off"], ""),
    ("gla", 1, 65, 1, 128, 128, ["off", "spread"], "o"), ("retention", 2, 33, 2, 32, 16, ["times", "off", "packed"], "t")]


def layout_case(op, B, T, H, M, N, layouts, state, mixed):
    step, ins, s, dy, dS = case(op, B, T, H, M, N, torch.bfloat16)
    if mixed:                                                                         # bf16 and fp16 inputs in one call
        ins = [x.half() if i % 2 else x for i, x in enumerate(ins)]
    ins = [LAYOUTS[layouts[i % len(layouts)]](x) if x.shape[1] > 1 else x for i, x in enumerate(ins)]
    if "t" in state:
        s = s.mT.contiguous().mT
    if "o" in state:
        s = off(s) if "t" not in state else off(s.mT).mT
    return step, ins, s, dy, dS


@pytest.mark.parametrize("op,B,T,H,M,N,layouts,state", LAYOUT_CASES)
def test_layouts_emulated(op, B, T, H, M, N, layouts, state):
    from emu.emu import EmuLauncher
    step, ins, s, dy, dS = layout_case(op, B, T, H, M, N, layouts, state, mixed=T % 2 == 0)
    fwd, bwd, _, _ = build_twopass(step, tuple(ins), (s,), _launcher=EmuLauncher)
    assert [ks.name for ks in fwd.sources] == ["frnn_cfw", "frnn_cbw"]
    if N == 128:                   # one buffer of raw inputs: two do not fit beside the operands
        assert "(c % 1)" in fwd.sources[1].source
    y, sT, ck, aux = fwd(tuple(ins), (s,))
    dx, ds = bwd((dy.to(y.dtype),), (dS,), tuple(ins), (ck,), (aux,))
    check([y, sT, *dx, *ds], step, ins, s, dy, dS, torch.bfloat16)
    check([*fwd.infer(tuple(ins), (s,))], step, ins, s, dy, dS, torch.bfloat16)
    for g, x in zip([*dx, *ds], [*ins, s]):
        assert g.dtype == x.dtype and g.stride() == torch.empty_like(x).stride()


@pytest.mark.gpu
@pytest.mark.parametrize("op,B,T,H,M,N,layouts,state", LAYOUT_CASES + [
    ("delta_rule", 3, 130, 3, 128, 128, ["off", "spread", "heads", "permuted"], "to"), ("mamba2", 2, 200, 5, 64, 128, ["packed"], "t"),
    ("rwkv7", 2, 100, 2, 128, 128, ["times", "off", "plain", "packed"], "o")])
def test_layouts_gpu(op, B, T, H, M, N, layouts, state):
    mixed = T % 2 == 0
    step, ins, s, dy, dS = layout_case(op, B, T, H, M, N, layouts, state, mixed)
    f = flex_rnn_b200.jit(step)
    # .cuda() keeps strides but neither offsets nor expanded dimensions: the layouts are made on the GPU
    base = case(op, B, T, H, M, N, torch.bfloat16)[1]
    gi = [x.cuda().half() if mixed and i % 2 else x.cuda() for i, x in enumerate(base)]
    gi = [LAYOUTS[layouts[i % len(layouts)]](x) if x.shape[1] > 1 else x for i, x in enumerate(gi)]
    gs = s.cuda() if "o" not in state else off(s.cuda().mT).mT if "t" in state else off(s.cuda())
    assert [x.stride() for x in [*gi, gs]] == [x.stride() for x in [*ins, s]]
    leaves = [x.detach().requires_grad_() for x in [*gi, gs]]
    for _ in range(2):
        y, sT = f(*leaves)
        grads = torch.autograd.grad((y, sT), leaves, (dy.cuda().to(y.dtype), dS.cuda()))
        assert f.forward_func.kernel_status("cuda:0") == 0
        check([y.detach(), sT.detach(), *grads], step, ins, s, dy, dS, torch.bfloat16)
    with torch.no_grad():
        short = f(*leaves)
    check(short, step, ins, s, dy, dS, torch.bfloat16)


@pytest.mark.gpu
def test_timed_candidates_are_checked_builds(monkeypatch):
    """With the checked build asked for, no candidate of the timing on the first call is an unchecked one (nothing is
    compiled or launched here)."""
    from flex_rnn_b200 import twopass
    made = []

    class Launcher:
        def __init__(self, ks):
            self.ks = ks
            made.append(ks)

        def __call__(self, ptrs, device):
            pass
    monkeypatch.setattr(twopass, "_CudaLauncher", Launcher)
    step, ins, s, dy, dS = case("delta_rule", 1, 64, 2, 64, 64, torch.bfloat16)
    ins, s = tuple(x.cuda() for x in ins), s.cuda()
    tu = dataclasses.replace(default_tuning(1, 64, 2, 64, 64, 1), bounds=1, autotune_min_work=0)
    fwd, bwd, _, _ = build_twopass(step, ins, (s,), tuning=tu)
    y, sT, ck, aux = fwd(ins, (s,))
    bwd((dy.cuda().to(y),), (dS.cuda().to(sT),), ins, (ck,), (aux,))
    fwd.infer(ins, (s,))
    assert [sum(ks.name == n for ks in made) for n in ("frnn_cfw", "frnn_cbw", "frnn_cvg")] == [6, 3, 1]
    assert all(ks.info.get("bounds") for ks in made)


def small_decays(op, B, T, H, M, N, small):
    """RWKV-7 with a few decays per chunk that are small, whose own gradients are not formed by a division, but whose
    products over a chunk are still divided by."""
    step, ins, s, dy, dS = case(op, B, T, H, M, N, torch.bfloat16)
    g = torch.Generator().manual_seed(5)
    hit = torch.rand(ins[1].shape, generator=g) < 0.02
    ins[1] = torch.where(hit, torch.full_like(ins[1], small), ins[1])
    return step, ins, s, dy, dS


# 40 columns: the last two warps of a tile have threads without one; 128 rows and columns: the benchmark's state
@pytest.mark.parametrize("T,M,N,small", [(33, 24, 40, 2e-4), (32, 16, 128, 1e-5)])
def test_small_decays_emulated(T, M, N, small):
    from emu.emu import EmuLauncher
    step, ins, s, dy, dS = small_decays("rwkv7", 1, T, 1, M, N, small)
    fwd, bwd, _, _ = build_twopass(step, tuple(ins), (s,), _launcher=EmuLauncher)
    y, sT, ck, aux = fwd(tuple(ins), (s,))
    dx, ds = bwd((dy.to(y.dtype),), (dS,), tuple(ins), (ck,), (aux,))
    check([y, sT, *dx, *ds], step, ins, s, dy, dS, torch.bfloat16)


@pytest.mark.gpu
@pytest.mark.parametrize("T,M,N,small", [(33, 24, 40, 2e-4), (100, 128, 128, 1e-5)])
def test_small_decays_gpu(T, M, N, small):
    step, ins, s, dy, dS = small_decays("rwkv7", 2, T, 2, M, N, small)
    f = flex_rnn_b200.jit(step)
    leaves = [x.cuda().requires_grad_() for x in [*ins, s]]
    y, sT = f(*leaves)
    grads = torch.autograd.grad((y, sT), leaves, (dy.cuda().to(y.dtype), dS.cuda()))
    assert f.forward_func.kernel_status("cuda:0") == 0
    check([y.detach(), sT.detach(), *grads], step, ins, s, dy, dS, torch.bfloat16)


# the state's update in one rolled loop: five blocks of 16 columns in four quarters; one block; chunks cut short
COMPACT = [("delta_rule", 5, 70, 15, 72, 72), ("mamba2", 3, 33, 26, 16, 16), ("rwkv7", 5, 33, 15, 64, 128)]


def test_compact_rule_and_emulated():
    from emu.emu import EmuLauncher
    for B, H, M, want in [(1, 74, 64, False), (1, 75, 64, True), (1, 37, 256, False), (1, 38, 256, True)]:
        args = [torch.empty(B, 64, H, *x, dtype=torch.bfloat16, device="meta") for x in ((1, 64), (1, 64), (M, 1), (1, 1))]
        plan = make_plan(W.delta_rule, args, [torch.empty(B, H, M, 64, dtype=torch.bfloat16, device="meta")])[0]
        assert chunk.chunk_plan(plan).compact == want
    for op, T, M, N in [("gated_delta_rule", 40, 24, 72), ("rwkv7", 33, 16, 16)]:
        step, ins, s, dy, dS = case(op, 1, T, 1, M, N, torch.bfloat16)
        plan = make_plan(step, ins, [s])[0]
        plan.n_sm = 1                                     # one head already fills it
        cp = chunk.chunk_plan(plan)
        assert cp.compact
        yf, sf = torch.empty(1, T, 1, M), torch.empty_like(s)
        err = torch.zeros(1, dtype=torch.int32)
        EmuLauncher(cp.infer())([t.data_ptr() for t in (*ins, s, yf, sf, err)])
        ry, rS, _, _ = O.fwd_bwd(step, [x.double() for x in ins], [s.double()], [dy.double()], [dS.double()], dtype=torch.float64)
        assert int(err) == 0 and O.rel_err(yf, ry[0]) < 2e-6 and O.rel_err(sf, rS[0]) < 2e-6


@pytest.mark.gpu
@pytest.mark.parametrize("op,B,T,H,M,N", COMPACT)
def test_compact_gpu(op, B, T, H, M, N):
    step, ins, s, dy, dS = case(op, B, T, H, M, N, torch.bfloat16)
    f = flex_rnn_b200.jit(step)
    leaves = [x.cuda().requires_grad_() for x in [*ins, s]]
    y, sT = f(*leaves)
    grads = torch.autograd.grad((y, sT), leaves, (dy.cuda().to(y.dtype), dS.cuda()))
    assert f.forward_func.kernel_status("cuda:0") == 0 and [k.name for k in f.forward_func.sources] == ["frnn_cfw", "frnn_cbw"]
    check([y.detach(), sT.detach(), *grads], step, ins, s, dy, dS, torch.bfloat16)


# beyond one CTA per SM states of fewer than 8192 elements, and calls without gradients of at most 64 rows, keep the recurrent
# kernels however long the call is: their operands are fp32 throughout, the chunked ones' two tf32 terms
def test_rule_of_small_states():
    for op, T, H, M, N, short, train in [("delta_rule", 255, 149, 64, 64, False, False), ("delta_rule", 256, 149, 64, 64, False, False),
                                         ("gla", 1024, 300, 72, 96, False, False), ("rwkv7", 256, 149, 64, 64, False, False),
                                         ("mamba2", 1024, 149, 64, 128, False, True), ("gla", 4096, 149, 32, 128, False, False),
                                         ("rwkv7", 256, 149, 64, 128, False, True), ("mamba2", 256, 149, 72, 128, True, True),
                                         ("delta_rule", 255, 148, 64, 64, True, True)]:
        step, ins, s, _, _ = case(op, 1, 2, 2, 2, 2, torch.bfloat16)
        at = lambda x: [1, T if x.shape[1] > 1 else 1, H, M if x.shape[3] > 1 else 1, N if x.shape[4] > 1 else 1]
        args = [torch.empty(at(x), dtype=torch.bfloat16, device="meta") for x in ins]
        cp = chunk.chunk_plan(make_plan(step, args, [torch.empty(1, H, M, N, dtype=torch.bfloat16, device="meta")])[0])
        assert (cp is not None and cp.short, cp is not None and cp.bp is not None) == (short, train), (op, T, H, M, N)


@pytest.mark.gpu
@pytest.mark.parametrize("op,T,M,N,name", [("delta_rule", 257, 64, 64, "frnn_fw"), ("gated_delta_rule", 256, 48, 88, "frnn_fw"),
                                           ("mamba2", 260, 32, 128, "frnn_fw"), ("gla", 256, 64, 128, "frnn_cfw")])
def test_long_small_states_gpu(op, T, M, N, name):
    """Which kernels train, and that a call without gradients takes the recurrent one, as accurate as it is."""
    step, ins, s, dy, dS = case(op, 3, T, 50, M, N, torch.bfloat16)
    f = flex_rnn_b200.jit(step)
    leaves = [x.cuda().requires_grad_() for x in [*ins, s]]
    y, sT = f(*leaves)
    grads = torch.autograd.grad((y, sT), leaves, (dy.cuda().to(y.dtype), dS.cuda()))
    assert f.forward_func.kernel_status("cuda:0") == 0 and f.forward_func.sources[0].name == name
    check([y.detach(), sT.detach(), *grads], step, ins, s, dy, dS, torch.bfloat16)
    with torch.no_grad():
        short = f(*leaves)
    assert f.forward_func.tuned["infer_src"].name == "frnn_fw"
    check(short, step, ins, s, dy, dS, torch.bfloat16)


def many_sums(nd, dt=torch.bfloat16, T=34, M=16, N=32):
    """``nd`` row sums of the state, whose gradients are no inputs and so have a second tf32 term."""
    def step(*a):
        *qs, v, k, S = a
        return sum((S * q).sum(-1, True) ** 2 for q in qs), S + v * k
    g = torch.Generator().manual_seed(nd)
    n = lambda *s: torch.randn(*s, generator=g)
    rows = [(n(1, T, 1, 1, N) * N ** -0.5).to(dt) for _ in range(nd + 1)]
    return step, [*rows[:nd], n(1, T, 1, M, 1).to(dt), rows[nd]], 0.1 * n(1, 1, M, N), n(1, T, 1, M), n(1, 1, M, N)


# 16 steps of each sum, and as many rests: 4 sums fill the 128 rows of a product, 5 to 7 fitted Tensor Memory
@pytest.mark.parametrize("nd,name", [(4, "frnn_cfw"), (5, "frnn_fw"), (7, "frnn_fw")])
def test_row_sums_beyond_a_product_train(nd, name):
    from emu.emu import EmuLauncher
    step, ins, s, dy, dS = many_sums(nd)
    fwd, bwd, _, _ = build_twopass(step, tuple(ins), (s,), _launcher=EmuLauncher)
    assert fwd.sources[0].name == name
    y, sT, ck, aux = fwd(tuple(ins), (s,))
    dx, ds = bwd((dy.to(y.dtype),), (dS,), tuple(ins), (ck,), (aux,))
    check([y, sT, *dx, *ds], step, ins, s, dy, dS, torch.bfloat16)


@pytest.mark.parametrize("nd,name", [(8, "frnn_cfw"), (9, "frnn_fw")])
def test_row_sums_beyond_a_product_infer(nd, name):
    """Gram has the row sums of 16 steps as rows: 8 sums fill the 128 of a product.  (Training is refused from 5 on.)"""
    from emu.emu import EmuLauncher
    step, ins, s, dy, dS = many_sums(nd)
    fwd, _, _, _ = build_twopass(step, tuple(ins), (s,), _launcher=EmuLauncher)
    check([*fwd.infer(tuple(ins), (s,))], step, ins, s, dy, dS, torch.bfloat16)
    assert fwd.tuned["infer_src"].name == name


def output_first(q, w, k, v, S):
    """The output reads the state before the update: no other term of a decay's gradient depends on the decay."""
    return (S * q).sum(-1, True), S * w + v * k


def bad_decay(op, T, M, N, bad, small):
    """One decay of one column is ``bad``, another one of that column, in the same chunk, ``small``."""
    g = torch.Generator().manual_seed(0)
    n = lambda *s: torch.randn(*s, generator=g)
    if op == "rwkv7":
        step, ins, s, dy, dS = case(op, 1, T, 1, M, N, torch.bfloat16)
    else:
        step, s, dy, dS = output_first, 0.1 * n(1, 1, M, N), n(1, T, 1, M), n(1, 1, M, N)
        ins = [(0.2 * n(1, T, 1, 1, N)).bfloat16(), torch.sigmoid(n(1, T, 1, 1, N) + 2).bfloat16(), (0.2 * n(1, T, 1, 1, N)).bfloat16(),
               n(1, T, 1, M, 1).bfloat16()]
    ins[1][0, T - 1, 0, 0, 5] = bad
    if small is not None:
        ins[1][0, T - 3, 0, 0, 5] = small
    return step, ins, s, dy, dS


def check_bad_decay(got, step, ins, s, dy, dS):
    """A number only where the oracle has one, and that one; the decays of the other columns all have their gradients."""
    ry, rS, rgx, rgs = O.fwd_bwd(step, [x.double() for x in ins], [s.double()], [dy.double()], [dS.double()], dtype=torch.float64)
    for i, (a, b) in enumerate(zip(got, [*ry, *rS, *rgx, *rgs])):
        a, b = a.cpu().double(), b.double()
        fin = torch.isfinite(a)
        assert torch.isfinite(b[fin]).all() and O.rel_err(a[fin], b[fin]) < 1e-2, i
        if step is output_first and i == 3:
            assert (~fin).sum() <= a.shape[1], i


BAD_DECAYS = [("output_first", 32, 16, 32, float("nan"), None), ("output_first", 34, 16, 40, float("nan"), 2e-4), ("output_first", 37, 24, 128, float("inf"), 0.0),
              ("output_first", 32, 16, 32, float("inf"), 1e-5), ("output_first", 32, 16, 32, float("nan"), 2.0 ** -10),
              ("rwkv7", 33, 24, 24, float("nan"), None), ("rwkv7", 33, 24, 24, float("inf"), 2e-4)]


@pytest.mark.parametrize("op,T,M,N,bad,small", BAD_DECAYS)
def test_bad_decay_emulated(op, T, M, N, bad, small):
    from emu.emu import EmuLauncher
    step, ins, s, dy, dS = bad_decay(op, T, M, N, bad, small)
    fwd, bwd, _, _ = build_twopass(step, tuple(ins), (s,), _launcher=EmuLauncher)
    assert fwd.sources[0].name == "frnn_cfw"
    y, sT, ck, aux = fwd(tuple(ins), (s,))
    dx, ds = bwd((dy.to(y.dtype),), (dS,), tuple(ins), (ck,), (aux,))
    check_bad_decay([y, sT, *dx, *ds], step, ins, s, dy, dS)


@pytest.mark.gpu
@pytest.mark.parametrize("op,T,M,N,bad,small", BAD_DECAYS)
def test_bad_decay_gpu(op, T, M, N, bad, small):
    step, ins, s, dy, dS = bad_decay(op, T, M, N, bad, small)
    f = flex_rnn_b200.jit(step)
    leaves = [x.cuda().requires_grad_() for x in [*ins, s]]
    y, sT = f(*leaves)
    grads = torch.autograd.grad((y, sT), leaves, (dy.cuda().to(y.dtype), dS.cuda()))
    assert f.forward_func.kernel_status("cuda:0") == 0
    check_bad_decay([y.detach(), sT.detach(), *grads], step, ins, s, dy, dS)


# rank-1 terms whose p are inputs need no rests, but a step that fits only without them keeps the recurrent backward
@pytest.mark.parametrize("nd,nr,train", [(1, 3, True), (1, 4, False), (2, 3, True), (2, 4, False), (3, 3, False)])
def test_rule_of_many_terms(nd, nr, train):
    def step(*a):
        qs, vs, ks, S = a[:nd], a[nd:nd + nr], a[nd + nr:-1], a[-1]
        y = sum((S * q).sum(-1, True) ** 2 for q in qs)
        for v, k in zip(vs, ks):
            S = S + v * k
        return y, S
    for M, N, T in [(16, 32, 40), (128, 128, 64)]:
        args = [torch.empty(1, T, 2, *x, dtype=torch.bfloat16, device="meta") for x in [(1, N)] * nd + [(M, 1)] * nr + [(1, N)] * nr]
        cp = chunk.chunk_plan(make_plan(step, args, [torch.empty(1, 2, M, N, dtype=torch.bfloat16, device="meta")])[0])
        assert cp.short and (cp.bp is not None) == train, (M, N)


def tanh_out(q, v, k, S):
    """The backward's p are made of the forward's tanh, and so are its outputs."""
    S = S + (v - (S * k).sum(-1, True)) * k
    return torch.tanh((S * q).sum(-1, True)), S


def tanh_p(q, v, k, S):
    """p is no output, but the output takes the tanh that p is made of."""
    e = torch.tanh(v - (S * k).sum(-1, True))
    S = S + (e * v) * k
    return (S * q).sum(-1, True) + e, S


def square_out(q, v, k, S):
    """p of the backward from the forward's sums, before its own: powf in each step."""
    S = S + v * k
    return (S * q).sum(-1, True) ** 2, S


def costly_case(step, T, M, N):
    g = torch.Generator().manual_seed(3)
    n = lambda *s: torch.randn(*s, generator=g)
    row = lambda: (n(1, T, 2, 1, N) * N ** -0.5).bfloat16()
    return [row(), n(1, T, 2, M, 1).bfloat16(), row()], 0.1 * n(1, 2, M, N), n(1, T, 2, M), n(1, 2, M, N)


COSTLY = [(tanh_out, "frnn_expf(", 32), (tanh_p, "frnn_expf(", 32), (square_out, "powf(", 32)]


@pytest.mark.parametrize("step,call,C", COSTLY)
def test_costly_values_are_computed_once(step, call, C):
    """The state warps' code for a chunk holds each step of it: a value that both the p and the outputs are made of is there once."""
    shapes = [(1, 64), (64, 1), (1, 64)]
    args = [torch.empty(1, 64, 2, *x, dtype=torch.bfloat16, device="meta") for x in shapes]
    cp = chunk.chunk_plan(make_plan(step, args, [torch.empty(1, 2, 64, 64, dtype=torch.bfloat16, device="meta")])[0])
    assert cp.C == C
    for ks in (cp.forward(), cp.infer(), cp.backward_scan()):
        assert ks.source[ks.source.index('extern "C"'):].count(call) <= C, ks.name


@pytest.mark.parametrize("step,T,M,N", [(tanh_out, 34, 16, 32), (tanh_p, 70, 24, 16), (square_out, 64, 16, 24)])
def test_costly_values_emulated(step, T, M, N):
    from emu.emu import EmuLauncher
    ins, s, dy, dS = costly_case(step, T, M, N)
    fwd, bwd, _, _ = build_twopass(step, tuple(ins), (s,), _launcher=EmuLauncher)
    assert fwd.sources[0].name == "frnn_cfw"
    y, sT, ck, aux = fwd(tuple(ins), (s,))
    dx, ds = bwd((dy.to(y.dtype),), (dS,), tuple(ins), (ck,), (aux,))
    check([y, sT, *dx, *ds], step, ins, s, dy, dS, torch.bfloat16)
    check([*fwd.infer(tuple(ins), (s,))], step, ins, s, dy, dS, torch.bfloat16)


@pytest.mark.gpu
@pytest.mark.parametrize("step,T,M,N", [(tanh_out, 100, 128, 128), (tanh_p, 70, 72, 80), (square_out, 64, 64, 64)])
def test_costly_values_gpu(step, T, M, N):
    ins, s, dy, dS = costly_case(step, T, M, N)
    f = flex_rnn_b200.jit(step)
    leaves = [x.cuda().requires_grad_() for x in [*ins, s]]
    y, sT = f(*leaves)
    grads = torch.autograd.grad((y, sT), leaves, (dy.cuda().to(y.dtype), dS.cuda()))
    assert f.forward_func.kernel_status("cuda:0") == 0 and f.forward_func.sources[0].name == "frnn_cfw"
    check([y.detach(), sT.detach(), *grads], step, ins, s, dy, dS, torch.bfloat16)


def sums_and_decay(q0, q1, q2, q3, v, k, w, S):
    """Four row sums beside a decay per column: the second phase of the vector gradients leaves room for one CTA per SM."""
    S = S * w + v * k
    return sum((S * q).sum(-1, True) ** 2 for q in (q0, q1, q2, q3)), S


def sums_and_decay_case(T, M, N):
    g = torch.Generator().manual_seed(4)
    n = lambda *s: torch.randn(*s, generator=g)
    row = lambda: (n(1, T, 2, 1, N) * N ** -0.5).bfloat16()
    ins = [row(), row(), row(), row(), n(1, T, 2, M, 1).bfloat16(), row(), torch.sigmoid(n(1, T, 2, 1, N) + 2).bfloat16()]
    return ins, 0.1 * n(1, 2, M, N), n(1, T, 2, M), n(1, 2, M, N)


# two slices of 16 rows in two buffers; three slices of 8 rows and a chunk cut short
@pytest.mark.parametrize("T,M,N", [(32, 32, 16), (37, 24, 32)])
def test_vector_gradients_with_one_cta_per_sm_emulated(T, M, N):
    from emu.emu import EmuLauncher
    ins, s, dy, dS = sums_and_decay_case(T, M, N)
    ks = chunk.chunk_plan(make_plan(sums_and_decay, ins, [s])[0]).vector_grads()
    assert "__launch_bounds__(256, 1)" in ks.source and "s < 2 || frnn_mbar_wait" in ks.source and ks.smem_bytes <= chunk.SMEM_BYTES
    fwd, bwd, _, _ = build_twopass(sums_and_decay, tuple(ins), (s,), _launcher=EmuLauncher)
    y, sT, ck, aux = fwd(tuple(ins), (s,))
    dx, ds = bwd((dy.to(y.dtype),), (dS,), tuple(ins), (ck,), (aux,))
    check([y, sT, *dx, *ds], sums_and_decay, ins, s, dy, dS, torch.bfloat16)


@pytest.mark.gpu
@pytest.mark.parametrize("T,M,N", [(100, 64, 64), (37, 24, 32)])
def test_vector_gradients_with_one_cta_per_sm_gpu(T, M, N):
    ins, s, dy, dS = sums_and_decay_case(T, M, N)
    f = flex_rnn_b200.jit(sums_and_decay)
    leaves = [x.cuda().requires_grad_() for x in [*ins, s]]
    y, sT = f(*leaves)
    grads = torch.autograd.grad((y, sT), leaves, (dy.cuda().to(y.dtype), dS.cuda()))
    assert f.forward_func.kernel_status("cuda:0") == 0 and f.forward_func.sources[0].name == "frnn_cfw"
    check([y.detach(), sT.detach(), *grads], sums_and_decay, ins, s, dy, dS, torch.bfloat16)
