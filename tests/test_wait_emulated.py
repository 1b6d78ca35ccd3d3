"""A wait that runs out in some threads of a chunked kernel only (chunk.py): every thread still reaches the kernel's
end, whatever the others saw, and the error word says why.

On the CPU, under the host emulation: a third of the threads are told that their first wait on one mbarrier failed.  The
emulation's barriers count threads like the hardware's, so a thread that skips a barrier the others wait at stops the run;
it runs in a process of its own with a time limit."""
import multiprocessing

import pytest
import torch

from flex_rnn_b200 import workloads as W
from flex_rnn_b200.lower import ERR_STAGE_TIMEOUT

WRAP = r"""
static thread_local int emu_waits = 0;
static bool emu_some_fail(u64* bar, u32 parity, int* err, int code) {
    const bool ok = frnn_mbar_wait(bar, parity, err, code);
    if (bar == (u64*)emu_ctx->smem + %d && threadIdx.x %% 3 == 1 && emu_waits++ == %d) { frnn_report(err, code); return false; }
    return ok;
}
#define frnn_mbar_wait emu_some_fail
extern "C" __global__"""


def _run(name, bar, nth, out):
    import dataclasses

    from emu.emu import EmuLauncher
    from flex_rnn_b200.twopass import build_twopass

    def launcher(ks):
        if ks.name == name:
            # the threads that wait for what a failed one would have done give up after a second
            src = "#undef FRNN_WAIT_LIMIT_NS\n#define FRNN_WAIT_LIMIT_NS 1000000000ull\n" + ks.source
            ks = dataclasses.replace(ks, source=src.replace('extern "C" __global__', WRAP % (bar, nth), 1))
        return EmuLauncher(ks)
    *ins, s = W.synthetic("delta_rule", 1, 48, 1, 64, 32, torch.bfloat16)[0]
    fwd, bwd, _, _ = build_twopass(W.delta_rule, tuple(ins), (s,), _launcher=launcher)
    y, sT, ck, aux = fwd(tuple(ins), (s,))
    bwd((torch.ones_like(y),), (torch.ones_like(sT),), tuple(ins), (ck,), (aux,))
    out.put(fwd.kernel_status())


# barriers by their index in shared memory: (kernel, barrier, which of a thread's waits on it)
@pytest.mark.parametrize("name,bar,nth", [("frnn_cvg", 1, 0), ("frnn_cvg", 1, 1), ("frnn_cvg", 0, 0), ("frnn_cvg", 2, 0),
                                          ("frnn_cfw", 13, 1), ("frnn_cfw", 21, 1), ("frnn_cbw", 14, 0)])
def test_some_threads_time_out(name, bar, nth):
    ctx = multiprocessing.get_context("spawn")
    out = ctx.SimpleQueue()
    p = ctx.Process(target=_run, args=(name, bar, nth, out))
    p.start()
    p.join(180)
    stranded = p.is_alive()
    if stranded:
        p.kill()
        p.join()
    assert not stranded, f"threads are stranded after a wait on barrier {bar} ran out in others"
    assert p.exitcode == 0 and out.get() == ERR_STAGE_TIMEOUT


def test_which_kernels_unroll_their_waits():
    """The recurrent backward only (its kernels measured slower with rolled waits, the others faster)."""
    from flex_rnn_b200 import chunk
    from flex_rnn_b200.twopass import generate, make_plan
    *ins, s = W.synthetic("delta_rule", 1, 64, 1, 64, 32, torch.bfloat16)[0]
    plan = make_plan(W.delta_rule, ins, (s,))[0]
    cp = chunk.chunk_plan(plan)
    for ks in (*generate(plan), cp.forward(), cp.infer(), cp.backward_scan(), cp.vector_grads()):
        assert ("#define FRNN_UNROLLED_WAITS" in ks.source) == (ks.name == "frnn_bw"), ks.name
