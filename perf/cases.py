"""Representative calls of this framework for performance measurements: each case is one call of a ``jit`` step
function (``train``: forward and backward through autograd; ``infer``: forward without gradients) at sizes, data
types and layouts that the repository's configurations, examples and tests use.

``listed()`` gives the fixed cases, ``draw(rng)`` further ones of the same ranges, ``prepare`` makes a case's tensors
from a seed, ``run`` does one call and returns everything it computes, ``work`` and ``tolerance`` state what a call
cannot do without and how closely two correct implementations agree.
"""
import math
import os
import tempfile

# Compiled kernels are kept on disk, as a long-running service or a training job that restarts would keep them.
os.environ.setdefault("FRNN_CACHE_DIR", os.path.join(tempfile.gettempdir(), f"frnn_cubins_{os.getuid()}"))

import torch  # noqa: E402
import torch.nn.functional as F  # noqa: E402

import flex_rnn_b200  # noqa: E402
from flex_rnn_b200 import examples as X  # noqa: E402
from flex_rnn_b200 import workloads as W  # noqa: E402

DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16, "fp32": torch.float32}
BYTES = {"bf16": 2, "fp16": 2, "fp32": 4}

#: The inputs of a step function in call order: what each is (row [1,N], col [M,1], scalar [1,1], head scalar, head
#: matrix: the last two do not depend on batch and time), and the operations per state element of one timestep,
#: forward and backward (multiplications, additions and the terms of row and column sums).
OPS = {
    "delta_rule": (["row", "row", "col", "sc"], 6, 12),
    "gated_delta_rule": (["row", "row", "col", "sc", "sc"], 7, 15),
    "rwkv7": (["row", "row", "row", "col", "row", "row"], 9, 19),
    "mamba2": (["col", "sc", "hsc", "row", "row"], 5, 11),
    "gla": (["row", "row", "col", "row"], 5, 11),
    "mamba": (["col", "col", "hmat", "row", "row"], 7, 14),
    "hgrn": (["col", "col"], 2, 3),
}
STEPS = {op: W.STEPS[op] if op in W.STEPS else X.ZOO[op] for op in OPS}
JIT = {op: flex_rnn_b200.jit(step) for op, step in STEPS.items()}


def case(name, op, mode, B, T, H, M, N, io, state, layout="plain"):
    c = {"op": op, "mode": mode, "B": B, "T": T, "H": H, "M": M, "N": N, "io": io, "state": state, "layout": layout}
    return {"name": name, **c} if name else c


def listed():
    return [
        # one token of generation for a batch of sequences; the state stays in fp32 between calls
        case("decode_gated_delta", "gated_delta_rule", "infer", 16, 1, 32, 128, 128, "bf16", "fp32"),
        # the parity configuration: what a gradient check or a unit test of a model runs, fp32 throughout
        case("check_delta_fp32", "delta_rule", "train", 2, 64, 4, 64, 64, "fp32", "fp32"),
        # a prompt of one sequence: few (batch, head) pairs, long in time, heads of 64
        case("prompt_rwkv7_b1", "rwkv7", "infer", 1, 2048, 32, 64, 64, "bf16", "fp32"),
        # prompts of a serving batch, inputs sliced out of one fused projection
        case("prompt_mamba2_packed", "mamba2", "infer", 4, 300, 24, 64, 128, "bf16", "fp32", "packed"),
        # fine-tuning on one sequence that is no multiple of anything, inputs sliced out of one fused projection
        case("tune_gated_delta_b1", "gated_delta_rule", "train", 1, 1500, 16, 128, 128, "bf16", "bf16", "packed"),
        # ragged sizes in fp16
        case("ragged_gla_fp16", "gla", "train", 3, 777, 5, 96, 80, "fp16", "fp16"),
        # a state with 16 columns and a time-invariant matrix input, fp32 as the example script runs it
        case("train_mamba_fp32", "mamba", "train", 2, 512, 16, 128, 16, "fp32", "fp32"),
        # an elementwise gated recurrence: one column, one head as wide as the model
        case("train_hgrn", "hgrn", "train", 8, 1024, 1, 4096, 1, "bf16", "bf16"),
        # the training steps of the benchmark configurations
        case("train_delta", "delta_rule", "train", 8, 1024, 32, 128, 128, "bf16", "bf16"),
        case("train_rwkv7", "rwkv7", "train", 8, 1024, 32, 128, 128, "bf16", "bf16"),
        case("train_mamba2", "mamba2", "train", 8, 1024, 32, 64, 128, "bf16", "bf16"),
        # one GPU's share of the scaling configuration
        case("train_gated_delta_long", "gated_delta_rule", "train", 8, 4096, 32, 128, 128, "bf16", "bf16"),
    ]


def _steps(c):
    """State elements times timesteps, a training call counted as three forward ones."""
    return c["B"] * c["T"] * c["H"] * c["M"] * c["N"] * (3 if c["mode"] == "train" else 1)


LARGEST = max(_steps(c) for c in listed())


def _log(rng, lo, hi):
    return min(hi, max(lo, round(math.exp(rng.uniform(math.log(lo), math.log(hi + 0.5))))))


def draw(rng):
    """A case of the same ranges: generation, prompts and training, batches of 1 to 64, sequences of up to 4096
    timesteps, 1 to 64 heads, states of 16 to 256 rows and columns (most of them 64 or 128)."""
    op = rng.choice(["delta_rule", "gated_delta_rule", "rwkv7", "mamba2"] * 3 + ["gla"] * 2 + ["mamba", "hgrn"])
    kind = rng.choice(["decode", "prompt", "prompt", "train", "train", "train", "train"])
    side = lambda: rng.choice([64, 128, 64, 128, 64, 128, 32, 48, 96, 256, rng.randrange(16, 161, 8)])
    M = side()
    N = M if rng.random() < 0.6 else side()
    H = _log(rng, 1, 64)
    if op == "mamba":
        N = 16
    if op == "hgrn":
        M, N, H = 64 * rng.randrange(4, 65), 1, 1
    B = _log(rng, 1, 64)
    T = rng.choice([1, 1, 1, 2, 4]) if kind == "decode" else _log(rng, 16, 4096)
    io = rng.choice(["bf16", "bf16", "bf16", "fp16", "fp32"])
    state = rng.choice(["fp32", io]) if kind != "train" else rng.choice([io, io, "fp32"])
    c = case(None, op, "train" if kind == "train" else "infer", B, T, H, M, N, io, state, rng.choice(["plain", "plain", "packed"]))
    while _steps(c) > LARGEST:
        c["B" if c["B"] > 1 else "T"] = (c["B"] if c["B"] > 1 else c["T"]) // 2
    return c


def _shapes(c):
    B, T, H, M, N = (c[k] for k in "BTHMN")
    full = {"row": (B, T, H, 1, N), "col": (B, T, H, M, 1), "sc": (B, T, H, 1, 1), "hsc": (1, 1, H, 1, 1), "hmat": (1, 1, H, M, N)}
    return [full[k] for k in OPS[c["op"]][0]]


def _values(c, n):
    """The inputs in fp32, with the distributions of the benchmark configurations and of the examples."""
    unit = lambda x: F.normalize(x, dim=-1)
    s, N, op = _shapes(c), c["N"], c["op"]
    if op == "delta_rule":
        return [unit(n(s[0])), unit(n(s[1])), n(s[2]), torch.sigmoid(n(s[3]))]
    if op == "gated_delta_rule":
        return [unit(n(s[0])), unit(n(s[1])), n(s[2]), torch.exp(-F.softplus(n(s[3]))), torch.sigmoid(n(s[4]))]
    if op == "rwkv7":
        kk = unit(n(s[4]))
        return [n(s[0]) * N ** -0.5, torch.exp(-torch.exp(0.5 * n(s[1]) - 0.5)), n(s[2]) * N ** -0.5, n(s[3]), -kk,
                kk * torch.sigmoid(n(s[5]))]
    if op == "mamba2":
        return [n(s[0]), F.softplus(n(s[1]) - 1.0), -torch.exp(n(s[2])), n(s[3]) * N ** -0.5, n(s[4]) * N ** -0.5]
    if op == "gla":
        return [n(s[0]) * N ** -0.5, n(s[1]) * N ** -0.5, n(s[2]), -torch.sigmoid(n(s[3]))]
    if op == "mamba":
        return [n(s[0]), torch.sigmoid(n(s[1])), -torch.sigmoid(n(s[2])), n(s[3]), n(s[4])]
    return [n(s[0]), -torch.sigmoid(n(s[1]))]


def prepare(c, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    n = lambda shape: torch.randn(shape, generator=g, device="cuda")
    io, st = DTYPES[c["io"]], DTYPES[c["state"]]
    B, T, H, M, N = (c[k] for k in "BTHMN")
    xs = [x.to(io) for x in _values(c, n)]
    if c["layout"] == "packed":
        # the vectors of a timestep and head are slices of one projection's output (scalars come from another)
        wide = [i for i, k in enumerate(OPS[c["op"]][0]) if k in ("row", "col")]
        sizes = [xs[i].shape[3] * xs[i].shape[4] for i in wide]
        flat = torch.cat([xs[i].reshape(B, T, H, -1) for i in wide], dim=-1)
        for i, part in zip(wide, flat.split(sizes, dim=-1)):
            xs[i] = part.unsqueeze(-2) if OPS[c["op"]][0][i] == "row" else part.unsqueeze(-1)
    xs.append((0.1 * n((B, H, M, N))).to(st))
    train = c["mode"] == "train"
    s = {"op": JIT[c["op"]], "xs": [x.detach().requires_grad_(train) for x in xs], "train": train}
    if train:
        s["up"] = (n((B, T, H, M)), n((B, H, M, N)).to(st))
        # an output has the data type that the step's own arithmetic gives it
        s["up"] = (s["up"][0].to(torch.promote_types(io, st)), s["up"][1])
    return s


def run(s):
    if not s["train"]:
        with torch.no_grad():
            y, sT = s["op"](*s["xs"])
        return {"y": y, "state": sT}
    y, sT = s["op"](*s["xs"])
    return {"y": y.detach(), "state": sT.detach(), "grads": torch.autograd.grad((y, sT), s["xs"], s["up"])}


def work(c):
    """One pass: inputs and initial state read, outputs and final state written; for training also the upstream
    gradients read and all gradients written (what a backward pass reads again is not counted)."""
    B, T, H, M, N = (c[k] for k in "BTHMN")
    _, fw, bw = OPS[c["op"]]
    train = c["mode"] == "train"
    ins = sum(math.prod(s) for s in _shapes(c)) * BYTES[c["io"]]
    y = B * T * H * M * max(BYTES[c["io"]], BYTES[c["state"]])
    st = B * H * M * N * BYTES[c["state"]]
    return {"bytes": (2 if train else 1) * (ins + y + 2 * st),
            "flops": B * T * H * M * N * (fw + (bw if train else 0))}


def tolerance(c):
    """Results in fp32 only (an fp32 state makes the outputs fp32 too): what sums in another order give, since all
    arithmetic is fp32; results in 16 bits: their rounding."""
    if c["io"] == "fp32" or (c["state"] == "fp32" and c["mode"] == "infer"):
        return {"rel": 2e-5, "max": 1e-3}
    return {"rel": 1e-2 if c["io"] == "bf16" else 2e-3, "max": 0.25}
