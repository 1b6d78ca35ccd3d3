"""Chunked form of step functions whose state update is a decay plus rank-1 terms.

Many step functions - Delta Rule, Gated Delta Rule, RWKV-7, Mamba-2, gated linear attention, retention - have the form

    sigma_d = S . alpha_d                    (row sums, d = 1..nd)
    S'      = S * w + sum_r p_r (x) kappa_r  (decay over columns, or one per head, or none; r = 1..nr)
    p_r, y  = row functions of (sigma, inputs)

with vectors alpha, kappa, w over the columns that depend on the inputs only.  ``normal_form`` finds it in a traced
step graph (``StepGraph``), whatever way the step function was written, or says that there is none.

C such steps in a row need the state only at their start:

    sigma_d,j = S_0 . (alpha_d,j * W_j-1) + sum_{i<j,r} p_r,i Gram_dr,ji,   Gram_dr,ji = alpha_d,j . (kappa_r,i * W_j-1/W_i)
    S_C       = S_0 * W_C + sum_{i,r} p_r,i (x) (kappa_r,i * W_C/W_i),      W_j = w_1 * ... * w_j

so that per chunk the state takes part in two matrix products of C columns instead of C times in two vector products,
which is work for the tensor cores (``emit_scan``).  The ratios W_j/W_i are products of the decays between, never
quotients: a decay of zero is nothing special.  The adjoint recurrence has the same form, with alpha and kappa
exchanged and time reversed, so one emitter makes the forward scan and the scan of the state gradient; the gradients of
the vectors then follow chunk by chunk, in parallel, from the states and state gradients at the chunk boundaries
(``emit_vector_grads``).

All products are fp32-accurate: an fp32 operand x enters the tf32 tensor cores as x (they read its leading 11 bits) and
as what that leaves out, rounded to 11 more; every pair of terms is multiplied, fp32 accumulators; the state itself is
accumulated by fp32 additions outside the tensor cores.
"""
from __future__ import annotations

import math
from dataclasses import dataclass, field
from typing import Callable, Dict, List, Optional, Sequence, Tuple

import torch as th

from . import lower
from .graph import MN, M1, N1, S11, Arg, Node, Shape, StepGraph
from .lower import DT_F32, ELT, KernelBuilder, KernelSource, Problem, TensorSpec, W, _contig, _elem_off, _spec_bytes, op_expr


# ---------------------------------------------------------------------------
# normal form
# ---------------------------------------------------------------------------

class _NotNormal(Exception):
    pass


@dataclass
class Normal:
    """A step function in the form above.  ``hoist``: nodes that depend on the inputs only; ``row``: nodes of the row
    functions, over the values ``sig<d>`` (row sums of the state), ``dg<k>`` (column sums of the vectors ``diags[k]``)
    and hoisted values."""
    inputs: List[str]
    shape: Dict[str, Shape]
    hoist: List[Node]
    row: List[Node]
    alphas: List[str]
    kappas: List[str]
    ps: List[str]                 # row values p_r (row or hoisted names)
    ys: List[str]
    decay: Optional[str]          # None: no decay; a column vector, or one value per head
    diags: List[str]              # vectors z_k whose column sums dg<k> the row functions read
    diag_at: List[Tuple[int, int]]    # dg<k> is the inner product of kappa_r and of alpha_d before its decay: (d, r)


@dataclass
class _Tile:
    coef: Optional[Arg]                    # factor of S: None = S does not occur, 1.0 or a name (N1 or S11)
    terms: List[Tuple[Arg, Arg]]           # (row value, column vector)


def normal_form(g: StepGraph, in_names: Sequence[str], st_name: str, n_out: int) -> Optional[Normal]:
    """``g`` computes [*outputs, new state, ...] from inputs and one state; None if it is not of the chunked form."""
    try:
        return _normal_form(g, list(in_names), st_name, n_out)
    except _NotNormal:
        return None


def _normal_form(g: StepGraph, in_names: List[str], st_name: str, n_out: int) -> Normal:
    shape = {k: v for k, v in g.shape.items()}
    hoist: List[Node] = []
    row: List[Node] = []
    val: Dict[str, object] = {}            # graph value -> Arg (free) | ("row", name) | _Tile
    known: Dict[tuple, str] = {}
    alphas: List[str] = []
    diags: List[str] = []
    rowset = set()

    def no():
        raise _NotNormal()

    def cls(a: Arg) -> Shape:
        return shape[a] if isinstance(a, str) else S11

    def is_row(a: Arg) -> bool:
        return isinstance(a, str) and a in rowset

    def mk(op: str, args: Sequence[Arg]) -> Arg:
        """A node of the hoisted or of the row graph, whichever its operands belong to."""
        args = list(args)
        if op == "mul":
            if 1.0 in args:
                args.remove(1.0)
                return args[0]
            if 0.0 in args:
                return 0.0
        if op in ("add", "sub") and args[1] == 0.0:
            return args[0]
        if op == "add" and args[0] == 0.0:
            return args[1]
        if op == "sub" and args[0] == 0.0:
            op, args = "neg", [args[1]]
        if op == "neg" and not isinstance(args[0], str):
            return -args[0]
        s = (max(cls(a)[0] for a in args), max(cls(a)[1] for a in args))
        rowy = any(is_row(a) for a in args)
        if s == MN or (rowy and s[1]):
            no()
        if op in ("mul", "add"):
            args.sort(key=lambda a: (shape.get(a) == N1, str(a)) if isinstance(a, str) else (False, str(a)))
        key = (op, *args)
        if key not in known:
            nm = f"c{len(known)}"
            known[key] = nm
            shape[nm] = s
            (row if rowy else hoist).append(Node(nm, op, args, s))
            if rowy:
                rowset.add(nm)
        return known[key]

    def factors(k: Arg) -> Tuple[Arg, Arg]:
        """A column vector as (scalar, vector): the scalar goes to the row side, so that the vectors that meet the
        state stay plain inputs where they can (16-bit inputs need no second tf32 term)."""
        n = next((n for n in hoist if n.name == k), None)
        if n is not None and n.op == "mul":
            s1, s2 = cls(n.args[0]), cls(n.args[1])
            if s2 == N1 and s1 == S11:
                f, v = factors(n.args[1])
                return mk("mul", [n.args[0], f]), v
            if s1 == N1 and s2 == N1:
                (f1, v1), (f2, v2) = factors(n.args[0]), factors(n.args[1])
                return mk("mul", [f1, f2]), mk("mul", [v1, v2])
        if n is not None and n.op == "neg" and cls(n.args[0]) == N1:
            f, v = factors(n.args[0])
            return mk("mul", [-1.0, f]), v
        return 1.0, k

    def tile_of(v) -> _Tile:
        return v if isinstance(v, _Tile) else no()

    def scale(t: _Tile, x: Arg, op: str = "mul") -> _Tile:
        if not is_row(x) and cls(x)[0] == 0:
            f = (lambda a: mk("mul", [a, x])) if op == "mul" else (lambda a: mk("div", [a, x]))
            coef = None if t.coef is None else f(t.coef)
            return _Tile(coef, [(p, f(k)) for p, k in t.terms])
        if t.coef is not None:
            no()
        return _Tile(None, [(mk(op, [p, x]), k) for p, k in t.terms])

    def neg(t: _Tile) -> _Tile:
        return _Tile(None if t.coef is None else mk("neg", [t.coef]), [(mk("neg", [p]), k) for p, k in t.terms])

    def add(a: _Tile, b: _Tile) -> _Tile:
        coef = a.coef if b.coef is None else (b.coef if a.coef is None else mk("add", [a.coef, b.coef]))
        terms = list(a.terms)
        for p, k in b.terms:
            for i, (p2, k2) in enumerate(terms):
                if k2 == k:
                    terms[i] = (mk("add", [p2, p]), k)
                    break
            else:
                terms.append((p, k))
        return _Tile(coef, terms)

    def diag(k: Arg) -> Arg:
        if not isinstance(k, str) or cls(k) != N1:
            no()
        f, k = factors(k)
        if f != 1.0:
            return mk("mul", [f, diag(k)])
        if k not in diags:
            diags.append(k)
            nm = f"dg{diags.index(k)}"
            shape[nm] = S11
            rowset.add(nm)
        return f"dg{diags.index(k)}"

    for i in in_names:
        val[i] = i
        if shape[i] == MN:
            no()
    val[st_name] = _Tile(1.0, [])
    for n in g.nodes:
        vs = [val[a] if isinstance(a, str) else a for a in n.args]
        tiles = [isinstance(v, _Tile) for v in vs]
        if n.op == "copy":
            val[n.name] = vs[0]
        elif n.op == "const":
            val[n.name] = n.args[0]
        elif n.op == "sum":
            if n.over_m or not n.over_n:
                no()
            if tiles[0]:
                t = vs[0]
                acc: Arg = 0.0
                if t.coef is not None:
                    if not isinstance(t.coef, str) or cls(t.coef) != N1:
                        no()
                    f, v = factors(t.coef)
                    if v not in alphas:
                        alphas.append(v)
                        shape[f"sig{alphas.index(v)}"] = M1
                        rowset.add(f"sig{alphas.index(v)}")
                    acc = mk("mul", [f, f"sig{alphas.index(v)}"])
                for p, k in t.terms:
                    acc = mk("add", [acc, mk("mul", [p, diag(k)])])
                val[n.name] = acc
            else:
                no()                        # sums of plain column vectors are not hoisted
        elif any(tiles):
            if n.op == "mul" and sum(tiles) == 1:
                t, x = (vs[0], vs[1]) if tiles[0] else (vs[1], vs[0])
                val[n.name] = scale(t, x)
            elif n.op == "div" and tiles[0] and not tiles[1]:
                val[n.name] = scale(vs[0], vs[1], "div")
            elif n.op == "neg":
                val[n.name] = neg(vs[0])
            elif n.op in ("add", "sub") and all(tiles):
                val[n.name] = add(vs[0], vs[1] if n.op == "add" else neg(vs[1]))
            else:
                no()
        elif n.shape == MN:
            if n.op != "mul":
                no()
            ca, cb = cls(vs[0]), cls(vs[1])
            if (ca, cb) == (M1, N1):
                val[n.name] = _Tile(None, [(vs[0], vs[1])])
            elif (ca, cb) == (N1, M1):
                val[n.name] = _Tile(None, [(vs[1], vs[0])])
            else:
                no()
        else:
            val[n.name] = mk(n.op, vs)
    ys = [val[o] for o in g.outputs[:n_out]]
    new = tile_of(val[g.outputs[n_out]])
    if any(isinstance(y, _Tile) or not isinstance(y, str) or cls(y) != M1 for y in ys):
        no()
    terms = []
    for p, k in new.terms:
        if p == 0.0 or k == 0.0:
            continue
        f, v = factors(k)
        p = mk("mul", [f, p])
        same = next((i for i, t in enumerate(terms) if t[1] == v), None)
        if same is None:
            terms.append((p, v))
        else:
            terms[same] = (mk("add", [terms[same][0], p]), v)
    if not terms or new.coef is None or any(not isinstance(k, str) or cls(k) != N1 or not isinstance(p, str) or cls(p) != M1
                                            for p, k in terms):
        no()
    decay = new.coef
    if decay == 1.0:
        decay = None
    elif not isinstance(decay, str):
        no()
    ps = [p for p, _ in terms]
    kap = [k for _, k in terms]
    by_name = {n.name: n for n in hoist}
    diag_at = []
    for z in diags:
        n = by_name.get(z)
        if n is None or n.op != "mul":
            no()
        at = None
        for k, x in ((n.args[0], n.args[1]), (n.args[1], n.args[0])):
            a = mk("mul", [decay, x]) if decay is not None and cls(decay) == N1 else x
            if k in kap and a in alphas:
                at = (alphas.index(a), kap.index(k))
        diag_at.append(at if at is not None else no())
    # only what the outputs and the state need
    need = set(ps) | set(ys) | set(alphas) | set(kap) | set(diags) | ({decay} if decay else set())
    for nodes in (row, hoist):
        for n in reversed(nodes):
            if n.name in need:
                need.update(n.value_args())
    used_sig = [f"sig{d}" in need for d in range(len(alphas))]
    if not alphas or not all(used_sig) or any(f"dg{k}" not in need for k in range(len(diags))):
        no()
    return Normal(in_names, shape, [n for n in hoist if n.name in need], [n for n in row if n.name in need], alphas, kap, ps, ys,
                  decay, diags, diag_at)


_TORCH_OPS: Dict[str, Callable] = {
    "mul": th.mul, "add": th.add, "sub": th.sub, "div": th.div, "neg": th.neg, "exp": th.exp, "log": th.log, "sqrt": th.sqrt,
    "rsqrt": th.rsqrt, "reciprocal": th.reciprocal, "abs": th.abs, "sigmoid": th.sigmoid, "tanh": th.tanh,
    "log1p": th.log1p, "expm1": th.expm1, "relu": th.relu, "erf": th.erf, "pow": th.pow,
    "copy": lambda x: x,
}


def local_vjp(nf: Normal, M: int, N: int) -> Optional[Tuple[StepGraph, bool]]:
    """The vector-Jacobian product of the row functions and of the vectors, traced: a graph with inputs [*inputs, *sig,
    *dg, *ga, *gk, (gw), *gp, *gy] (cotangents of alpha, kappa, decay, p, y) and outputs [*d inputs, *d sig], and
    whether the decay is an exponential and gw the cotangent of its exponent; None where an operation has no derivative
    here."""
    from torch.fx.experimental.proxy_tensor import make_fx
    from .graph import UnsupportedStepOp, from_fx
    from .trace import clean_dispatch
    if any(n.op not in _TORCH_OPS for n in nf.hoist + nf.row):
        return None
    extra = [f"sig{d}" for d in range(len(nf.alphas))] + [f"dg{k}" for k in range(len(nf.diags))]
    names = list(nf.inputs) + extra
    dims = (max(2, M), max(2, N))
    nin = len(nf.inputs)
    by_name = {n.name: n for n in nf.hoist}
    dn = by_name.get(nf.decay)
    log_decay = dn is not None and dn.op == "exp" and isinstance(dn.args[0], str)
    vectors = nf.alphas + nf.kappas + ([dn.args[0] if log_decay else nf.decay] if nf.decay else [])

    def evaluate(a, outs, diags):
        env: Dict[str, th.Tensor] = dict(zip(names, a))
        get = lambda x: env[x] if isinstance(x, str) else x
        for n in nf.hoist + (nf.row if len(a) == len(names) else []):
            args = [get(x) for x in n.args]
            if not any(isinstance(x, th.Tensor) for x in args):
                raise UnsupportedStepOp("literal operands only")
            if n.op in ("mul", "add", "sub", "div") and not isinstance(args[0], th.Tensor):
                args[0] = th.full((1, 1), args[0], device="meta")
            env[n.name] = _TORCH_OPS[n.op](*args)
        return tuple(env[o] * 1.0 for o in outs) + tuple(env[z].sum(-1, True) for z in diags)

    try:
        with clean_dispatch():
            args = [th.empty(dims[0] if nf.shape[n][0] else 1, dims[1] if nf.shape[n][1] else 1, device="meta") for n in names]

            def joint(*a):
                x, gv, gr = a[:len(args)], a[len(args):len(args) + len(vectors)], a[len(args) + len(vectors):]
                _, pull = th.func.vjp(lambda *z: evaluate(z, nf.ps + nf.ys, ()), *x)
                d_row = pull(tuple(gr))
                _, pull = th.func.vjp(lambda *z: evaluate(z, vectors, nf.diags), *x[:nin])
                d_vec = pull(tuple(gv) + tuple(d_row[nin + len(nf.alphas):]))
                return tuple(r + v for r, v in zip(d_row, d_vec)) + tuple(d_row[nin:nin + len(nf.alphas)])
            outs = evaluate(args[:nin], vectors, ()) + evaluate(args, nf.ps + nf.ys, ())
            gm = make_fx(joint)(*args, *[th.empty_like(o) for o in outs])
        gj = from_fx(gm, "local_vjp", dims)
    except (UnsupportedStepOp, KeyError):
        return None
    ren = dict(zip(gj.inputs, names + [f"ga{d}" for d in range(len(nf.alphas))] + [f"gk{r}" for r in range(len(nf.kappas))]
                   + (["gw"] if nf.decay else []) + [f"gp{r}" for r in range(len(nf.ps))] + [f"gy{j}" for j in range(len(nf.ys))]))
    for n in gj.nodes:
        ren[n.name] = "b_" + n.name
    f = lambda a: ren.get(a, a) if isinstance(a, str) else a
    return simplified(StepGraph("local_vjp", [f(i) for i in gj.inputs],
                                [Node(f(n.name), n.op, [f(a) for a in n.args], n.shape, n.over_m, n.over_n) for n in gj.nodes],
                                [f(o) for o in gj.outputs], {f(k): v for k, v in gj.shape.items()})), log_decay


def simplified(g: StepGraph) -> StepGraph:
    """``g`` without multiplications by one or zero, copies, repeated expressions and dead nodes."""
    alias: Dict[str, Arg] = {}
    known: Dict[tuple, str] = {}
    nodes: List[Node] = []
    f = lambda a: alias.get(a, a) if isinstance(a, str) else a
    for n in g.nodes:
        args = [f(a) for a in n.args]
        if n.op == "copy" or (n.op == "mul" and 1.0 in args and any(isinstance(a, str) for a in args)):
            rest = [a for a in args if a != 1.0]
            alias[n.name] = rest[0]
            continue
        if n.op == "const":
            alias[n.name] = n.args[0]
            continue
        if n.op == "mul" and 0.0 in args or (n.op == "sum" and args[0] == 0.0) or (n.op == "neg" and args[0] == 0.0):
            alias[n.name] = 0.0
            continue
        if n.op == "add" and 0.0 in args:
            alias[n.name] = args[1] if args[0] == 0.0 else args[0]
            continue
        key = (n.op, n.over_m, n.over_n, *args)
        if key in known:
            alias[n.name] = known[key]
            continue
        known[key] = n.name
        nodes.append(Node(n.name, n.op, args, n.shape, n.over_m, n.over_n))
    g2 = StepGraph(g.name, list(g.inputs), nodes, [f(o) for o in g.outputs], dict(g.shape))
    return g2.pruned(g2.outputs, g2.name)


# ---------------------------------------------------------------------------
# the scan over chunks
# ---------------------------------------------------------------------------

_CHUNK_PRELUDE: Optional[str] = None


def chunk_prelude() -> str:
    global _CHUNK_PRELUDE
    if _CHUNK_PRELUDE is None:
        import os
        from .twopass import prelude
        with open(os.path.join(os.path.dirname(os.path.abspath(__file__)), "csrc", "frnn_chunk.cuh")) as f:
            _CHUNK_PRELUDE = prelude() + f.read()
    return _CHUNK_PRELUDE


@dataclass
class Staged:
    """One per-timestep vector a chunked kernel reads: see ``KernelBuilder.add_item``."""
    key: str
    cls: Shape
    spec: TensorSpec
    ptr: str
    dims: Dict[str, int]
    const_off: int = 0


@dataclass
class ScanSpec:
    """What ``emit_scan`` makes a kernel of: a recurrence in the chunked form (module docstring)."""
    name: str
    params: List[Tuple[str, str, bool, int]]         # (name, C type, read only, bytes)
    items: List[Staged]
    const_scalars: List[Tuple[str, TensorSpec, str]]  # time-invariant [1,1] inputs: (name, spec, pointer)
    shape: Dict[str, Shape]
    hoist: List[Node]
    row: List[Node]
    alphas: List[str]
    kappas: List[str]
    ps: List[str]
    decay: Optional[str]
    diags: List[str]
    diag_at: List[Tuple[int, int]]
    outs: List[Tuple[str, int, str, Callable[[str], str], int]]   # (row value, dtype, pointer, element offset of row m0's head at time t, row stride)
    init: Tuple[TensorSpec, str]
    final: Tuple[TensorSpec, str]
    dg_out: Optional[str]                            # where to keep the dg<k>, [k, B, H, T] fp32
    ckpt: Optional[str]                              # state at each chunk's start (in processing order), [B, H, chunk, N, M] fp32
    reverse: bool


SMEM_BYTES = 227 * 1024
SCAN_PREP = 256          # threads that prepare the vectors (beside the 128 that own the state's rows)
TMEM_COLS = 512


def _tmem_pow2(cols: int) -> int:
    c = 32
    while c < cols:
        c *= 2
    return c


class ColumnCode:
    """Code for one column n of the hoisted column vectors at one timestep, read from the raw stage buffer: the
    vectors are evaluated where they are used, in registers, and never stored as fp32."""

    def __init__(self, kb: KernelBuilder, hoist: Sequence[Node], shape: Dict[str, Shape], scalar: Callable[[str], str]):
        self.kb, self.shape, self.scalar = kb, shape, scalar
        self.nodes = {n.name: n for n in hoist}

    def scalars(self, names: Sequence[str]) -> List[str]:
        """The [1,1] values that the vectors ``names`` are made of."""
        out: List[str] = []

        def visit(a):
            if not isinstance(a, str):
                return
            if self.shape[a] == S11:
                if a not in out:
                    out.append(a)
            elif a in self.nodes:
                for x in self.nodes[a].args:
                    visit(x)
        for n in names:
            visit(n)
        return out

    def leaves(self, names: Sequence[str]) -> List[str]:
        """The staged vectors that the vectors ``names`` are made of."""
        out: List[str] = []

        def visit(a):
            if not isinstance(a, str) or self.shape[a] == S11:
                return
            if a in self.nodes:
                for x in self.nodes[a].args:
                    visit(x)
            elif a not in out:
                out.append(a)
        for n in names:
            visit(n)
        return out

    def load(self, a: str, stage: str, tl: str, n: str) -> str:
        it = self.kb.item_by_key[a]
        return f"frnn_io<{it.dt}>::ld({stage} + {it.off} + ({tl}) * {it.rowb}, {n})"

    def emit(self, names: Sequence[str], stage: str, tl: str, n: str, pre: str, given: Optional[Dict[str, str]] = None) -> Dict[str, str]:
        """Declare the values of ``names`` (and what they need) as floats with prefix ``pre``; ``given``: staged vectors
        that are in registers already."""
        w, done = self.kb.w, dict(given or {})

        def visit(a) -> str:
            if not isinstance(a, str):
                return lower.flit(a)
            if a in done:
                return done[a]
            v = pre + a.replace(".", "_")
            if self.shape[a] == S11:
                w(f"const float {v} = {self.scalar(a)};")
            elif a in self.nodes:
                ops = [visit(x) for x in self.nodes[a].args]
                w(f"const float {v} = {op_expr(self.nodes[a], ops)};")
            else:
                w(f"const float {v} = {self.load(a, stage, tl, n)};")
            done[a] = v
            return v
        for nm in names:
            visit(nm)
        return done


def row_closure(nodes: Sequence[Node], names: Sequence[Arg], made: Sequence[str] = ()) -> set:
    """``names`` and everything that they are computed from, except what is ``made`` and what only that is computed from."""
    need = {a for a in names if isinstance(a, str)}
    for n in reversed(nodes):
        if n.name in need and n.name not in made:
            need.update(n.value_args())
    return need - set(made)


#: operations of more than a few instructions
COSTLY = ("div", "exp", "log", "sqrt", "rsqrt", "reciprocal", "sigmoid", "tanh", "log1p", "expm1", "erf", "pow")


def exact_vectors(names: Sequence[str], items: Sequence[Staged], decay_vec: bool) -> bool:
    """Whether the vectors are plain 16-bit inputs, which tf32 holds exactly."""
    dt = {it.key: it.spec.dt for it in items}
    return not decay_vec and all(dt.get(n) in (lower.DT_BF16, lower.DT_F16) for n in names)


def emit_scan(p: Problem, s: ScanSpec, C: int, MB: int, use_tma: bool = True, state_unroll: int = 0, compact: bool = False) -> KernelSource:
    """Scan over chunks of ``C`` timesteps; a CTA owns ``MB`` <= 128 rows of one (b, h).

    Row m of the state lives in lane m of Tensor Memory (columns: S, then what tf32 truncation leaves out of it), and
    state thread m does everything that concerns the row.  Per chunk:

      products 1   S . alpha for all C steps: [S and rest of S] x [alpha | rest of alpha]
      rows         forward substitution over the steps: sigma, row functions, outputs; p goes to Tensor Memory
      products 2   sum_i p_i (x) kappa_i
      state        S = S * W_C + that, in fp32 registers; rest of S; checkpoint

    One warp issues all products.  Products 1 start on the first columns of the new state while the state threads are
    still at the others.  Eight more warps keep a chunk ahead: raw inputs by TMA, row vectors and scalars in fp32, the
    operands alpha and kappa in the tensor cores' layout (thread n converts column n), and the C x C inner products Gram
    of the vectors, on the tensor cores too, while the state threads are at the substitution.  Decays over columns are folded into the operands (alpha W_j-1, kappa W_C/W_i), decays per head
    stay scalars on the row side, so that vectors that are plain 16-bit inputs remain exact in tf32 and need no second
    term.  Gram needs the ratios W_j-1/W_i: as kappa/W_i where no W of the chunk is tiny, else (a reset, an extreme
    decay) as running products, by a slower path for that chunk alone.

    The chain of one chunk - products 1, substitution, products 2, state - bounds the kernel.
    """
    import types
    from .lower import Body
    N, nd, nr = p.N, len(s.alphas), len(s.kappas)
    Np = (N + 15) // 16 * 16
    PT = SCAN_PREP
    Tl = types.SimpleNamespace(MB=MB, NT=PT, R=1, C=1)
    kb = KernelBuilder(p, Tl, C, use_tma)
    w = kb.w
    for nm, ct, const, nb in s.params:
        kb.add_param(nm, ct, const, nb)
    for nm, spec, ptr in s.const_scalars:
        kb.const_scalars[nm] = f"{lower.vname(nm)}[0]"
    for it in s.items:
        kb.add_item(it.key, it.cls, it.spec, it.ptr, it.dims, it.const_off)
    dec_vec = bool(s.decay) and s.shape[s.decay] == N1
    dec_sc = bool(s.decay) and not dec_vec
    xa, xk = exact_vectors(s.alphas, s.items, dec_vec), exact_vectors(s.kappas, s.items, dec_vec)
    row_names = {n.name for n in s.row}
    special = {f"sig{d}" for d in range(nd)} | {f"dg{k}" for k in range(len(s.diags))}
    col = ColumnCode(kb, s.hoist, s.shape, lambda a: "")
    need: List[str] = []            # hoisted row vectors and scalars
    for a in [a for n in s.row for a in n.value_args()] + list(s.ps) + [o[0] for o in s.outs]:
        if a not in row_names and a not in special and a not in need:
            need.append(a)
    row_in = list(need)
    vec_names = s.alphas + s.kappas + ([s.decay] if dec_vec else []) + s.diags
    for a in col.scalars(vec_names) + ([s.decay] if dec_sc else []):
        if a not in need:
            need.append(a)
    if any(nm in kb.const_scalars for nm in need):
        raise lower.LoweringError("a time-invariant scalar is read directly")
    g = StepGraph("vec", [it.key for it in s.items] + list(kb.const_scalars), list(s.hoist), need, dict(s.shape))
    kb.plan([g.pruned(need)], need)
    mk_row = 0
    for want, ln in ((M1, MB), (S11, 1)):
        mk_row = (mk_row + 3) // 4 * 4
        for nm, (cls, _) in list(kb.wk.items()):
            if cls == want:
                kb.wk[nm] = (cls, mk_row)
                mk_row += ln
    mk_row = (mk_row + 3) // 4 * 4
    # shared memory
    al = lambda x: (x + 127) // 128 * 128
    nA, nK = nd * C, nr * C
    RA, RK = nA * (1 if xa else 2), nK * (1 if xk else 2)
    if nA > 128:              # Gram has them as rows: lanes of Tensor Memory
        raise lower.LoweringError("the row sums of a chunk have more rows than a product")
    GS = C + 4
    gram_f = nd * nr * C * GS
    dec_f = Np if dec_vec else (3 * C if dec_sc else 0)        # W_C; or, per head, W_j-1 | W_C/W_i | W_C: three of them, the
    o_dec = 0                                                  # state threads still read one when gram is free again
    o_dg = gram_f
    o_end = o_dg + (len(s.diags) * C + 3) // 4 * 4
    lboA, lboH, lboK = RA * 16 + 16, RK * 16 + 16, Np * 16
    # two buffers of raw inputs, or one where two do not fit (the next copies then wait for the last column to be read)
    for NS in (2, 1):
        off_stage = 256
        off_mk = off_stage + NS * al(kb.stage_bytes)
        mk_bytes = al(mk_row * C * 4)
        off_gr = off_mk + 2 * mk_bytes
        gr_bytes = al(o_end * 4)
        off_dec = off_gr + 2 * gr_bytes
        off_al = off_dec + al(3 * dec_f * 4)
        al_bytes = al((N // 4 - 1) * lboA + max(2048 + 16, lboA))     # Gram reads 128 rows of alpha, whatever is there
        off_ka = off_al + 2 * al_bytes
        ka_bytes = al(nK // 4 * lboK)
        off_kh = off_ka + (1 if xk else 2) * ka_bytes
        smem_bytes = off_kh + al(N // 4 * lboH)
        if smem_bytes <= SMEM_BYTES:
            break
    # Tensor Memory columns: S | rest of S | products 2 | p | rest of p, over products 1 (read before p is written) | Gram
    colS, colL, colD, colP = 0, Np, 2 * Np, 3 * Np
    colA = colP
    colG = colP + max(2 * nK, RA)
    # the row sums that a p depends on (products 2 wait for them), and the others, which only outputs depend on
    p_need, out_names = row_closure(s.row, s.ps), [o[0] for o in s.outs]
    # what the outputs take over from the p instead of computing it again: the p themselves and costly values on the way to them
    # (64x64, 64 heads, T1024, backward scan, with p computed twice and once: y = (S q)^2 368 and 212 us, two such sums 1347 and 697)
    made = [nm for nm in s.ps if nm in {n.name for n in s.row}]
    kept: List[str] = []
    for n in reversed(s.row):
        if n.op in COSTLY and n.name in p_need & row_closure(s.row, out_names, made + kept):
            kept.append(n.name)
    o_need = row_closure(s.row, out_names, made + kept)
    first_sums = [d for d in range(nd) if f"sig{d}" in p_need]
    other_sums = [d for d in range(nd) if d not in first_sums]
    p_early = not first_sums and colP + 2 * nK + RA + RK <= TMEM_COLS      # p beside products 1, not over them
    if p_early:
        colA, colG = colP + 2 * nK, colP + 2 * nK + RA
    late_gram = colG + RK > TMEM_COLS and RA + RK <= 2 * nK
    if late_gram:                     # Gram over p as well: read before p is written, computed once products 2 have read p
        colG = colP + RA
    tm_cols = _tmem_pow2(max(colG + RK, colP + 2 * nK))
    if tm_cols > TMEM_COLS:
        raise lower.LoweringError("the chunk's operands do not fit Tensor Memory")
    nchunk = (p.T + C - 1) // C
    B_RAW, B_AF, B_AE, B_HF, B_KF, B_KE, B_GF, B_GE, B_M1, B_M2, B_SB, B_PB, B_HS, B_MG, B_SE = 0, 2, 4, 6, 7, 8, 9, 11, 13, 14, 15, 19, 20, 21, 25
    nblk = Np // 16
    quarters = [(nblk * q // min(4, nblk) * 16, nblk * (q + 1) // min(4, nblk) * 16) for q in range(min(4, nblk))]
    whole = p.T % C == 0
    ERR = lower.ERR_STAGE_TIMEOUT

    w(lower._header(chunk_prelude()))
    w(f"// chunked scan {s.name}: B={p.B} T={p.T} H={p.H} M={p.M} N={N}; {MB} rows per CTA, {C} steps per chunk, {nd} row sums, "
      f"{nr} rank-1 terms" + (", reversed" if s.reverse else ""))
    kb.emit_tma_issue("sc_issue")
    w(f'extern "C" __global__ void __launch_bounds__({128 + PT + 128}, 1)')
    w.open(f"{s.name}({', '.join(kb.param_decl)})")
    w("FRNN_DYN_SMEM(smem);")
    w("const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5; (void)lane;")
    w(f"const int m0 = blockIdx.x * {MB}, h = blockIdx.y, b = blockIdx.z; (void)m0; (void)h; (void)b;")
    kb.emit_bounds_prologue()
    w("u64* bar = (u64*)smem;")
    w(f"unsigned char* kappaB = smem + {off_ka};")
    w.open("if (tid == 0)")
    for bi, cnt in ((B_RAW, 1), (B_RAW + 1, 1), (B_AF, 128), (B_AF + 1, 128), (B_AE, 1), (B_AE + 1, 1), (B_HF, 128), (B_KF, 128),
                    (B_KE, 1), (B_GF, PT), (B_GF + 1, PT), (B_GE, 128), (B_GE + 1, 128), (B_M1, 1), (B_M2, 1), (B_SB, 128),
                    (B_SB + 1, 128), (B_SB + 2, 128), (B_SB + 3, 128), (B_PB, 128), (B_HS, PT), (B_MG, 1), (B_SE, PT), (B_SE + 1, PT)):
        w(f"frnn_mbar_init(&bar[{bi}], {cnt});")
    w("((int*)&bar[23])[0] = 0;      // warps that are done with Tensor Memory")
    w("bar[24] = 0;                  // two ints: a chunk (even, odd) whose decays are too small to divide by, its number plus one")
    w("frnn_mbar_init_fence();")
    w.close()
    w.open("if (warp == 0)")
    w(f"frnn_tmem_alloc((u32*)&bar[22], {tm_cols}u);")
    w("frnn_tmem_fence_before_sync();")
    w.close()
    w("frnn_block_sync();")
    w("frnn_tmem_fence_after_sync();")
    w("const u32 tm = *(volatile u32*)&bar[22];")
    tma_call = (", " + kb.tma_issue_call) if kb.tma_items else ""

    def chunk_head():
        """kc: the chunk in time order, t0 / nv: its first timestep and length."""
        w(f"const int kc = {f'{nchunk - 1} - c' if s.reverse else 'c'}, t0 = kc * {C}, nv = min({C}, {p.T} - t0), buf = c & 1; (void)kc;")
        w(f"{{0}}float* mk = ({{0}}float*)(smem + {off_mk} + buf * {mk_bytes}); (void)mk;")
        w(f"{{0}}float* gram = ({{0}}float*)(smem + {off_gr} + buf * {gr_bytes});")
        if dec_f:
            w(f"{{0}}float* dec = ({{0}}float*)(smem + {off_dec} + (c % 3) * {dec_f * 4}); (void)dec;")

    def head(const: str):
        n0 = len(w.lines)
        chunk_head()
        for i in range(n0, len(w.lines)):
            w.lines[i] = w.lines[i].replace("{0}", const)
    pos = (lambda q: f"({C - 1 if whole else 'nv - 1'} - ({q}))") if s.reverse else (lambda q: f"({q})")

    # ------------------------------------------------------------------ preparing warps
    # registers: 512 threads start with 128 each; the state's rows need more, the others less (state, preparing twice, products:
    # 4 x 128 together).  A preparing thread holds nK values of kappa.  With 64 of them either split spills 10 to 100 bytes and
    # they measure alike (backward of 256 heads T512, 128x128: Delta Rule 653 us both, Gated Delta 797 against 794 us); with 32
    # the second is the better one (RWKV-7 forward, 128x64: 365 against 382 us) or equal within 1 %.
    regs = (192, 112, 96) if nK >= 64 else (200, 104, 104)
    w("auto work = [&]() -> void {")
    w.ind += 1
    w.open(f"if (tid >= 128 && tid < {128 + PT})")
    w(f"frnn_regs_release<{regs[1]}>();")
    w("const int hl = tid - 128, hw = hl >> 5; (void)hw;")
    w("u32 hs_par = 0; (void)hs_par;")
    w(f"float k[{nr}][{C}];     // kappa of the last chunk: stored when the products of the chunk before are complete")

    def put_kappa():
        """Column hl of kappa of chunk c - 1, from registers to the operand."""
        w(f"if (c > 1 && !frnn_mbar_wait(&bar[{B_KE}], c & 1, err, {ERR})) return;      // products 2 of chunk c - 2 are complete")
        w.open(f"if (hl < {Np})")
        w("#pragma unroll")
        w.open(f"for (int q = 0; q < {C}; q += 4)")
        for r in range(nr):
            w(f"unsigned char* dst{r} = kappaB + (({r * C} + q) >> 2) * {lboK} + (hl >> 3) * 128 + (hl & 7) * 16;")
            if xk:
                w(f"frnn_stv<0,4>(dst{r}, 0, &k[{r}][q]);")
            else:
                w(f"{{ float hi[4]; for (int e = 0; e < 4; e++) {{ hi[e] = k[{r}][q + e]; k[{r}][q + e] = frnn_tf32_rest(hi[e]); }}")
                w(f"frnn_stv<0,4>(dst{r}, 0, hi); frnn_stv<0,4>(dst{r} + {ka_bytes}, 0, &k[{r}][q]); }}")
        w.close()
        w.close()
        w("frnn_async_proxy_fence();")
        w(f"frnn_mbar_arrive(&bar[{B_KF}]);")
    for nm, spec, ptr in s.const_scalars:
        kb.emit_const_input(Body(w, Tl, {}, False, False), nm, S11, spec, ptr, lower.IN_DIMS)

    def hsync():
        w(f"frnn_mbar_arrive(&bar[{B_HS}]); if (!frnn_mbar_wait(&bar[{B_HS}], hs_par, err, {ERR})) return; hs_par ^= 1;")

    def h_issue(t0e, nve, be):
        """Plain copies of one chunk into stage buffer ``be`` (inputs no tensor copy reaches)."""
        if kb.plain_items:
            w.open("")
            w(f"unsigned char* stage = smem + {off_stage} + (({be}) % {NS}) * {al(kb.stage_bytes)}; (void)stage;")
            kb.emit_plain_direct("stage", t0e, nve, "hl", PT)
            w.close()
    first = nchunk - 1 if s.reverse else 0
    h_issue(str(first * C), str(min(C, p.T - first * C)), "0")
    w("#pragma unroll 1")
    w.open(f"for (int c = 0; c < {nchunk}; c++)")
    head("")
    w(f"const unsigned char* stage = smem + {off_stage} + (c % {NS}) * {al(kb.stage_bytes)};")
    w(f"unsigned char* alphaB = smem + {off_al} + buf * {al_bytes};")
    def next_plain():
        if kb.plain_items:
            nxt = f"(kc {'-' if s.reverse else '+'} 1)"
            w.open(f"if (c + 1 < {nchunk})")
            h_issue(f"{nxt} * {C}", f"min({C}, {p.T} - {nxt} * {C})", "c + 1")
            w.close()
    if NS == 2:
        next_plain()
    if kb.tma_items:
        w(f"if (!frnn_mbar_wait(&bar[{B_RAW} + c % {NS}], (c / {NS}) & 1, err, {ERR})) return;")
    if kb.plain_items:
        hsync()
    w(f"if (c >= 2 && !frnn_mbar_wait(&bar[{B_GE} + buf], ((c >> 1) - 1) & 1, err, {ERR})) return;")
    if kb.wk:
        kb.emit_convert("stage", "mk", "nv", "hl", PT, rows={M1: ("mk", mk_row), S11: ("mk", mk_row)})
        w(f"for (int e = hl; e < ({C} - nv) * {mk_row}; e += {PT}) mk[nv * {mk_row} + e] = 0.0f;")
    col.scalar = lambda a: f"mk[tl * {mk_row} + {kb.wk[a][1]}]"
    if col.scalars(vec_names) or dec_sc:
        hsync()
    if dec_sc:
        od = kb.wk[s.decay][1]
        # lane q: the products of the decays before step q and after it, doubling the steps that a product covers
        w.open("if (hw == 0)")
        w("const int j = lane;")
        ok = " && ".join((["j < " + str(C)] if C < 32 else []) + ([] if whole else ["j < nv"]))
        x = f"mk[max({pos('j')}, 0) * {mk_row} + {od}]"
        w("float W = " + (f"({ok}) ? {x} : 1.0f" if ok else x) + ", before = 1.0f, after = 1.0f;")
        w("#pragma unroll")
        w("for (int o = 1; o < 32; o <<= 1) { const float x = frnn_shfl_xor(W, o); if (j & o) before *= x; else after *= x; W *= x; }")
        w((f"if (j < {C}) " if C < 32 else "") + f"{{ dec[{o_dec} + j] = before; dec[{o_dec + C} + j] = after; }}")
        w(f"if (j == 0) dec[{o_dec + 2 * C}] = W;")
        w.close()

    def steps(names, n, body):
        """``body(values)`` for the steps q of the chunk in order, eight at a time: their loads come before the first
        store, which the compiler would not move them across (a step at a time cost 240 cycles, all of them latencies)."""
        lv = col.leaves(names)
        where = (lambda q: f"const bool live = true; const int tl = {pos(q)}; (void)live; (void)tl;") if whole else \
            (lambda q: f"const bool live = {q} < nv; const int tl = live ? {pos(q)} : 0; (void)live; (void)tl;")
        for q8 in range(0, C, 8):
            w.open("")
            for a in lv:
                w(f"float l_{a.replace('.', '_')}[8];")
            w("#pragma unroll")
            w.open("for (int e = 0; e < 8; e++)")
            w(where(f"({q8} + e)"))
            for a in lv:
                w(f"l_{a.replace('.', '_')}[e] = {col.load(a, 'stage', 'tl', n)};")
            w.close()
            w("#pragma unroll")
            w.open("for (int e = 0; e < 8; e++)")
            w(f"const int q = {q8} + e;")
            w(where("q"))
            body(col.emit(names, "stage", "tl", n, "x_", {a: f"l_{a.replace('.', '_')}[e]" for a in lv}))
            w.close()
            w.close()

    def put_km(base, lbo, row, n, val):
        """Store into a K-major operand over columns: element (row, n)."""
        w(f"*(float*)({base} + ({n} >> 2) * {lbo} + (({row}) >> 3) * 128 + (({row}) & 7) * 16 + ({n} & 3) * 4) = {val};")
    # --- thread n of the first four warps: column n of alpha (times the decays before the step) and of kappa (times those
    # after it)
    w.open("if (hl < 128)")
    w.open("if (c > 0)")
    put_kappa()
    w.close()
    w(f"if (c >= 2 && !frnn_mbar_wait(&bar[{B_AE} + buf], ((c >> 1) - 1) & 1, err, {ERR})) return;   // products 1 two chunks back are complete")
    w(f"float x[{C if dec_vec else 1}]; (void)x;")
    w.open(f"if (hl < {N})")
    w("float W = 1.0f; (void)W;")

    def alpha_step(v):
        for d, nm in enumerate(s.alphas):
            w(f"const float a{d} = live ? {v[nm]}{' * W' if dec_vec else ''} : 0.0f;")
            put_km("alphaB", lboA, f"{d * C} + q", "hl", f"a{d}")
            if not xa:
                put_km("alphaB", lboA, f"{nA + d * C} + q", "hl", f"frnn_tf32_rest(a{d})")
        for r, nm in enumerate(s.kappas):
            w(f"k[{r}][q] = live ? {v[nm]} : 0.0f;")
        if dec_vec:
            w(f"x[q] = live ? {v[s.decay]} : 1.0f; W *= x[q];")
    steps(s.alphas + s.kappas + ([s.decay] if dec_vec else []), "hl", alpha_step)
    if dec_vec:
        w(f"dec[{o_dec} + hl] = W;")
    w.close()
    w.open("else")
    w("#pragma unroll")
    w(f"for (int q = 0; q < {C}; q++) {{ " + " ".join(f"k[{r}][q] = 0.0f;" for r in range(nr)) + " }")
    if dec_vec:
        w("#pragma unroll")
        w(f"for (int q = 0; q < {C}; q++) x[q] = 1.0f;")
        if Np > N:
            w(f"if (hl < {Np}) dec[{o_dec} + hl] = 1.0f;")
    w.close()
    w("frnn_async_proxy_fence();")
    w(f"frnn_mbar_arrive(&bar[{B_AF} + buf]);")
    if dec_vec:
        w("float S = 1.0f;")
        w("#pragma unroll")
        w(f"for (int q = {C - 1}; q >= 0; q--) {{ " + " ".join(f"k[{r}][q] *= S;" for r in range(nr)) + " S *= x[q]; }")
    w.close()
    # --- thread n of the last four warps: column n of kappa over W, for Gram (its previous products are complete: below)
    w.open("else")
    w("const int n = hl - 128;")
    w.open(f"if (n < {N})")
    if dec_vec:
        w("float W = 1.0f, R = 1.0f, wlo = 1.0f, whi = 1.0f;")

    def kappa_step(v):
        if dec_vec:
            w(f"const float x = live ? {v[s.decay]} : 1.0f;")
            w("W *= x; R *= frnn_rcp1(x); wlo = fminf(wlo, fabsf(W)); whi = fmaxf(whi, fabsf(W));")
        for r, nm in enumerate(s.kappas):
            w(f"const float y{r} = live ? {v[nm]}{' * R' if dec_vec else ''} : 0.0f;")
            put_km(f"(smem + {off_kh})", lboH, f"{r * C} + q", "n", f"y{r}")
            if not xk:
                put_km(f"(smem + {off_kh})", lboH, f"{nK + r * C} + q", "n", f"frnn_tf32_rest(y{r})")
    steps(s.kappas + ([s.decay] if dec_vec else []), "n", kappa_step)
    if dec_vec:
        w("if (!(wlo > 1e-25f && whi < 1e25f)) ((volatile int*)&bar[24])[buf] = c + 1;")
    w.close()
    w("frnn_async_proxy_fence();")
    w(f"frnn_mbar_arrive(&bar[{B_HF}]);")
    w.close()
    if not dec_vec:
        w(f"frnn_mbar_arrive(&bar[{B_SE} + c % {NS}]);       // the raw inputs are read")
    # --- Gram: alpha against kappa, rows (d, j), columns (r, i)
    w(f"if (!frnn_mbar_wait(&bar[{B_MG}], c & 1, err, {ERR})) return;")
    slow = "((volatile int*)&bar[24])[buf] == c + 1"
    if dec_vec:
        w(f"const bool slow = {slow};")
        w.open("if (!slow)")
    w("frnn_tmem_fence_after_sync();")
    w("const u32 gt = tm + frnn_tmem_lane_base(hw);")
    # the rows' two halves of the threads take half of the columns each, where that is whole vectors or half of the only one
    parts = 2 if nr == 1 or nr % 2 == 0 else 1
    KC = nK // parts
    w(f"const int ml = hl & 127, half = hl >> 7, d = ml / {C}, j = ml % {C}; (void)d; (void)j; (void)half;")
    w.open(f"if (ml < {(nA + 31) // 32 * 32}" + (" && half == 0)" if parts == 1 else ")"))
    w(f"const int i0 = half * {KC if parts == 2 else 0}; (void)i0;")
    w(f"float v[{KC}];")
    w(f"frnn_tmem_ld<{KC}>(gt + {colG}u + (u32)i0, v);")
    if not xk:
        w(f"float u[{KC}];")
        w(f"frnn_tmem_ld<{KC}>(gt + {colG + nK}u + (u32)i0, u);")
    w("frnn_tmem_wait_ld();")
    w.open(f"if (ml < {nA})")
    if not xk:
        w("#pragma unroll")
        w(f"for (int i = 0; i < {KC}; i++) v[i] += u[i];")
    for k in range(len(s.diags)):
        d_, r_ = s.diag_at[k]
        w.open(f"if (d == {d_} && j >= i0 - {r_ * C} && j < i0 - {r_ * C} + {KC})")
        w("float z = 0.0f;")
        w("#pragma unroll")
        w(f"for (int i = 0; i < {KC}; i++) z = i0 + i == {r_ * C} + j ? v[i] : z;")
        w(f"gram[{o_dg + k * C} + j] = z;")
        if s.dg_out:
            w(f"if (j < nv) frnn_st_raw<float>({s.dg_out}, {dg_off(p, k, f't0 + {pos(chr(106))}')}, z);")
        w.close()
    if dec_sc:
        # the decays between step j and step i, from the last i to the first; all of them are loaded first: loaded where the running
        # product wants them, each waited for the one before (4700 of a chunk's 16000 cycles, Gated Delta Rule backward)
        xs = lambda q: f"mk[max({pos(q)}, 0) * {mk_row} + {od}]"
        per = min(KC, C)                 # positions of one vector that a half holds
        live = lambda i: "" if whole else f" && {i} < nv"
        w(f"float W = 1.0f, xv[{per}];")
        if per < C:
            w("#pragma unroll")
            w(f"for (int i = 0; i < {C - per}; i++) xv[i] = {xs(f'({per} + i)')};")
            w("#pragma unroll")
            w(f"for (int i = {C - per - 1}; i >= 0; i--) W *= half == 0 && {per} + i < j{live(f'{per} + i')} ? xv[i] : 1.0f;")
        w("#pragma unroll")
        w(f"for (int i = 0; i < {per}; i++) xv[i] = {xs('(i0 + i)' if per < C else 'i')};")
        w("#pragma unroll")
        at = "i0 + i" if per < C else "i"
        w(f"for (int i = {per - 1}; i >= 0; i--) {{ const bool in = {at} < j; " + " ".join(f"v[{x * C} + i] *= in ? W : 1.0f;" for x in range(max(1, KC // C)))
          + f" W *= in{live(at)} ? xv[i] : 1.0f; }}")
    w("#pragma unroll")
    w(f"for (int i = 0; i < {KC}; i++) {{ const int ci = i0 + i; gram[((d * {nr} + ci / {C}) * {C} + ci % {C}) * {GS} + j] = v[i]; }}")
    w.close()
    w.close()
    if dec_vec:
        w.close()
        w.open("else")
        NE = (N + 31) // 32
        w("#pragma unroll 1")
        w.open(f"for (int j = hw; j < {C}; j += {PT // 32})")
        w(f"float A[{nd}][{NE}], acc[{nd * nr}];")
        w("#pragma unroll 1")
        w.open("for (int i = j; i >= 0; i--)")
        w(" ".join(f"acc[{x}] = 0.0f;" for x in range(nd * nr)))
        w("#pragma unroll")
        w.open(f"for (int e = 0; e < {NE}; e++)")
        w("const int n = lane + 32 * e;")
        w.open(f"if (n < {N} && j < nv)")
        w.open("if (i == j)")
        w(f"const int tl = {pos('j')};")
        v = col.emit(s.alphas, "stage", "tl", "n", "x_")
        for d, nm in enumerate(s.alphas):
            w(f"A[{d}][e] = {v[nm]};")
        w.close()
        w.open("else")
        w(f"const int tl = {pos('i')};")
        v = col.emit(s.kappas + [s.decay], "stage", "tl", "n", "x_")
        for d in range(nd):
            for r, nm in enumerate(s.kappas):
                w(f"acc[{d * nr + r}] = fmaf(A[{d}][e], {v[nm]}, acc[{d * nr + r}]);")
        for d in range(nd):
            w(f"A[{d}][e] *= {v[s.decay]};")
        w.close()
        w.close()
        w.close()
        w("#pragma unroll")
        w.open(f"for (int x = 0; x < {nd * nr}; x++)")
        w("float z = acc[x];")
        w("#pragma unroll")
        w("for (int o = 16; o > 0; o >>= 1) z += frnn_shfl_xor(z, o);")
        w(f"if (lane == 0 && i < j) gram[(x * {C} + i) * {GS} + j] = z;")
        w.close()
        w.close()
        for k, zn in enumerate(s.diags):
            w.open("")
            w("float z = 0.0f;")
            w("#pragma unroll")
            w.open(f"for (int e = 0; e < {NE}; e++)")
            w("const int n = lane + 32 * e;")
            w.open(f"if (n < {N} && j < nv)")
            w(f"const int tl = {pos('j')};")
            v = col.emit([zn], "stage", "tl", "n", "x_")
            w(f"z += {v[zn]};")
            w.close()
            w.close()
            w("#pragma unroll")
            w("for (int o = 16; o > 0; o >>= 1) z += frnn_shfl_xor(z, o);")
            w(f"if (lane == 0) gram[{o_dg + k * C} + j] = z;")
            if s.dg_out:
                w(f"if (lane == 0 && j < nv) frnn_st_raw<float>({s.dg_out}, {dg_off(p, k, f't0 + {pos(chr(106))}')}, z);")
            w.close()
        w.close()
        w.close()
    w("frnn_tmem_fence_before_sync();")
    w(f"frnn_mbar_arrive(&bar[{B_GF} + buf]);" + (f" frnn_mbar_arrive(&bar[{B_SE} + c % {NS}]);" if dec_vec else ""))
    if kb.plain_items:
        hsync()
    if NS == 1:
        next_plain()
    w.close()     # chunk loop
    w.open("if (hl < 128)")
    w(f"const int c = {nchunk};")
    put_kappa()
    w.close()
    w("return;")
    w.close()     # preparing warps

    # ------------------------------------------------------------------ the warp that starts the copies of the inputs
    w.open(f"if (tid >= {128 + PT})")
    w(f"frnn_regs_release<{regs[2]}>();")
    w.close()
    w.open(f"if (tid >= {128 + PT + 32})")
    if kb.tma_items:
        w(f"if (tid >= {128 + PT + 64}) return;")
        w("#pragma unroll 1")
        w.open(f"for (int c = 0; c < {nchunk}; c++)")
        chunk_head_line = f"const int kc = {f'{nchunk - 1} - c' if s.reverse else 'c'}, t0 = kc * {C}, nv = min({C}, {p.T} - t0);"
        w(chunk_head_line)
        w(f"if (c >= {NS} && !frnn_mbar_wait(&bar[{B_SE} + c % {NS}], (c / {NS} - 1) & 1, err, {ERR})) return;")
        w(f"sc_issue(smem + {off_stage} + (c % {NS}) * {al(kb.stage_bytes)}, &bar[{B_RAW} + c % {NS}], t0, nv, lane, b, h, m0{tma_call});")
        w.close()
    w("return;")
    w.close()

    # ------------------------------------------------------------------ the warp that issues the products
    w.open(f"if (tid >= {128 + PT} && tid < {128 + PT + 32})")
    w("if (!frnn_elect()) return;")

    for nm, off, lbo in (("dA", off_al, lboA), ("dH", off_kh, lboH), ("dK", off_ka, lboK)):
        w(f"const u64 {nm} = frnn_mma_desc(smem + {off}, {lbo});")
    w(f"const u64 dKlo = frnn_mma_desc(smem + {off_ka + (0 if xk else ka_bytes)}, {lboK}), dA1 = frnn_mma_desc(smem + {off_al + al_bytes}, {lboA}); (void)dKlo;")

    # Gram in pieces, so that products the state threads wait for never queue behind all of it.  256 heads T512, 128 rows,
    # forward + backward, in one piece and in four, us: 128 columns Mamba-2 230 + 681 and 203 + 651, GLA 248 + 608 and 240 + 601,
    # Delta Rule 17 % and 12 % less in four (two measure like four); 64 columns Mamba-2 177 + 570 and 175 + 566, GLA 213 + 517
    # and 213 + 522, Gated Delta alike, Delta Rule 10 % and 3 % less in four.  80 to 112 columns divide into two pieces (72, 104
    # and 120 do not), which this rule does not use although they measured faster: Mamba-2 with 96 columns 197 + 608 and
    # 193 + 604, GLA 235 + 573 and 227 + 559, the Delta families' backward 12 to 22 %.
    pieces = 4 if N == 128 else 1

    def gram_piece(c: str, g: str):
        """Piece ``g`` of Gram of chunk ``c``."""
        kp = N // 8 // pieces
        w.open("")
        w(f"const u64 dga = frnn_mma_next((({c}) & 1) ? dA1 : dA, {lboA}, ({g}) * {kp}), dgh = frnn_mma_next(dH, {lboH}, ({g}) * {kp});")
        w("#pragma unroll")
        w.open(f"for (int k = 0; k < {kp}; k++)")
        w(f"frnn_mma_ss_d(tm + {colG}u, frnn_mma_next(dga, {lboA}, k), frnn_mma_next(dgh, {lboH}, k), FRNN_MMA_IDESC({RK}), ({g}) > 0 || k > 0);")
        if not xa:      # the rest of alpha, nA rows further on, onto the same rows of the result
            w(f"frnn_mma_ss_d(tm + {colG}u, frnn_mma_next(dga, {lboA}, k) + {nA // 8 * 128 // 16}ull, frnn_mma_next(dgh, {lboH}, k), FRNN_MMA_IDESC({RK}), true);")
        w.close()
        w(f"if (({g}) == {pieces - 1}) frnn_mma_commit(&bar[{B_MG}]);")
        w.close()
    w(f"if (!frnn_mbar_wait(&bar[{B_AF}], 0, err, {ERR}) || !frnn_mbar_wait(&bar[{B_HF}], 0, err, {ERR})) return;")
    w("frnn_tmem_fence_after_sync();")
    w("#pragma unroll 1")
    w.open(f"for (int g = 0; g < {pieces}; g++)")
    gram_piece("0", "g")
    w.close()
    w("#pragma unroll 1")
    w.open(f"for (int c = 0; c < {nchunk}; c++)")
    w("const u64 da = (c & 1) ? dA1 : dA;")
    for qi, (n0, n1) in enumerate(quarters):
        w(f"if (!frnn_mbar_wait(&bar[{B_SB + qi}], c & 1, err, {ERR})) return;")
        w("frnn_tmem_fence_after_sync();")
        k0, k1 = n0 // 8, min(n1, N) // 8
        for a, n_, first_ in ((colS, RA, "k > 0"), (colL, RA, "true")):
            w("#pragma unroll")
            w(f"for (int k = {k0}; k < {k1}; k++) frnn_mma_ts_d(tm + {colA}u, tm + {a}u + k * 8, frnn_mma_next(da, {lboA}, k), FRNN_MMA_IDESC({n_}), {first_});")
    w(f"frnn_mma_commit(&bar[{B_M1}]); frnn_mma_commit(&bar[{B_AE} + (c & 1)]);")
    # Gram of the next chunk as soon as its operands are there, but never in the way of products 2
    w(f"int g = c + 1 < {nchunk} ? 0 : {pieces}; bool ready = false; (void)ready;")
    w("const u64 t_wait = frnn_now_ns();")
    w.open("for (;;)")
    if not late_gram:
        w.open(f"if (g < {pieces})")
        w.open("if (!ready)")
        w(f"ready = frnn_mbar_try(&bar[{B_AF} + ((c + 1) & 1)], ((c + 1) >> 1) & 1) && frnn_mbar_try(&bar[{B_HF}], (c + 1) & 1);")
        w("if (ready) frnn_tmem_fence_after_sync();")
        w.close()
        w.open("if (ready)")
        gram_piece("c + 1", "g")
        w("g++;")
        w.close()
        w.close()
    w(f"if (frnn_mbar_try(&bar[{B_PB}], c & 1)) break;")
    w(f"if (frnn_now_ns() - t_wait > FRNN_WAIT_LIMIT_NS) {{ frnn_report(err, {ERR}); return; }}")
    w.close()
    w(f"if (!frnn_mbar_wait(&bar[{B_KF}], c & 1, err, {ERR})) return;")
    w("frnn_tmem_fence_after_sync();")
    passes = ([] if xk else [(colP + nK, "dKlo"), (colP, "dKlo")]) + [(colP + nK, "dK"), (colP, "dK")]
    for i, (a, dsc) in enumerate(passes):
        w("#pragma unroll")
        w(f"for (int k = 0; k < {nK // 8}; k++) frnn_mma_ts_d(tm + {colD}u, tm + {a}u + k * 8, frnn_mma_next({dsc}, {lboK}, k), FRNN_MMA_IDESC({Np}), {'k > 0' if i == 0 else 'true'});")
    w(f"frnn_mma_commit(&bar[{B_M2}]); frnn_mma_commit(&bar[{B_KE}]);")
    w.open(f"if (g < {pieces})")
    if late_gram:
        w(f"if (!frnn_mbar_wait(&bar[{B_M2}], c & 1, err, {ERR})) return;")
    w(f"if (!frnn_mbar_wait(&bar[{B_AF} + ((c + 1) & 1)], ((c + 1) >> 1) & 1, err, {ERR}) || !frnn_mbar_wait(&bar[{B_HF}], (c + 1) & 1, err, {ERR})) return;")
    w("frnn_tmem_fence_after_sync();")
    w("#pragma unroll 1")
    w.open(f"for (; g < {pieces}; g++)")
    gram_piece("c + 1", "g")
    w.close()
    w.close()
    w.close()
    w("return;")
    w.close()

    # ------------------------------------------------------------------ state warps
    w(f"frnn_regs_acquire<{regs[0]}>();")
    w("const u32 mine = tm + frnn_tmem_lane_base(warp);")
    w(f"const int m = m0 + tid; const bool row = tid < {MB};")
    nck = nchunk

    def tile_io(spec: TensorSpec, ptr: str, n0: str, cnt: int, load: bool):
        """``cnt`` columns from n0 of this thread's row, between x[] and a tensor of any layout."""
        base = _elem_off(spec, [(0, "b"), (1, "h"), (2, "m")])
        e = ELT[spec.dt]
        fast = spec.st(3) == 1 and spec.aligned16 and all((st * e) % 16 == 0 for st in spec.stride[:-1]) and N % 16 == 0
        w.open("if (row)")
        if fast:
            v = 16 // e if e < 4 else 4
            for q in range(0, cnt, v):
                w(f"{'frnn_ldv' if load else 'frnn_stv'}<{spec.dt},{v}>({ptr}, {base} + {n0} + {q}, &x[{q}]);")
        else:
            w("#pragma unroll")
            w.open(f"for (int k = 0; k < {cnt}; k++)")
            idx = f"{base} + (long)({n0} + k) * {spec.st(3)}L"
            w(f"if ({n0} + k < {N}) " + (f"x[k] = frnn_io<{spec.dt}>::ld({ptr}, {idx});" if load else f"frnn_io<{spec.dt}>::st({ptr}, {idx}, x[k]);"))
            w.close()
        w.close()

    def put_state(ck: Optional[str], guard: str = ""):
        """Columns n0.. of the state (x[]): into Tensor Memory with their rest, and into checkpoint ``ck``."""
        w(f"frnn_tmem_st<16>(mine + {colS}u + n0, x);")
        if ck and s.ckpt:
            w.open(f"if (row{guard})")
            w(f"float* cp = {s.ckpt} + ((((long)b * {p.H} + h) * {nck} + {ck}) * {N}L + n0) * {p.M}L + m;")
            w("#pragma unroll")
            w(f"for (int k = 0; k < 16; k++) " + ("" if N % 16 == 0 else f"if (n0 + k < {N}) ") + f"frnn_st_raw<float>(cp, k * {p.M}L, x[k]);")
            w.close()
        w("#pragma unroll")
        w("for (int k = 0; k < 16; k++) x[k] = frnn_tf32_rest(x[k]);")
        w(f"frnn_tmem_st<16>(mine + {colL}u + n0, x);")
    for qi, (n0, n1) in enumerate(quarters):
        w("#pragma unroll 1")
        w.open(f"for (int n0 = {n0}; n0 < {n1}; n0 += 16)")
        w("float x[16];")
        w("#pragma unroll")
        w("for (int k = 0; k < 16; k++) x[k] = 0.0f;")
        tile_io(s.init[0], s.init[1], "n0", 16, True)
        put_state(str(first))
        w.close()
        w(f"frnn_tmem_wait_st(); frnn_tmem_fence_before_sync(); frnn_mbar_arrive(&bar[{B_SB + qi}]);")
    w("#pragma unroll 1")
    w.open(f"for (int c = 0; c < {nchunk}; c++)")
    head("const ")
    w(f"if (!frnn_mbar_wait(&bar[{B_GF} + buf], (c >> 1) & 1, err, {ERR})) return;")

    def wait_m1():
        w(f"if (!frnn_mbar_wait(&bar[{B_M1}], c & 1, err, {ERR})) return;")
        w("frnn_tmem_fence_after_sync();")

    def ld_sums(ds: Sequence[int]):
        for d in ds:
            w(f"frnn_tmem_ld<{C}>(mine + {colA + d * C}u, &g[{d * C}]);")
            if not xa:
                w(f"frnn_tmem_ld<{C}>(mine + {colA + nA + d * C}u, &lo[{d * C}]);")

    def got_sums(ds: Sequence[int]):
        w("frnn_tmem_wait_ld();")
        for d in ds:
            w("#pragma unroll")
            v = (lambda k: f"g[{d * C} + {k}]") if xa else (lambda k: f"(g[{d * C} + {k}] + lo[{d * C} + {k}])")
            f = (lambda k: f"{v(k)} * dec[{o_dec} + {k}]") if dec_sc else v
            w(f"for (int k = 0; k < {C}; k += 2) g2[({d * C} + k) / 2] = frnn_pk_make({f('k')}, {f('k + 1')});")

    def steps_in_turn(ds: Sequence[int], nodes: Sequence[Node], outs: Sequence[Arg], finish: Callable, midway: Optional[Callable] = None,
                      regs: Dict[str, str] = {}):
        """Substitution into the row sums ``ds`` (a step's p enter the sums of the later steps) and, step by step, ``nodes``;
        ``finish(q, value)``.  What step q reads from shared memory is loaded a step ahead.  ``regs``: values that are in registers."""
        read = ({x for n in nodes for x in n.value_args()} | {o for o in outs if isinstance(o, str)}) - set(regs)
        names = {n.name for n in nodes}

        def val(a: Arg, q: int) -> str:
            if not isinstance(a, str):
                return lower.flit(a)
            if a in regs:
                return f"{regs[a]}[{q}]"
            if a.startswith("sig") and a in special:
                return f"g2[{(int(a[3:]) * C + q) // 2}].{'xy'[q % 2]}"
            return f"{'v' if a in names else 'i'}{q}_" + a.replace(".", "_")

        def load(q: int):
            for nm in row_in:
                if nm in read:
                    cls, o = kb.wk[nm]
                    tl = pos(str(q)) if whole or not s.reverse else f"max({pos(str(q))}, 0)"
                    w(f"const float {val(nm, q)} = mk[{tl} * {mk_row} + {o}" + ((f" + min(tid, {MB - 1})" if MB < 128 else " + tid") if cls == M1 else "") + "];")
            for a in sorted(read):
                if a.startswith("dg") and a in special:
                    w(f"const float {val(a, q)} = gram[{o_dg + int(a[2:]) * C + q}];")
            if q + 1 < C:
                for d in ds:
                    for r in range(nr):
                        j0 = (q + 1) // 4 * 4
                        w(f"float G{q}_{d}_{r}[{C - j0}];")
                        for j4 in range(j0, C, 4):
                            w(f"frnn_ldv<0,4>(gram, {((d * nr + r) * C + q) * GS + j4}, &G{q}_{d}_{r}[{j4 - j0}]);")
        w.open("")
        load(0)
        for q in range(C):
            if midway and q == C // 2:
                midway()
            if q + 1 < C:
                load(q + 1)
            for n in nodes:
                w(f"const float {val(n.name, q)} = {op_expr(n, [val(a, q) for a in n.args])};")
            finish(q, val)
            # the next step's sums first, alone where the pair's other one is this step's
            j0, jp = (q + 1) // 4 * 4, (q + 2) // 2 * 2
            for d in ds:
                for r in range(nr):
                    if jp > q + 1 < C:
                        w(f"g2[{(d * C + q) // 2}].y = fmaf(ph[{r}][{q}], G{q}_{d}_{r}[{q + 1 - j0}], g2[{(d * C + q) // 2}].y);")
            if ds and jp < C:
                w.open("")
                for r in range(nr):
                    w(f"const frnn_pk pp{r} = frnn_pk_make(ph[{r}][{q}], ph[{r}][{q}]);")
                for j in range(jp, C, 2):
                    for d in ds:
                        for r in range(nr):
                            w(f"g2[{(d * C + j) // 2}] = frnn_fma2(pp{r}, frnn_pk_make(G{q}_{d}_{r}[{j - j0}], G{q}_{d}_{r}[{j + 1 - j0}]), g2[{(d * C + j) // 2}]);")
                w.close()
        w.close()
    w.open("")
    w(f"float g[{nA}], ph[{nr}][{C}]; frnn_pk g2[{nA // 2}];")
    for x in range(len(kept)):
        w(f"float kept{x}[{C}];")
    if not xa:
        w(f"float lo[{nA}];")
    if not p_early:
        wait_m1()
        ld_sums(first_sums or other_sums)
        got_sums(first_sums or other_sums)

    def put_p(q: int, val):
        ok = ([] if whole else [f"{q} < nv"]) + ([] if MB == 128 else ["row"])
        for r, nm in enumerate(s.ps):
            w(f"ph[{r}][{q}] = " + (f"{' && '.join(ok)} ? {val(nm, q)} : 0.0f;" if ok else f"{val(nm, q)};"))
        for x, nm in enumerate(kept):
            w(f"kept{x}[{q}] = {val(nm, q)};")
    # p first, from the sums that it depends on alone; the sums that only outputs depend on, and the outputs, while products 2 run
    steps_in_turn(first_sums, [n for n in s.row if n.name in p_need], s.ps, put_p,
                  (lambda: ld_sums(other_sums)) if first_sums and other_sums else None)
    if first_sums and other_sums:
        got_sums(other_sums)           # before p is written over them
    for r in range(nr):
        for q in range(0, C, 16):
            w.open("")
            w("float x[16];")
            w("#pragma unroll")
            w(f"for (int k = 0; k < 16; k++) x[k] = ph[{r}][{q} + k]" + (f" * dec[{o_dec + C + q} + k];" if dec_sc else ";"))
            w(f"frnn_tmem_st<16>(mine + {colP + r * C + q}u, x);")
            w("#pragma unroll")
            w("for (int k = 0; k < 16; k++) x[k] = frnn_tf32_rest(x[k]);")
            w(f"frnn_tmem_st<16>(mine + {colP + nK + r * C + q}u, x);")
            w.close()
    w("frnn_tmem_wait_st(); frnn_tmem_fence_before_sync();")
    w(f"frnn_mbar_arrive(&bar[{B_PB}]);")
    if p_early:
        wait_m1()
        ld_sums(other_sums)
        got_sums(other_sums)

    def put_outs(q: int, val):
        """The outputs of eight steps at a time, so that a chunk cut short costs one branch per eight."""
        for k, o in enumerate(s.outs):
            w(f"const float o{q}_{k} = {val(o[0], q)};")
        if q % 8 < 7:
            return

        def store(x: int):
            w(f"{{ const long t = t0 + {pos(str(x))}; " + " ".join(f"frnn_io<{dt}>::st({ptr}, {at('t')} + (long)m * {sm}L, o{x}_{k});"
                                                                  for k, (nm, dt, ptr, at, sm) in enumerate(s.outs)) + " }")
        row = "" if MB == 128 else "row"
        w.open(f"if ({' && '.join(x for x in ('' if whole else f'{q} < nv', row) if x)})" if not whole or row else "")
        for x in range(q - 7, q + 1):
            store(x)
        w.close()
        if not whole:
            w.open("else" + (f" if ({row})" if row else ""))
            for x in range(q - 7, q):
                w(f"if ({x} < nv)")
                store(x)
            w.close()
    # (a step or row whose p is 0 instead of its value stores no outputs)
    regs = {**{nm: f"ph[{r}]" for r, nm in enumerate(s.ps) if nm in made}, **{nm: f"kept{x}" for x, nm in enumerate(kept)}}
    steps_in_turn(other_sums, [n for n in s.row if n.name in o_need], out_names, put_outs, regs=regs)
    w(f"frnn_mbar_arrive(&bar[{B_GE} + buf]);")
    w.close()
    w(f"if (!frnn_mbar_wait(&bar[{B_M2}], c & 1, err, {ERR})) return;")
    w("frnn_tmem_fence_after_sync();")
    if dec_sc:
        w(f"const float y = dec[{o_dec + 2 * C}];")
    w("float x[16], u[16];")
    w(f"frnn_tmem_ld<16>(mine + {colS}u, x); frnn_tmem_ld<16>(mine + {colD}u, u);")

    def update_block():
        """Columns n0.. of the state: decay and products 2, back into Tensor Memory, checkpoint."""
        if dec_vec:
            w("float y[16];")
            w("#pragma unroll")
            w(f"for (int k = 0; k < 16; k += 4) frnn_ldv<0,4>(dec, n0 + k, &y[k]);")
        w("frnn_tmem_wait_ld();")
        w("#pragma unroll")
        w("for (int k = 0; k < 16; k++) x[k] = " + ("fmaf(x[k], y[k], u[k]);" if dec_vec else "fmaf(x[k], y, u[k]);" if dec_sc else "x[k] + u[k];"))
        # the next columns come in while these are split and stored
        w("float z[16];")
        w(f"if (n0 + 16 < {Np}) {{ frnn_tmem_ld<16>(mine + {colS}u + n0 + 16, z); frnn_tmem_ld<16>(mine + {colD}u + n0 + 16, u); }}")
        put_state("(kc - 1)" if s.reverse else "(kc + 1)", f" && c + 1 < {nchunk}")
        w("#pragma unroll")
        w("for (int k = 0; k < 16; k++) x[k] = z[k];")

    # one loop of 16 columns, or one per quarter of the state unrolled twice: see ChunkPlan.compact
    quarter = f"frnn_tmem_wait_st(); frnn_tmem_fence_before_sync(); frnn_mbar_arrive(&bar[{B_SB} + qi]);"
    if compact:
        w("int qi = 0;")
        w(f"#pragma unroll {state_unroll or 1}")
        w.open(f"for (int n0 = 0; n0 < {Np}; n0 += 16)")
        update_block()
        w(f"if (n0 + 16 == {nblk} * (qi + 1) / {len(quarters)} * 16) {{ {quarter} qi++; }}")
        w.close()
    else:
        for qi, (n0, n1) in enumerate(quarters):
            w(f"#pragma unroll {state_unroll or 2}")
            w.open(f"for (int n0 = {n0}; n0 < {n1}; n0 += 16)")
            update_block()
            w.close()
            w(quarter.replace("qi]", f"{qi}]"))
    w.close()     # chunk loop
    w("frnn_tmem_wait_st();")
    w("#pragma unroll 1")
    w.open(f"for (int n0 = 0; n0 < {Np}; n0 += 16)")
    w("float x[16];")
    w(f"frnn_tmem_ld<16>(mine + {colS}u + n0, x);")
    w("frnn_tmem_wait_ld();")
    tile_io(s.final[0], s.final[1], "n0", 16, False)
    w.close()
    w.ind -= 1
    w("};")
    w("work();")
    w("// done, normally or after a timed-out wait: check in, and the allocating warp frees Tensor Memory")
    w("frnn_tmem_fence_before_sync();")
    w("frnn_warp_sync();")
    w("if (lane == 0) frnn_smem_add((int*)&bar[23], 1);")
    w.open("if (warp == 0)")
    w("const u64 t_exit = frnn_now_ns();")
    w(f"while (frnn_smem_add((int*)&bar[23], 0) < {(128 + PT) // 32 + 4} && frnn_now_ns() - t_exit < 2 * FRNN_WAIT_LIMIT_NS) {{}}")
    w("frnn_tmem_fence_after_sync();")
    w(f"frnn_tmem_dealloc(tm, {tm_cols}u);")
    w.close()
    w.close()
    # cycles the tensor cores are busy for one CTA: products 1 (the state and its rest), Gram, products 2, per chunk
    busy = nchunk * (2 * (N // 8) * product_cycles(RA) + (N // 8) * (1 if xa else 2) * product_cycles(RK, True)
                     + len(passes) * (nK // 8) * product_cycles(Np))
    return KernelSource(s.name, w.text().replace("@SMEM_BYTES@", str(smem_bytes)), (p.M // MB, p.H, p.B), 128 + PT + 128, smem_bytes,
                        kb.params, kb.param_decl, {"chunk": C, "tile": [1, N, MB], "packed": False, "tmem_cols": tm_cols, "nck": nck, "tensor_cycles": busy,
                                                   "tma_items": len(kb.tma_items), "plain_items": len(kb.plain_items)}, kb.tmaps)


#: timesteps per chunk when the chunk boundaries are also the checkpoints of the backward pass
CHUNK = 16


def ck_bytes(p: Problem, C: int) -> int:
    """Bytes of the fp32 states at the starts of chunks of C timesteps."""
    return p.B * p.H * ((p.T + C - 1) // C) * p.N * p.M * 4


def product_cycles(n: int, smem: bool = False) -> float:
    """Cycles of one tf32 product of 128 rows, 8 values of k and ``n`` columns (measured on a B200, see csrc/frnn_chunk.cuh),
    its first operand in Tensor Memory or in shared memory."""
    return max(10.0, n / 2, max(39.5, 32 + n / 4) if smem else 0.0)


def rows_per_cta(M: int) -> Optional[int]:
    """State rows of one CTA: all up to the 128 lanes of Tensor Memory, else a divisor of M."""
    for mb in range(min(M, 128), 0, -1):
        if M % mb == 0:
            return mb if mb >= 16 or mb == M else None
    return None


def forward_spec(p: Problem, nf: Normal, saved: Sequence[int], train: bool, C: int) -> ScanSpec:
    """The forward scan.  Parameters, in order: used inputs, initial state, outputs, final state and, for training,
    checkpoints [B, H, chunk, N, M] and the row sums ``saved`` [len, B, H, T, M]; error word."""
    yshape = (p.B, p.T, p.H, p.M)
    used = nf_inputs(nf)
    params = [(f"in{i}", "void", True, _spec_bytes(p.inputs[i])) for i in range(len(p.inputs)) if used[i]]
    params.append(("s0", "void", True, _spec_bytes(p.states[0])))
    params += [(f"out{j}", "void", False, p.B * p.T * p.H * p.M * ELT[p.out_dt[j]]) for j in range(len(nf.ys))]
    params.append(("sT", "void", False, _spec_bytes(p.res_states[0])))
    if train:
        params.append(("ck", "float", False, ck_bytes(p, C)))
        params.append(("aux", "float", False, len(saved) * p.B * p.H * p.T * p.M * 4))
    params.append(("err", "int", False, 4))
    outs = []
    for j, y in enumerate(nf.ys):
        ys = TensorSpec(yshape, _contig(yshape), p.out_dt[j])
        outs.append((y, p.out_dt[j], f"out{j}", lambda t, ys=ys: _elem_off(ys, [(0, "b"), (1, t), (2, "h")]), 1))
    if train:
        for k, d in enumerate(saved):
            outs.append((f"sig{d}", DT_F32, "aux", lambda t, k=k: aux_off(p, k, t), 1))
    items, consts = staged_inputs(p, nf, used)
    return ScanSpec("frnn_cfw", params, items, consts, nf.shape, nf.hoist, nf.row, nf.alphas, nf.kappas, nf.ps, nf.decay, nf.diags, nf.diag_at,
                    outs, (p.states[0], "s0"), (p.res_states[0], "sT"), None, "ck" if train else None, False)


def aux_off(p: Problem, k: int, t: str) -> str:
    """Element offset of time t in the k-th member of a [*, B, H, T, M] fp32 buffer."""
    return f"(((({k}L * {p.B} + b) * {p.H} + h) * {p.T}L + ({t})) * {p.M}L)"


def dg_off(p: Problem, k: int, t: str) -> str:
    """Element offset of dg<k> at time t in a [*, B, H, T] fp32 buffer."""
    return f"((({k}L * {p.B} + b) * {p.H} + h) * {p.T}L + ({t}))"


def aux_item(p: Problem, key: str, ptr: str, k: int) -> Staged:
    sh = (p.B, p.H, p.T, p.M)
    return Staged(key, M1, TensorSpec(sh, _contig(sh), DT_F32), ptr, {"b": 0, "h": 1, "t": 2, "v": 3}, k * p.B * p.H * p.T * p.M)


def nf_inputs(nf: Normal) -> List[bool]:
    read = {a for n in nf.hoist + nf.row for a in n.value_args()} | set(nf.ps) | set(nf.ys) | set(nf.alphas) | set(nf.kappas) | {nf.decay}
    return [i in read for i in nf.inputs]


def staged_inputs(p: Problem, nf: Normal, used: Sequence[bool]):
    items, consts = [], []
    for i, spec in enumerate(p.inputs):
        if not used[i]:
            continue
        cls = p.in_cls(i)
        if spec.shape[1] == 1 and p.T > 1:
            if cls != S11:
                raise lower.LoweringError("time-invariant vectors are not staged")
            consts.append((nf.inputs[i], spec, f"in{i}"))
        else:
            items.append(Staged(nf.inputs[i], cls, spec, f"in{i}", lower._in_dims(cls)))
    return items, consts


# ---------------------------------------------------------------------------
# backward: the scan of the state gradient, then the gradients of the vectors
# ---------------------------------------------------------------------------

@dataclass
class BackwardPlan:
    """How the backward pass of a normal form is divided.  ``vjp``: ``local_vjp``.  ``saved``: row sums the forward has to
    keep; ``kept``: row sums of the state gradient that its scan keeps for the vector gradients."""
    vjp: StepGraph
    saved: List[int]
    kept: List[int]
    kept_dg: bool                             # the scan of the state gradient also keeps the dg<k>
    dsig: List[Arg]
    row_grads: List[Tuple[int, Arg]]          # (input, value): gradients of row-vector inputs
    grads: List[Tuple[int, Arg]]              # the others
    log_decay: bool


def backward_plan(p: Problem, nf: Normal, v: StepGraph, log_decay: bool) -> Optional[BackwardPlan]:
    """None when the gradients do not divide into row functions, vectors and scalars as the two kernels need it."""
    nin, nd, nr = len(nf.inputs), len(nf.alphas), len(nf.kappas)
    nodes = v.node_map()
    late = [f"ga{d}" for d in range(nd)] + [f"gk{r}" for r in range(nr)] + ["gw"]
    dep_late = v.depends_on([x for x in late if x in v.inputs])
    msums = [n.name for n in v.nodes if n.op == "sum" and n.over_m]
    nsums = [n.name for n in v.nodes if n.op == "sum" and n.over_n]
    after_m = v.depends_on(msums)
    after_n = v.depends_on(nsums + (["gw"] if nf.decay and nf.shape[nf.decay] == S11 else []))
    for n in v.nodes:
        if n.shape == MN or (n.op == "sum" and n.over_m and n.over_n):
            return None
        if n.shape == M1 and (n.name in dep_late or n.name in after_m or n.name in after_n):
            return None
        if n.shape == N1 and n.name in after_n:
            return None
        if n.op == "sum" and n.over_m and v.shape.get(n.args[0]) != M1:
            return None
        if n.op == "sum" and n.over_n and v.shape.get(n.args[0]) != N1:
            return None
    dsig = list(v.outputs[nin:])
    row_grads, grads = [], []
    for i in range(nin):
        cls, o = p.in_cls(i), v.outputs[i]
        s = v.shape[o] if isinstance(o, str) else S11
        if cls == M1:
            if isinstance(o, str) and s != M1:
                return None
            row_grads.append((i, o))
        else:
            if isinstance(o, str) and s != cls:
                return None
            grads.append((i, o))
    if any(not isinstance(x, str) or v.shape[x] != M1 for x in dsig):
        return None

    def leaves(outs) -> set:
        need = set(o for o in outs if isinstance(o, str))
        for n in reversed(v.nodes):
            if n.name in need:
                need.update(n.value_args())
        return need
    k2 = leaves(dsig + [o for _, o in row_grads])
    k3 = leaves(dsig + [o for _, o in grads])
    rowdep = set()
    pn = {n.name: n for n in nf.row}
    todo = [x for x in nf.ps]
    while todo:
        a = todo.pop()
        if isinstance(a, str) and a not in rowdep:
            rowdep.add(a)
            if a in pn:
                todo += pn[a].value_args()
    if any(f"dg{k}" in rowdep for k in range(len(nf.diags))):
        return None
    saved = [d for d in range(nd) if f"sig{d}" in (k2 | k3 | rowdep)]
    kept = [r for r in range(nr) if f"gp{r}" in k3]
    return BackwardPlan(v, saved, kept, any(f"dg{k}" in k3 for k in range(len(nf.diags))), dsig, row_grads, grads, log_decay)


def backward_scan_spec(p: Problem, nf: Normal, bp: BackwardPlan, dspec: Sequence[TensorSpec], C: int) -> ScanSpec:
    """The scan of the state gradient E: E' = E * w + sum_d dsig_d (x) alpha_d with the row sums E . kappa_r, from the
    last timestep to the first.  Parameters, in order: used inputs, d outputs, d final state, forward row sums, d initial
    state, gradients of the row-vector inputs, checkpoints of E, kept row sums, error word."""
    v, nin = bp.vjp, len(nf.inputs)
    fs = {f"sig{d}": f"fsig{d}" for d in range(len(nf.alphas))}
    fs.update({f"gp{r}": f"sig{r}" for r in range(len(nf.kappas))})
    f = lambda a: fs.get(a, a) if isinstance(a, str) else a
    outs = [o for o in bp.dsig + [o for _, o in bp.row_grads] if isinstance(o, str)]
    g = v.pruned(outs)
    shape = dict(nf.shape)
    shape.update({f(k): s for k, s in v.shape.items()})
    for d in range(len(nf.alphas)):
        shape[f"fsig{d}"] = M1
    for r in range(len(nf.kappas)):
        shape[f"sig{r}"] = M1
    dyn = {f"sig{r}" for r in range(len(nf.kappas))} | {f"dg{k}" for k in range(len(nf.diags))}
    row, hoist = [], list(nf.hoist)
    for n in g.nodes:
        m = Node(f(n.name), n.op, [f(a) for a in n.args], n.shape)
        if any(a in dyn for a in m.value_args()):
            dyn.add(m.name)
            row.append(m)
        else:
            hoist.append(m)
    read = {a for n in hoist + row for a in n.value_args()} | {f(o) for o in outs} | set(nf.alphas) | set(nf.kappas) | {nf.decay}
    # hoisted nodes that nothing here reads (row functions of the forward) are pruned by the emitter
    keep, need = [], {a for n in row for a in n.value_args()} | {f(o) for o in outs} | set(nf.alphas) | set(nf.kappas) | set(nf.diags) | {nf.decay}
    for n in reversed(hoist):
        if n.name in need:
            need.update(n.value_args())
            keep.append(n)
    hoist = keep[::-1]
    used = [i in need for i in nf.inputs]
    items, consts = staged_inputs(p, nf, used)
    yshape = (p.B, p.T, p.H, p.M)
    params = [(f"in{i}", "void", True, _spec_bytes(p.inputs[i])) for i in range(nin) if used[i]]
    dys = [j for j in range(len(nf.ys)) if f"gy{j}" in need]
    for j in dys:
        params.append((f"dy{j}", "void", True, p.B * p.T * p.H * p.M * ELT[p.out_dt[j]]))
        items.append(Staged(f"gy{j}", M1, TensorSpec(yshape, _contig(yshape), p.out_dt[j]), f"dy{j}", {"b": 0, "t": 1, "h": 2, "v": 3}))
    sshape = (p.B, p.H, p.M, p.N)
    params.append(("dsT", "void", True, p.B * p.H * p.M * p.N * ELT[p.states[0].dt]))
    aux = [d for d in bp.saved if f"fsig{d}" in need]
    if aux:
        params.append(("aux", "float", True, len(bp.saved) * p.B * p.H * p.T * p.M * 4))
        for d in aux:
            items.append(aux_item(p, f"fsig{d}", "aux", bp.saved.index(d)))
    params.append(("ds0", "void", False, _spec_bytes(p.res_states[0])))
    louts = []
    for i, o in bp.row_grads:
        params.append((f"dx{i}", "void", False, _spec_bytes(dspec[i])))
        if not isinstance(o, str):
            raise lower.LoweringError("a constant gradient")
        louts.append((f(o), dspec[i].dt, f"dx{i}", lambda t, sp=dspec[i]: _elem_off(sp, [(0, "b"), (1, t), (2, "h")]), dspec[i].st(3)))
    params.append(("eck", "float", False, ck_bytes(p, C)))
    if bp.kept:
        params.append(("tau", "float", False, len(bp.kept) * p.B * p.H * p.T * p.M * 4))
        for k, r in enumerate(bp.kept):
            louts.append((f"sig{r}", DT_F32, "tau", lambda t, k=k: aux_off(p, k, t), 1))
    if bp.kept_dg:
        params.append(("dgk", "float", False, len(nf.diags) * p.B * p.H * p.T * 4))
    params.append(("err", "int", False, 4))
    return ScanSpec("frnn_cbw", params, items, consts, shape, hoist, row, nf.kappas, nf.alphas, [f(x) for x in bp.dsig], nf.decay,
                    nf.diags, [(r, d) for d, r in nf.diag_at], louts, (TensorSpec(sshape, _contig(sshape), p.states[0].dt), "dsT"),
                    (p.res_states[0], "ds0"), "dgk" if bp.kept_dg else None, "eck", True)


def emit_vector_grads(p: Problem, nf: Normal, bp: BackwardPlan, dspec: Sequence[TensorSpec], atomic: Sequence[bool], C: int) -> KernelSource:
    """Gradients of the column vectors and scalars, one CTA per chunk of ``C`` timesteps: with the state S_0 at the
    chunk's start, the state gradient E_C at its end, X = dsig and Z = p (vectors over the rows, per timestep),

      d alpha_d,j = W_j-1 * (S_0^T X_d,j) + sum_{i<j,r} L_dj,ri kappa_r,i W_j-1/W_i          L = X Z^T (over the rows)
      d kappa_r,i = W_C/W_i * (E_C^T Z_r,i) + sum_{j>i,d} L_dj,ri alpha_d,j W_j-1/W_i
      w_j d w_j   = R_j - sum_r kappa_r,j * d kappa_r,j,   R_j-1 = w_j d w_j + sum_d alpha_d,j * d alpha_d,j

    (R_j: sums over the rows of E_j * S_j, at the chunk's end from S_0 and E_C), then the chain rule to the inputs
    (``local_vjp``).  All products run on the tensor cores.  Where a decay of the chunk is too small to divide by, the
    chunk takes a slower path of plain loops with running products instead.

    S_0, E_C and the row vectors stream through in slices of 16 rows, which are what the products sum over: X and Z of a slice are
    made beside it (all of X and Z at once took 100 KB, one CTA per SM, and the load phases of all SMs coincided: Delta Rule
    128x128 B8 T1024 H32 640 us, in slices 493).  The bytes of a chunk, 200 KB for the Delta Rule, take half of its time
    at the copy rate; the stores of the slices and the products' reads of them keep shared memory busy 62 % of it (ncu).
    Parameters, in order: inputs, d outputs, forward row sums, kept row sums, checkpoints of S, of E,
    gradients, error word.
    """
    v = bp.vjp
    M, N, B, T, H = p.M, p.N, p.B, p.T, p.H
    nd, nr = len(nf.alphas), len(nf.kappas)
    nA, nK = nd * C, nr * C
    dec_vec = bool(nf.decay) and nf.shape[nf.decay] == N1
    dec_sc = bool(nf.decay) and not dec_vec
    w = W()
    nin = len(nf.inputs)
    shape = dict(nf.shape)
    shape.update(v.shape)
    # ---- stages
    msums = [n for n in v.nodes if n.op == "sum" and n.over_m]
    nsums = [n for n in v.nodes if n.op == "sum" and n.over_n]
    gouts = [o for _, o in bp.grads if isinstance(o, str)]
    need = set(gouts) | set(x for x in bp.dsig)
    live_nodes = []
    for n in reversed(v.nodes):
        if n.name in need:
            need.update(n.value_args())
            live_nodes.append(n)
    live_nodes.reverse()
    msums = [n for n in msums if n.name in need]
    nsums = [n for n in nsums if n.name in need]
    g = StepGraph("v", v.inputs, live_nodes, gouts, dict(v.shape))
    after_m = g.depends_on([n.name for n in msums])
    after_n = g.depends_on([n.name for n in nsums] + (["gw"] if dec_sc else []))
    # the forward's own nodes, and those of p
    fnodes = {n.name: n for n in nf.hoist + nf.row}
    # scalars of the first stage: forward ones and those of the vjp that depend on inputs and dg only
    first_s = [n for n in list(nf.hoist) + live_nodes if n.shape == S11 and n.op != "sum" and n.name not in after_m and n.name not in after_n]
    second_s = [n for n in live_nodes if n.shape == S11 and n.op != "sum" and n.name in after_m and n.name not in after_n]
    third_s = [n for n in live_nodes if n.shape == S11 and n.op != "sum" and n.name in after_n]
    s_inputs = [i for i in range(nin) if p.in_cls(i) == S11]
    use_dg = [k for k in range(len(nf.diags)) if f"dg{k}" in need]
    # ---- parameters
    params, decl, nbytes = [], [], {}

    def param(nm, ct, const, nb):
        params.append(nm)
        decl.append(f"{'const ' if const else ''}{ct}*{' __restrict__' if const else ''} {nm}")
        nbytes[nm] = nb
    for i in range(nin):
        param(f"in{i}", "void", True, _spec_bytes(p.inputs[i]))
    for j in range(len(nf.ys)):
        param(f"dy{j}", "void", True, B * T * H * M * ELT[p.out_dt[j]])
    if bp.saved:
        param("aux", "float", True, len(bp.saved) * B * H * T * M * 4)
    if bp.kept:
        param("tau", "float", True, len(bp.kept) * B * H * T * M * 4)
    if bp.kept_dg:
        param("dgk", "float", True, len(nf.diags) * B * H * T * 4)
    nchunk = (T + C - 1) // C
    param("ck", "float", True, ck_bytes(p, C))
    param("eck", "float", True, ck_bytes(p, C))
    for i, _ in bp.grads:
        param(f"dx{i}", "void", False, _spec_bytes(dspec[i]))
    param("err", "int", False, 4)
    # ---- shared memory
    al = lambda x: (x + 127) // 128 * 128
    sc_slots: Dict[str, int] = {}           # scalar arrays [C]

    def slot(nm: str) -> str:
        if nm not in sc_slots:
            sc_slots[nm] = len(sc_slots)
        return f"sc[{sc_slots[nm] * C}"
    for i in s_inputs:
        slot(nf.inputs[i])
    for n in first_s + second_s + third_s:
        slot(n.name)
    for k in use_dg:
        slot(f"dg{k}")
    for n in msums:
        slot(n.name)
    want_gw = bool(nf.decay) and "gw" in need
    n_nsum = len(nsums) + (2 if dec_sc and want_gw else 0)
    for x in ("Wp", "Ws", "gw"):
        slot(x)
    npart = n_nsum + 1
    # which operands are plain 16-bit inputs, exact in tf32: they have no second term
    dt16 = (lower.DT_BF16, lower.DT_F16)
    leaf_dt = {nf.inputs[i]: p.inputs[i].dt for i in range(nin)}
    leaf_dt.update({f"gy{j}": p.out_dt[j] for j in range(len(nf.ys))})
    is16 = lambda a: isinstance(a, str) and leaf_dt.get(a) in dt16
    restX = [d for d in range(nd) if not is16(bp.dsig[d])]
    restZ = [r for r in range(nr) if not is16(nf.ps[r])]
    xa, xk = not dec_vec and all(map(is16, nf.alphas)), not dec_vec and all(map(is16, nf.kappas))
    RX, RZ = nA + C * len(restX), nK + C * len(restZ)        # rows of X and Z: the vectors, then the rests of the inexact ones
    slow_path = bool(nf.decay) and (dec_vec or want_gw)
    few = dec_vec and want_gw and not bp.log_decay
    # which gradients of single decays are formed by running products; one expression for those who mark them and those who read the
    # results, so that what is read has been written (a NaN is none of them: its gradient is the quotient, a NaN)
    by_products = lambda x: f"(fabsf({x}) <= 0.0009765625f)"
    # padding: the eight threads of a store's phase write to different banks
    lboX, lboZ = RX * 16 + 32, RZ * 16 + 32
    lboT, lbo1, lbo2 = 128 * 16, 2 * nA * 16, 2 * nK * 16 + 16
    LS = nK + 1
    kT_b, aT_b = nK // 4 * lboT, nA // 4 * lboT

    NT = 256                                 # 128 rows or columns times two halves of the chunk's timesteps
    HC = C // 2                              # timesteps of one thread

    class Layout:
        """Shared memory with slices of ``MS`` rows in ``NB`` buffers."""

        def __init__(self, MS: int, NB: int):
            self.MS, self.NB = MS, NB
            self.sc = 256
            self.part = self.sc + al(len(sc_slots) * C * 4)
            self.z0 = self.part + al(npart * 4 * C * 4)
            self.xr = self.z0 + al(128 * 4)             # what the threads of a column exchange
            self.few = self.xr + al(2 * NT * 4)         # per column and half, the steps whose decays are too small to divide by
            # a buffer holds a slice of S_0, E_C and their rests, and of X (as first operand 128 rows of it are read) and Z
            self.sl = self.few + (al(NT * 2) if few else 0)
            self.lboS = 128 * 16 + 128 // (MS // 4)
            self.sl_bytes = al(MS // 4 * self.lboS)
            self.X = 4 * self.sl_bytes
            self.Z = self.X + al((MS // 4 - 1) * lboX + max(2048, RX * 16))
            self.buf = self.Z + al(MS // 4 * lboZ)
            end1 = self.sl + NB * self.buf
            # second phase, over the same memory
            self.kT = self.sl
            self.aT = self.kT + (1 if xk else 2) * kT_b
            self.L1 = self.aT + (1 if xa else 2) * aT_b
            self.L2 = self.L1 + nK // 4 * lbo1
            self.Lr = self.L2 + nA // 4 * lbo2
            # the slow path's results: (nA + nK) x 128 floats over the operands it does without, gradients of the decays beside them
            self.slow = self.kT
            if slow_path and dec_vec:
                self.Lr = max(self.Lr, self.slow + (nA + nK) * 512)
            self.gw = al(self.Lr + nA * LS * 4)
            self.bytes = al(max(end1, self.gw + (C * 512 if slow_path and want_gw else 0)))
            self.ctas = 2 if self.bytes <= SMEM_BYTES // 2 - 1024 else 1
    # two CTAs of 256 threads share an SM and hide each other's latencies, with two buffers of slices where they fit (B8 T1024 H32,
    # us, two buffers, one, and one CTA of 512 threads with two: Delta Rule 128x128 493, 519, 508; RWKV-7 988, 1019, 1322; Mamba-2
    # 64x128 441, 441, 457)
    for NB in (2, 1):
        lay = Layout(16 if M % 16 == 0 else 8, NB)
        if lay.ctas == 2:
            break
    else:
        # one CTA per SM, which then has two buffers as well (steps with a decay per column and several sums; 64x64, 64 heads, T1024, us, one
        # buffer and two: two sums 197 and 190, four 344 and 331, four and two terms 383 and 368)
        two = Layout(lay.MS, 2)
        lay = two if two.bytes <= SMEM_BYTES else lay
    MS, NB, ctas = lay.MS, lay.NB, lay.ctas
    DP = 2                                   # slices that are loaded ahead
    nsl = M // MS
    lboS, sl_bytes, smem_bytes = lay.lboS, lay.sl_bytes, lay.bytes
    off_sc, off_part, off_z0, off_xr, off_sl = lay.sc, lay.part, lay.z0, lay.xr, lay.sl
    off_kT, off_aT, off_L1, off_L2, off_Lr, off_slow, off_gw = lay.kT, lay.aT, lay.L1, lay.L2, lay.Lr, lay.slow, lay.gw
    cD1, cD2 = 0, RX
    cL = cD2 + RZ
    tm_cols = _tmem_pow2(cL + RZ)
    if 2 * nA + 4 * nK > 256:
        # with a rest for every vector, whether it has one or not: further rank-1 terms would fit, but a backward that fits only
        # so makes the outputs of training chunked as well, with two tf32 terms for fp32 (one row sum and four exact terms
        # with 16x32, outputs against fp64: 1.4e-7 recurrent, 3.2e-7 chunked)
        raise lower.LoweringError("the vector gradients of a chunk do not fit half of Tensor Memory")
    if RX > 128:              # L has them as rows: lanes of Tensor Memory
        raise lower.LoweringError("X and its rests have more rows than a product")
    at_rest = lambda inexact, x, n: n + C * inexact.index(x)     # row or column where the rest of vector x begins
    ERR = lower.ERR_STAGE_TIMEOUT
    full_n = N == 128
    # loads are never predicated (the compiler would wait for each in turn): past the ends they repeat the last timestep,
    # row or column, and a select drops what they bring
    whole = T % C == 0
    tq = lambda q: f"t0 + {q}" if whole else f"t0 + min({q}, nv - 1)"
    live_n = " && ".join(([] if whole else ["q < nv"]) + ([] if full_n else ["ncol"])) or "true"
    sel = lambda live, e, z="0.0f": e if live == "true" else f"(live ? {e} : {z})"

    w(lower._header(chunk_prelude()))
    w(f"// vector gradients: B={B} T={T} H={H} M={M} N={N}; {C} steps per chunk, {nd} row sums, {nr} rank-1 terms")
    w(f'extern "C" __global__ void __launch_bounds__({NT}, {ctas})')
    w.open(f"frnn_cvg({', '.join(decl)})")
    w("FRNN_DYN_SMEM(smem);")
    w("const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;")
    w(f"const int kc = blockIdx.x, h = blockIdx.y, b = blockIdx.z, t0 = kc * {C}, nv = min({C}, {T} - t0); (void)nv;")
    w("#ifdef FRNN_BOUNDS")
    w.open("if (tid == 0)")
    w("frnn_bounds_begin(err, smem, @SMEM_BYTES@L);")
    for nm, nb in nbytes.items():
        w(f"frnn_bounds_add({nm}, {nb}L);")
    w.close()
    w("frnn_block_sync();")
    w("#endif")
    w("u64* bar = (u64*)smem;")
    w(f"float* sc = (float*)(smem + {off_sc});")
    w(f"float* part = (float*)(smem + {off_part});")
    w(f"float* z0 = (float*)(smem + {off_z0}); (void)z0;")
    w(f"float* xr = (float*)(smem + {off_xr}); (void)xr;")

    def in_off(i: int, t: str, extra: str = "") -> str:
        sp = p.inputs[i]
        o = _elem_off(sp, [(0, "b"), (1, t), (2, "h")])
        return o + (f" + (long)({extra}) * {sp.st(4 if p.in_cls(i) == N1 else 3)}L" if extra else "")
    by_in = {nm: i for i, nm in enumerate(nf.inputs)}

    def leaf(a: str, t: str, idx: str) -> Optional[str]:
        """Load expression of a per-timestep vector that comes from global memory."""
        if a in by_in:
            i = by_in[a]
            return f"frnn_io<{p.inputs[i].dt}>::ld(in{i}, {in_off(i, t, idx)})"
        if a.startswith("gy"):
            j = int(a[2:])
            return f"frnn_io<{p.out_dt[j]}>::ld(dy{j}, ((((long)b * {T} + {t}) * {H} + h) * {M}L + {idx}))"
        if a.startswith("sig") or a.startswith("gp"):
            k, ptr = (bp.saved.index(int(a[3:])), "aux") if a.startswith("sig") else (bp.kept.index(int(a[2:])), "tau")
            return f"frnn_ld_raw<float>({ptr}, (((({k}L * {B} + b) * {H} + h) * {T}L + {t}) * {M}L + {idx}))"
        return None
    all_nodes = {n.name: n for n in live_nodes}
    all_nodes.update(fnodes)

    def leaves_of(names: Sequence[Arg], cls: Shape, given: Sequence[str] = ()) -> List[str]:
        out: List[str] = []

        def visit(a):
            if not isinstance(a, str) or a in given or shape[a] != cls:
                return
            if a in all_nodes:
                for x in all_nodes[a].args:
                    visit(x)
            elif a not in out:
                out.append(a)
        for a in names:
            visit(a)
        return out

    class Stage:
        """Values of one timestep: scalars from shared memory, vectors from the registers ``regs`` names."""

        def __init__(self, pre: str, q: str, cls: Shape, regs: Dict[str, str]):
            self.pre, self.q, self.cls, self.done = pre, q, cls, dict(regs)

        def get(self, a) -> str:
            if not isinstance(a, str):
                return lower.flit(a)
            if a in self.done:
                return self.done[a]
            if shape[a] == S11:
                if a not in sc_slots:
                    raise lower.LoweringError(f"scalar {a} is not available at this stage")
                self.done[a] = f"{slot(a)} + {self.q}]"
                return self.done[a]
            if shape[a] != self.cls or a not in all_nodes:
                raise lower.LoweringError(f"{a} is not available at this stage")
            nm = self.pre + a.replace(".", "_")
            ops = [self.get(x) for x in all_nodes[a].args]
            w(f"const float {nm} = {op_expr(all_nodes[a], ops)};")
            self.done[a] = nm
            return nm

    def reduce_lanes(arr: str, cnt: int, dst: str):
        """Sum ``arr[cnt]`` over the lanes of a warp, all values at once; ``dst`` receives value @."""
        c, o, idx = cnt, 16, []
        while c > 1 and o >= 1:
            hf = c // 2
            w("#pragma unroll")
            w(f"for (int k = 0; k < {hf}; k++) {{ const bool up = lane & {o}; const float snd = up ? {arr}[k] : {arr}[k + {hf}], own = up ? {arr}[k + {hf}] : {arr}[k]; "
              f"{arr}[k] = own + frnn_shfl_xor(snd, {o}); }}")
            idx.append((o, hf))
            c, o = hf, o // 2
        mask = 0
        while o >= 1:
            w(f"{arr}[0] += frnn_shfl_xor({arr}[0], {o});")
            mask |= o
            o //= 2
        e = " + ".join(f"((lane & {o_}) ? {hf} : 0)" for o_, hf in idx) or "0"
        w(f"if ((lane & {mask}) == 0) {dst.replace('@', '(' + e + ')')} = {arr}[0];")

    def scalar_nodes(nodes, q="q"):
        for n in nodes:
            w(f"{slot(n.name)} + {q}] = {op_expr(n, [lower.flit(a) if not isinstance(a, str) else f'{slot(a)} + {q}]' for a in n.args])};")

    # ---- what can be loaded at once: the rows' vectors, the first slices of S_0 and E_C
    w(f"const int x128 = tid & 127, hf = tid >> 7, q0 = hf * {HC};")
    w(f"const int nc = {'x128' if full_n else f'min(x128, {N - 1})'};")
    w(f"const bool ncol = x128 < {N}; (void)ncol; (void)nc;")
    mleaves = leaves_of(list(bp.dsig) + list(nf.ps) + [n.args[0] for n in msums], M1)
    reg = lambda a: "r_" + a.replace(".", "_")
    QG = NT // MS                            # in a slice a thread has row mi and every QG-th timestep
    nq = max(1, C // QG)
    w(f"const int mi = tid % {MS}, qg = tid / {MS};")
    for a in mleaves:
        w(f"float {reg(a)}[{DP}][{nq}];")
    at_q = lambda i: f"qg + {QG * i}" if QG <= C else f"min(qg, {C - 1})"
    q4 = MS // 4
    per = 128 // (NT // q4)        # columns per thread and slice
    w(f"const int sm4 = tid % {q4}, sn = tid / {q4};")
    w(f"const float* ckp = ck + (((long)b * {H} + h) * {nchunk} + kc) * {N}L * {M}L; const float* ekp = eck + (((long)b * {H} + h) * {nchunk} + kc) * {N}L * {M}L;")
    w(f"float zz[{per}], sv[{DP}][{per}][4], ev[{DP}][{per}][4];")
    w("#pragma unroll")
    w(f"for (int i = 0; i < {per}; i++) zz[i] = 0.0f;")

    def load_slice(sx, u):
        w("#pragma unroll")
        w.open(f"for (int i = 0; i < {per}; i++)")
        w(f"const int n = {'sn' if full_n else 'min(sn'} + i * {NT // q4}{'' if full_n else f', {N - 1})'};")
        w(f"frnn_ldv<0,4>(ckp, n * {M}L + ({sx}) * {MS} + sm4 * 4, sv[{u}][i]);")
        w(f"frnn_ldv<0,4>(ekp, n * {M}L + ({sx}) * {MS} + sm4 * 4, ev[{u}][i]);")
        w.close()
        for i in range(nq):
            w(f"{{ const int t = {tq(f'({at_q(i)})')}, m = ({sx}) * {MS} + mi; " + " ".join(f"{reg(a)}[{u}][{i}] = {leaf(a, 't', 'm')};" for a in mleaves) + " }")
    for u in range(min(DP, nsl)):
        load_slice(str(u), str(u))
    w("if (tid == 0) { frnn_mbar_init(&bar[0], 1); frnn_mbar_init(&bar[1], 1); frnn_mbar_init(&bar[2], 1); frnn_mbar_init(&bar[5], 1); frnn_mbar_init_fence(); }")
    if few:
        w(f"unsigned short* fewm = (unsigned short*)(smem + {lay.few});")
    w.open("if (warp == 0)")
    w(f"frnn_tmem_alloc((u32*)&bar[3], {tm_cols}u);")
    w("frnn_tmem_fence_before_sync();")
    w.close()
    # ---- scalars of the inputs, decay products
    w.open(f"if (tid >= 32 && tid < {32 + C})")
    w(f"const int q = tid - 32, t = {'t0 + q' if whole else 't0 + min(q, nv - 1)'}; (void)t;")
    w("if (q == 0) bar[4] = 0;      // two flags, set by these threads after they have met, or by all after the block barrier")
    for i in s_inputs:
        w(f"{slot(nf.inputs[i])} + q] = frnn_io<{p.inputs[i].dt}>::ld(in{i}, {in_off(i, 't')});")
    for k in use_dg:
        w(f"{slot(f'dg{k}')} + q] = frnn_ld_raw<float>(dgk, {dg_off(p, k, 't')});")
    scalar_nodes(first_s)
    if dec_sc:
        w("frnn_warp_sync();" if C == 32 else "frnn_half_warp_sync();")
        w("float a = 1.0f, c = 1.0f;")
        w("#pragma unroll")
        w(f"for (int l = 0; l < {C}; l++) {{ const float x = {slot(nf.decay)} + l]; if (l < q) a *= x; if (l > q && l < nv) c *= x; }}")
        w(f"{slot('Wp')} + q] = a; {slot('Ws')} + q] = c;")
        if want_gw:
            # the gradient of a decay per head divides by it only where the step reads it as it is (an exponential's does not)
            cond = f"!(fabsf({slot(nf.decay)} + q]) > 0.0009765625f)"
            if not bp.log_decay:
                w(f"if (q < nv && {cond}) *(volatile int*)&bar[4] = 1;")
    w.close()
    w("frnn_block_sync();")
    w("frnn_tmem_fence_after_sync();")
    w("const u32 tm = *(volatile u32*)&bar[3];")
    for x in range(len(msums)):
        w(f"float rs{x}[{nq}];")
        w("#pragma unroll")
        w(f"for (int i = 0; i < {nq}; i++) rs{x}[i] = 0.0f;")
    live_m = " && ".join(([] if whole else ["q < nv"]) + ([] if QG <= C else [f"qg < {C}"])) or "true"

    def put_rows(u: int, buf: int):
        """This thread's values of X and Z for a slice of rows, into buffer ``buf``, and their parts of the sums over the rows."""
        for i in range(nq):
            w.open("")
            w(f"const int q = {at_q(i)}; const bool live = {live_m}; (void)live;")
            st = Stage("x_", "q", M1, {a: f"{reg(a)}[{u}][{i}]" for a in mleaves})
            vals = [(d, st.get(x), "X") for d, x in enumerate(bp.dsig)] + [(r, st.get(x), "Z") for r, x in enumerate(nf.ps)]
            for x, n in enumerate(msums):
                w(f"rs{x}[{i}] += {sel(live_m, st.get(n.args[0]))};")
            w.open("" if QG <= C else f"if (qg < {C})")
            for v_, val, which in vals:
                lbo, off, inexact, n2 = (lboX, lay.X, restX, nA) if which == "X" else (lboZ, lay.Z, restZ, nK)
                put = lambda row0, x: f"{{ const int row = {row0} + q; *(float*)(dst + (row >> 3) * 128 + (row & 7) * 16) = {x}; }}"
                w(f"{{ const float a = {sel(live_m, val)}; unsigned char* dst = smem + {buf + off} + (mi >> 2) * {lbo} + (mi & 3) * 4; {put(v_ * C, 'a')}"
                  + (" " + put(at_rest(inexact, v_, n2), "frnn_tf32_rest(a)") if v_ in inexact else "") + " }")
            w.close()
            w.close()
    # ---- S_0, E_C, X and Z, a slice of rows at a time, loaded two slices ahead
    colv = nf.alphas + nf.kappas + ([nf.decay] if dec_vec else [])
    ngiven = [f"ga{d}" for d in range(nd)] + [f"gk{r}" for r in range(nr)] + ["gw"]
    n_outs = [o for i, o in bp.grads if p.in_cls(i) == N1]
    nleaves = leaves_of(list(colv) + [n.args[0] for n in nsums] + n_outs, N1, ngiven)
    for a in nleaves:
        w(f"float {reg(a)}[{HC}];")
    # where a wait ran out in some threads all leave the loop together, by the vote at its barrier: every thread meets every
    # block barrier (a flag that each thread carries through the loop instead cost 3 to 4 % of the backward pass for RWKV-7,
    # Mamba-2 and the Gated Delta Rule at B8 T1024; the vote 0.1 to 0.8 %)
    w("#pragma unroll 1")
    w.open(f"for (int s2 = 0; s2 < {nsl}; s2 += {DP})")
    for u in range(DP):
        bb = 5 if u % NB else 1
        w.open(f"if (s2 + {u} < {nsl})")
        w(f"const int s = s2 + {u};")
        w(f"const bool arrived = s < {NB} || frnn_mbar_wait(&bar[{bb}], (s / {NB} - 1) & 1, err, {ERR});     // the products that read this buffer are complete")
        w("#pragma unroll")
        w.open(f"for (int i = 0; i < {per}; i++)")
        w(f"const int n = sn + i * {NT // q4};")
        off_b = off_sl + (u % NB) * lay.buf
        w(f"unsigned char* dst = smem + {off_b} + sm4 * {lboS} + (n >> 3) * 128 + (n & 7) * 16;")
        w("float r[4];")
        w("#pragma unroll")
        w(f"for (int k = 0; k < 4; k++) {{ r[k] = frnn_tf32_rest(sv[{u}][i][k]); zz[i] = fmaf(sv[{u}][i][k], ev[{u}][i][k], zz[i]); }}")
        w(f"frnn_stv<0,4>(dst, 0, sv[{u}][i]); frnn_stv<0,4>(dst + {sl_bytes}, 0, r);")
        w("#pragma unroll")
        w(f"for (int k = 0; k < 4; k++) r[k] = frnn_tf32_rest(ev[{u}][i][k]);")
        w(f"frnn_stv<0,4>(dst + {2 * sl_bytes}, 0, ev[{u}][i]); frnn_stv<0,4>(dst + {3 * sl_bytes}, 0, r);")
        w.close()
        put_rows(u, off_b)
        w(f"if (s + {DP} < {nsl}) {{")
        w.ind += 1
        load_slice(f"s + {DP}", str(u))
        w.ind -= 1
        w("}")
        w("frnn_async_proxy_fence();")
        w("if (!frnn_block_and(arrived)) break;")
        w.open("if (warp == 0 && frnn_elect())")
        first = lambda k: "s > 0" if k == 0 else "true"
        for k in range(MS // 8):
            w(f"frnn_mma_ss_d(tm + {cL}u, frnn_mma_desc(smem + {off_b + lay.X + k * 2 * lboX}, {lboX}), frnn_mma_desc(smem + {off_b + lay.Z + k * 2 * lboZ}, {lboZ}), FRNN_MMA_IDESC({RZ}), {first(k)});")
        w(f"if (s == {nsl - 1}) frnn_mma_commit(&bar[0]);")
        for k in range(MS // 8):
            for which, (col_, at, lbo, n2) in enumerate(((cD1, lay.X, lboX, RX), (cD2, lay.Z, lboZ, RZ))):
                sb = off_b + 2 * which * sl_bytes + k * 2 * lboS
                for part_ in (sb, sb + sl_bytes):
                    w(f"frnn_mma_ss_d(tm + {col_}u, frnn_mma_desc(smem + {part_}, {lboS}), frnn_mma_desc(smem + {off_b + at + k * 2 * lbo}, {lbo}), FRNN_MMA_IDESC({n2}), {first(k) if part_ == sb else 'true'});")
        w(f"frnn_mma_commit(&bar[{bb}]);")
        w.close()
        w.close()
    w.close()
    # the columns' vectors come in while the last products run
    w("#pragma unroll")
    w.open(f"for (int k = 0; k < {HC}; k++)")
    w(f"const int t = {tq('q0 + k')};")
    for a in nleaves:
        w(f"{reg(a)}[k] = {leaf(a, 't', 'nc')};")
    w.close()
    if nf.decay:
        w("#pragma unroll")
        w.open(f"for (int i = 0; i < {per}; i++)")
        w("#pragma unroll")
        w(f"for (int o = {q4 // 2}; o > 0; o >>= 1) zz[i] += frnn_shfl_xor(zz[i], o);")
        w(f"if (sm4 == 0) z0[sn + i * {NT // q4}] = zz[i];")
        w.close()
    for x, n in enumerate(msums):
        w("#pragma unroll")
        w.open(f"for (int i = 0; i < {nq}; i++)")
        w("#pragma unroll")
        w(f"for (int o = {MS // 2}; o > 0; o >>= 1) rs{x}[i] += frnn_shfl_xor(rs{x}[i], o);")
        w(f"if (mi == 0{'' if QG <= C else f' && qg < {C}'}) {slot(n.name)} + qg + {QG} * i] = rs{x}[i];")
        w.close()
    w(f"bool ok = frnn_mbar_wait(&bar[0], 0, err, {ERR});")
    for u in range(min(NB, nsl)):
        uses = (nsl - u + NB - 1) // NB
        w(f"ok = frnn_mbar_wait(&bar[{5 if u else 1}], {(uses - 1) & 1}, err, {ERR}) && ok;")
    w("frnn_tmem_fence_after_sync();")
    w("frnn_block_sync();       // X, Z and the slices are no longer read")
    if second_s:
        w.open(f"if (tid >= 32 && tid < {32 + C})")
        w("const int q = tid - 32; (void)q;")
        scalar_nodes(second_s)
        w.close()
    w("const u32 lanes = tm + frnn_tmem_lane_base(warp);")
    w(f"float* Lr = (float*)(smem + {off_Lr});")
    # ---- L: rows (d, j) of hi and of rest, columns (r, i) of hi and of rest; each half of the threads takes half of the i
    def ld_L(dst):
        w(f"float {dst}[{nr * HC}];")
        w.open("")
        if restZ:
            w(f"float lo[{len(restZ) * HC}];")
        for r in range(nr):
            w(f"frnn_tmem_ld<{HC}>(lanes + {cL + r * C}u + (u32)q0, &{dst}[{r * HC}]);")
        for x, r in enumerate(restZ):
            w(f"frnn_tmem_ld<{HC}>(lanes + {cL + at_rest(restZ, r, nK)}u + (u32)q0, &lo[{x * HC}]);")
        w("frnn_tmem_wait_ld();")
        for x, r in enumerate(restZ):
            w("#pragma unroll")
            w(f"for (int k = 0; k < {HC}; k++) {dst}[{r * HC} + k] += lo[{x * HC} + k];")
        w.close()
    if restX:
        w.open(f"if (x128 >= {nA // 32 * 32} && x128 < {(RX + 31) // 32 * 32})")
        ld_L("u")
        w.open(f"if (x128 >= {nA} && x128 < {RX})")
        w("int at = x128 - %d;%s" % (nA, "".join(f" if (x128 >= {nA + x * C} && x128 < {nA + (x + 1) * C}) at += {(d - x) * C};" for x, d in enumerate(restX) if d != x)))
        w("#pragma unroll")
        w(f"for (int k = 0; k < {nr * HC}; k++) Lr[at * {LS} + (k / {HC}) * {C} + q0 + k % {HC}] = u[k];")
        w.close()
        w.close()
        w("frnn_block_sync();")
    w.open(f"if (x128 < {(nA + 31) // 32 * 32})")
    ld_L("u")
    w.open(f"if (x128 < {nA})")
    w(f"const int j = x128 % {C};")
    if restX:
        w.open(f"if ({' || '.join(f'x128 / {C} == {d}' for d in restX)})" if len(restX) < nd else "")
        w("#pragma unroll")
        w(f"for (int k = 0; k < {nr * HC}; k++) u[k] += Lr[x128 * {LS} + (k / {HC}) * {C} + q0 + k % {HC}];")
        w.close()
    if dec_sc:
        w(f"float D = 1.0f;          // decays between step j and the last of this part")
        w(f"for (int l = q0 + {HC}; l < {C}; l++) if (l < j && l < nv) D *= {slot(nf.decay)} + l];")
    # four columns of a row are one store of the operand with rows (d, j), and four single ones of the other
    w(f"unsigned char* d2 = smem + {off_L2} + (x128 >> 2) * {lbo2} + (x128 & 3) * 4;")
    w("#pragma unroll")
    w.open(f"for (int k4 = {HC - 4}; k4 >= 0; k4 -= 4)")
    w(f"float a[{nr}][4], lo[{nr}][4];")
    w("#pragma unroll")
    w.open("for (int k = 3; k >= 0; k--)")
    w("const int i = q0 + k4 + k;")
    w("#pragma unroll")
    w.open(f"for (int r = 0; r < {nr}; r++)")
    w(f"const int ri = r * {C} + i;")
    w(f"const float x = i < j ? u[r * {HC} + k4 + k] : 0.0f;")
    w(f"Lr[x128 * {LS} + ri] = x;")
    w("a[r][k] = x" + (" * D;" if dec_sc else ";") + " lo[r][k] = frnn_tf32_rest(a[r][k]);")
    w(f"const int rd = ri + {nK};")
    w("*(float*)(d2 + (ri >> 3) * 128 + (ri & 7) * 16) = a[r][k]; *(float*)(d2 + (rd >> 3) * 128 + (rd & 7) * 16) = lo[r][k];")
    w.close()
    if dec_sc:
        w(f"if (i < j && i < nv) D *= {slot(nf.decay)} + i];")
    w.close()
    w("#pragma unroll")
    w.open(f"for (int r = 0; r < {nr}; r++)")
    w(f"unsigned char* d1 = smem + {off_L1} + ((r * {C} + q0 + k4) >> 2) * {lbo1}; const int ra = x128, rb = x128 + {nA};")
    w("frnn_stv<0,4>(d1 + (ra >> 3) * 128 + (ra & 7) * 16, 0, a[r]); frnn_stv<0,4>(d1 + (rb >> 3) * 128 + (rb & 7) * 16, 0, lo[r]);")
    w.close()
    w.close()
    w.close()
    w.close()
    # ---- operands over the columns: kappa (over W) and alpha (times W), this thread's part of the timesteps
    if dec_vec:
        w(f"float xw[{HC}], pre = 1.0f, post = 1.0f, rpre = 1.0f, wlo = 1.0f, whi = 1.0f, prod = 1.0f;   // decays; products of the other parts'")
        w("#pragma unroll")
        w.open(f"for (int k = 0; k < {HC}; k++)")
        w.open("")
        w(f"const int q = q0 + k; const bool live = {live_n}; (void)live;")
        e = Stage("x_", "q", N1, {a: f"{reg(a)}[k]" for a in nleaves}).get(nf.decay)
        w(f"xw[k] = {sel(live_n, e, '1.0f')};")
        w("wlo = fminf(wlo, fabsf(xw[k]));")
        w.close()
        w("prod *= xw[k];")
        w.close()
        # the product of the other half's decays comes through shared memory
        w("xr[tid] = prod;")
        w("frnn_block_sync();")
        w("#pragma unroll")
        w("for (int o = 0; o < 2; o++) { const float x = xr[o * 128 + x128]; if (o < hf) pre *= x; if (o > hf) post *= x; }")
        w("rpre = frnn_rcp1(pre);")
        w("float rw = rpre, pw = pre;")
        if few:
            # a decay that is merely too small for its own gradient (dW/W, by a division) does not send the chunk down the slow
            # path, 160 us for a CTA: RWKV-7's decays fall below 2^-10 about once in two million
            w("u32 marks = 0;")
            w.open(f"if ({by_products('wlo')})")
            w("#pragma unroll")
            w(f"for (int k = 0; k < {HC}; k++) if ({by_products('xw[k]')}) marks |= 1u << k;")
            w("((volatile int*)&bar[4])[1] = 1;")
            w.close()
            w("fewm[tid] = (unsigned short)marks;")
    w("#pragma unroll")
    w.open(f"for (int k4 = 0; k4 < {HC}; k4 += 4)")
    names = nf.kappas + nf.alphas
    w(f"float x[{len(names)}][4];")
    w("#pragma unroll")
    w.open("for (int k = 0; k < 4; k++)")
    w(f"const int q = q0 + k4 + k; const bool live = {live_n}; (void)live; (void)q;")
    st = Stage("x_", "q", N1, {a: f"{reg(a)}[k4 + k]" for a in nleaves})
    if dec_vec:
        w("rw *= frnn_rcp1(xw[k4 + k]); whi = fmaxf(whi, fabsf(rw));")
    for x, nm in enumerate(names):
        f = "" if not dec_vec else (" * rw" if x < nr else " * pw")
        w(f"x[{x}][k] = {sel(live_n, st.get(nm) + f)};")
    if dec_vec:
        w("pw *= xw[k4 + k];")
    w.close()
    for x in range(len(names)):
        off, tb, r, exact = (off_kT, kT_b, x, xk) if x < nr else (off_aT, aT_b, x - nr, xa)
        w(f"{{ unsigned char* dst = smem + {off} + (({r * C} + q0 + k4) >> 2) * {lboT} + (x128 >> 3) * 128 + (x128 & 7) * 16; frnn_stv<0,4>(dst, 0, x[{x}]);")
        if not exact:
            w("#pragma unroll")
            w(f"for (int k = 0; k < 4; k++) x[{x}][k] = frnn_tf32_rest(x[{x}][k]);")
            w(f"frnn_stv<0,4>(dst + {tb}, 0, x[{x}]);")
        w("}")
    w.close()
    if dec_vec:
        w("if (!(wlo > 1e-25f && whi < 1e25f)) *(volatile int*)&bar[4] = 1;")
    # ---- the parts of the accumulators so far, from S_0 and E_C, scaled to what those from L need
    w("float R = 0.0f; (void)R;")

    def ld_part(dst: str, vecs: int, col0: int, inexact: Sequence[int], n: int):
        """dst[v * HC + k] = value of vector v at timestep q0 + k, with what the rest of the operand gave."""
        w.open("")
        if inexact:
            w(f"float lo[{len(inexact) * HC}];")
        for x in range(vecs):
            w(f"frnn_tmem_ld<{HC}>(lanes + {col0 + x * C}u + (u32)q0, &{dst}[{x * HC}]);")
        for k, x in enumerate(inexact):
            w(f"frnn_tmem_ld<{HC}>(lanes + {col0 + at_rest(inexact, x, n)}u + (u32)q0, &lo[{k * HC}]);")
        w("frnn_tmem_wait_ld();")
        for k, x in enumerate(inexact):
            w("#pragma unroll")
            w(f"for (int k = 0; k < {HC}; k++) {dst}[{x * HC} + k] += lo[{k * HC} + k];")
        w.close()

    def st_part(src: str, vecs: int, col0: int):
        for x in range(vecs):
            w(f"frnn_tmem_st<{HC}>(lanes + {col0 + x * C}u + (u32)q0, &{src}[{x * HC}]);")
    if dec_sc:
        w(f"float xw[{HC}], pre = {slot('Wp')} + q0], post = {slot('Ws')} + q0 + {HC - 1}];")
        w("#pragma unroll")
        w.open(f"for (int k = 0; k < {HC}; k++)")
        w("xw[k] = " + (f"{slot(nf.decay)} + q0 + k];" if whole else f"q0 + k < nv ? {slot(nf.decay)} + q0 + k] : 1.0f;"))
        w.close()
    w("frnn_block_sync();")
    w("const bool slow = *(volatile int*)&bar[4] != 0; (void)slow;")
    if few:
        w("const bool few = ((volatile int*)&bar[4])[1] != 0;")
    if slow_path:
        emit_slow_columns(w, C, nd, nr, nA, nK, tq, live_n, sel, nf, bp, dec_vec, want_gw, Stage, leaf, leaves_of, slot, LS, ((cD1, restX), (cD2, restZ)), off_slow, off_gw, few)
    if nf.decay:
        w.open("if (!slow)" if dec_vec else "")
        w(f"float dk[{nr * HC}];")
        ld_part("dk", nr, cD2, restZ, nK)
        w("float a = post;")
        if dec_vec:
            w(f"float y[{nr * HC}];")
            w("#pragma unroll")
            w(f"for (int k = 0; k < {nr * HC}; k++) y[k] = dk[k];")
        w("#pragma unroll")
        w(f"for (int k = {HC - 1}; k >= 0; k--) {{ " + " ".join(f"dk[{r * HC} + k] *= a;" for r in range(nr)) + " a *= xw[k]; }")
        if want_gw:
            # R_C = W_C Z + sum kappa (W_C / W) (E^T p)
            w("R = (ncol && hf == 0) ? z0[x128] * a : 0.0f;")
            w("#pragma unroll")
            w.open(f"for (int k = 0; k < {HC}; k++)")
            w(f"const int q = q0 + k; const bool live = {live_n}; (void)live; (void)q;")
            st = Stage("x_", "q", N1, {a: f"{reg(a)}[k]" for a in nleaves})
            for r, nm in enumerate(nf.kappas):
                w(f"R = fmaf({st.get(nm)}, {sel(live_n, f'dk[{r * HC} + k]')}, R);")
            w.close()
        if dec_vec:
            # kappa's: times W_C, over W_j at the end; alpha's: as they are, times W_j-1 at the end
            w("const float wc = a * pre;")
            w("#pragma unroll")
            w(f"for (int k = 0; k < {nr * HC}; k++) dk[k] = y[k] * wc;")
            st_part("dk", nr, cD2)
            if restX:
                w(f"float da[{nd * HC}];")
                ld_part("da", nd, cD1, restX, nA)
                st_part("da", nd, cD1)
        else:
            st_part("dk", nr, cD2)
            w(f"float da[{nd * HC}];")
            ld_part("da", nd, cD1, restX, nA)
            w("a = pre;")
            w("#pragma unroll")
            w(f"for (int k = 0; k < {HC}; k++) {{ " + " ".join(f"da[{d * HC} + k] *= a;" for d in range(nd)) + " a *= xw[k]; }")
            st_part("da", nd, cD1)
        w("frnn_tmem_wait_st();")
        w.close()
    w("frnn_async_proxy_fence(); frnn_tmem_fence_before_sync();")
    w("frnn_block_sync();")
    w.open("if (warp == 0 && frnn_elect())")
    w.open("if (ok)" if not dec_vec else "if (ok && !slow)")
    w("frnn_tmem_fence_after_sync();")
    for cd, offA, tb, exact, nk, offB, lboB, n2 in ((cD1, off_kT, kT_b, xk, nK, off_L1, lbo1, nA), (cD2, off_aT, aT_b, xa, nA, off_L2, lbo2, nK)):
        for part_ in ([offA] if exact else [offA, offA + tb]):
            for row in (0, n2):              # L and its rest
                w(f"{{ const u64 da = frnn_mma_desc(smem + {part_}, {lboT}), db = frnn_mma_desc(smem + {offB + row // 8 * 128}, {lboB});")
                w("#pragma unroll")
                w(f"for (int k = 0; k < {nk // 8}; k++) frnn_mma_ss_d(tm + {cd}u, frnn_mma_next(da, {lboT}, k), frnn_mma_next(db, {lboB}, k), FRNN_MMA_IDESC({n2}), true); }}")
    w.close()
    w("frnn_mma_commit(&bar[2]);")
    w.close()
    w(f"ok = frnn_mbar_wait(&bar[2], 0, err, {ERR}) && ok;")
    w("frnn_tmem_fence_after_sync();")
    # ---- columns: this thread's part of the timesteps
    w(f"float da[{nd * HC}], dk[{nr * HC}];")
    ld_part("da", nd, cD1, [] if nf.decay else restX, nA)
    ld_part("dk", nr, cD2, [] if nf.decay else restZ, nK)
    if dec_vec:
        # the accumulators held W_C/W_j of kappa's part times W_j and alpha's part over W_j-1
        w.open("if (!slow)")
        w("float a = pre, ra = rpre;")
        w("#pragma unroll")
        w(f"for (int k = 0; k < {HC}; k++) {{ ra *= frnn_rcp1(xw[k]); " + " ".join(f"da[{d * HC} + k] *= a;" for d in range(nd)) + " "
          + " ".join(f"dk[{r * HC} + k] *= ra;" for r in range(nr)) + " a *= xw[k]; }")
        w.close()
    if slow_path:
        w(f"const float* sl = (const float*)(smem + {off_slow}); const float* gwp = (const float*)(smem + {off_gw}); (void)sl; (void)gwp;")
    if dec_vec:
        w.open("if (slow)")
        w("#pragma unroll")
        w.open(f"for (int k = 0; k < {HC}; k++)")
        w(" ".join(f"da[{d * HC} + k] = sl[({d * C} + q0 + k) * 128 + x128];" for d in range(nd)) + " "
          + " ".join(f"dk[{r * HC} + k] = sl[({nA + r * C} + q0 + k) * 128 + x128];" for r in range(nr)))
        w.close()
        w.close()
    if dec_vec and want_gw:
        # the later half's share of the sums that lead from R_C to the earlier one
        w("float P = 0.0f;")
        w("#pragma unroll")
        w.open(f"for (int k = 0; k < {HC}; k++)")
        w(f"const int q = q0 + k; const bool live = {live_n}; (void)live; (void)q;")
        st = Stage("x_", "q", N1, {a: f"{reg(a)}[k]" for a in nleaves})
        kd = " + ".join(f"{st.get(nm)} * dk[{r * HC} + k]" for r, nm in enumerate(nf.kappas))
        ad = " + ".join(f"{st.get(nm)} * da[{d * HC} + k]" for d, nm in enumerate(nf.alphas))
        w(f"P += {sel(live_n, f'(({ad}) - ({kd}))')};")
        w.close()
        w(f"xr[tid] = R; xr[{NT} + tid] = P;")
        w("frnn_block_sync();")
        w("R = 0.0f;")
        w("#pragma unroll")
        w(f"for (int o = 0; o < 2; o++) R += xr[o * 128 + x128] + (o > hf ? xr[{NT} + o * 128 + x128] : 0.0f);")
    for x in range(n_nsum):
        w(f"float e{x}[{HC}];")
    w("#pragma unroll")
    w.open(f"for (int k = {HC - 1}; k >= 0; k--)")
    w(f"const int q = q0 + k, t = t0 + q; const bool live = {live_n}; (void)t; (void)live;")
    given = {f"ga{d}": f"da[{d * HC} + k]" for d in range(nd)}
    given.update({f"gk{r}": f"dk[{r * HC} + k]" for r in range(nr)})
    given.update({a: f"{reg(a)}[k]" for a in nleaves})
    st = Stage("x_", "q", N1, given)
    if want_gw:
        kd = " + ".join(f"{st.get(nm)} * dk[{r * HC} + k]" for r, nm in enumerate(nf.kappas))
        ad = " + ".join(f"{st.get(nm)} * da[{d * HC} + k]" for d, nm in enumerate(nf.alphas))
        gws = "gwp[q * 128 + x128]"
        if dec_vec:
            w(f"const float wdw = R - {sel(live_n, f'({kd})')};")
            w(f"R = wdw + {sel(live_n, f'({ad})')};")
            w(f"const float gw = slow{' || ' + by_products('xw[k]') if few else ''} ? {gws} : " + ("wdw;" if bp.log_decay else "frnn_divf(wdw, xw[k]);"))
            st.done["gw"] = "gw"
        else:
            w(f"e{n_nsum - 2}[k] = {sel(live_n, f'(slow ? {gws} : {kd})')}; e{n_nsum - 1}[k] = {sel(live_n, f'({ad})')};")
    for x, n in enumerate(nsums):
        w(f"e{x}[k] = {sel(live_n, st.get(n.args[0]))};")
    for i, o in bp.grads:
        if p.in_cls(i) != N1:
            continue
        val = st.get(o)
        sp = dspec[i]
        w(f"{'' if live_n == 'true' else 'if (live) '}frnn_io<{sp.dt}>::st(dx{i}, {_elem_off(sp, [(0, 'b'), (1, 't'), (2, 'h')])} + (long)x128 * {sp.st(4)}L, {val});")
    w.close()
    for x in range(n_nsum):
        reduce_lanes(f"e{x}", HC, f"part[{x * 4 * C} + (warp & 3) * {C} + q0 + @]")
    if dec_sc and want_gw:
        w("#pragma unroll")
        w("for (int o = 16; o > 0; o >>= 1) R += frnn_shfl_xor(R, o);")
        w(f"if (lane == 0) part[{n_nsum * 4 * C} + warp] = R;")
    w("frnn_tmem_fence_before_sync();")
    w("frnn_block_sync();")
    w(f"if (warp == 0) frnn_tmem_dealloc(tm, {tm_cols}u);")
    # ---- scalars
    total = lambda x, q: f"((part[{x * 4 * C} + {q}] + part[{x * 4 * C + C} + {q}]) + (part[{x * 4 * C + 2 * C} + {q}] + part[{x * 4 * C + 3 * C} + {q}]))"
    sgrads = [(i, o) for i, o in bp.grads if p.in_cls(i) == S11]
    if sgrads:
        w.open(f"if (tid >= 32 && tid < {32 + C})")
        w("const int q = tid - 32, t = t0 + q; const bool live = q < nv; (void)t;")
        for x, n in enumerate(nsums):
            w(f"{slot(n.name)} + q] = {total(x, 'q')};")
        if dec_sc and want_gw:
            w("float R = 0.0f, wdw = 0.0f;")
            w("#pragma unroll")
            w(f"for (int k = 0; k < {NT // 32}; k++) R += part[{n_nsum * 4 * C} + k];")
            w(f"for (int l = nv - 1; l >= q; l--) {{ wdw = R - {total(n_nsum - 2, 'l')}; R = wdw + {total(n_nsum - 1, 'l')}; }}")
            w(f"{slot('gw')} + q] = slow ? {total(n_nsum - 2, 'q')} : " + ("wdw;" if bp.log_decay else f"frnn_divf(wdw, {slot(nf.decay)} + q]);"))
        scalar_nodes(third_s)
        for i, o in sgrads:
            sp = dspec[i]
            val = f"{slot(o)} + q]" if isinstance(o, str) else lower.flit(o)
            off = _elem_off(sp, [(0, "b"), (1, "t"), (2, "h")])
            if atomic[i]:
                w(f"if (live) frnn_atomic_add_c((float*)dx{i} + ({off}), {val});")
            else:
                w(f"if (live) frnn_io<{sp.dt}>::st(dx{i}, {off}, {val});")
        w.close()
    w("(void)ok;")
    w.close()
    # cycles the tensor cores are busy for one CTA: L, the slices of S_0 and E_C (each in two terms), what follows from L
    pa, pk = product_cycles(RX, True), product_cycles(RZ, True)
    busy = M // 8 * (pk + 2 * pa + 2 * pk) + nK // 8 * (2 if xk else 4) * product_cycles(nA, True) + nA // 8 * (2 if xa else 4) * product_cycles(nK, True)
    return KernelSource("frnn_cvg", w.text().replace("@SMEM_BYTES@", str(smem_bytes)), (nchunk, H, B), NT, smem_bytes, params, decl,
                        {"chunk": C, "tile": [1, N, M], "packed": False, "tmem_cols": tm_cols, "tensor_cycles": busy}, [])


def emit_slow_columns(w, C, nd, nr, nA, nK, tq, live_n, sel, nf, bp, dec_vec, want_gw, Stage, leaf, leaves_of, slot, LS, acc, off_slow, off_gw, few):
    """Columns of a chunk with a decay too small to divide by: running products in plain loops, by the first four warps;
    the results (d alpha, d kappa, d decay for all timesteps) go through shared memory.  ``few``: where only
    single decays are too small for their own gradients, these alone."""
    w.open("if (slow || few)" if few else "if (slow)")
    w("frnn_tmem_fence_before_sync();")
    w("frnn_block_sync();         // the operands are no longer read")
    w.open("if (tid < 128)")
    w(f"float* sl = (float*)(smem + {off_slow}); float* gwp = (float*)(smem + {off_gw}); (void)sl; (void)gwp;")
    w(f"float ka[{nK}], aa[{nA}], ta[{nA}], tk[{nK}], xs[{C}];")
    for arr, cnt, (colx, inexact) in (("ta", nA, acc[0]), ("tk", nK, acc[1])):
        w.open("")
        w(f"float u[{cnt}], lo[{max(1, len(inexact)) * C}]; (void)lo;")
        w(f"frnn_tmem_ld<{cnt}>(lanes + {colx}u, u);" + (f" frnn_tmem_ld<{len(inexact) * C}>(lanes + {colx + cnt}u, lo);" if inexact else "") + " frnn_tmem_wait_ld();")
        for k, x in enumerate(inexact):
            w("#pragma unroll")
            w(f"for (int k = 0; k < {C}; k++) u[{x * C} + k] += lo[{k * C} + k];")
        w("#pragma unroll")
        w(f"for (int k = 0; k < {cnt}; k++) {arr}[k] = u[k];")
        w.close()
    if few:                                  # (Tensor Memory is read by whole warps)
        w.open("if (slow || fewm[x128] || fewm[128 + x128])")
    names = nf.alphas + nf.kappas + [nf.decay]
    lv = leaves_of(names, (0, 1))
    w("#pragma unroll 1")
    w.open(f"for (int q = 0; q < {C}; q++)")
    w(f"const int t = {tq('q')}; const bool live = {live_n}; (void)live; (void)t;")
    for a in lv:
        w(f"const float l_{a.replace('.', '_')} = {leaf(a, 't', 'nc')};")
    st = Stage("x_", "q", (0, 1), {a: f"l_{a.replace('.', '_')}" for a in lv})
    for r, nm in enumerate(nf.kappas):
        w(f"ka[{r * C} + q] = {sel(live_n, st.get(nm))};")
    for d, nm in enumerate(nf.alphas):
        w(f"aa[{d * C} + q] = {sel(live_n, st.get(nm))};")
    w(f"xs[q] = {sel(live_n, st.get(nf.decay), '1.0f')};")
    w.close()
    if want_gw:
        w("const float Z = ncol ? z0[x128] : 0.0f;")
        w("#pragma unroll 1")
        w.open(f"for (int j = 0; j < {C}; j++)")
        if few:
            w(f"if (!slow && !(fewm[j / {C // 2} * 128 + x128] >> (j % {C // 2}) & 1)) continue;")
        w("float A = 1.0f, Bj = 1.0f, g = 0.0f, s0 = 0.0f, Q = 1.0f;")
        w("for (int l = 0; l < j; l++) A *= xs[l];")
        w(f"for (int l = j + 1; l < {C}; l++) Bj *= xs[l];")
        w("#pragma unroll 1")
        w(f"for (int i = j + 1; i < {C}; i++) {{ " + " ".join(f"s0 += aa[{d * C} + i] * ta[{d * C} + i] * Q;" for d in range(nd)) + " Q *= xs[i]; }")
        w("g = A * (Bj * Z + s0);")
        w("float P = 1.0f;")
        w("#pragma unroll 1")
        w.open("for (int l = j - 1; l >= 0; l--)")
        w("#pragma unroll 1")
        w.open(f"for (int r = 0; r < {nr}; r++)")
        w(f"float e = Bj * tk[r * {C} + l]; Q = 1.0f;")
        w("#pragma unroll 1")
        w(f"for (int i = j + 1; i < {C}; i++) {{ " + " ".join(f"e += Lr[({d * C} + i) * {LS} + r * {C} + l] * aa[{d * C} + i] * Q;" for d in range(nd)) + " Q *= xs[i]; }")
        w(f"g += ka[r * {C} + l] * P * e;")
        w.close()
        w("P *= xs[l];")
        w.close()
        w(f"gwp[j * 128 + x128] = g" + (" * xs[j];" if bp.log_decay else ";"))
        w.close()
    if dec_vec:
        w.open("if (slow)")
        w("float a = 1.0f;")
        w("#pragma unroll 1")
        w(f"for (int q = 0; q < {C}; q++) {{ for (int d = 0; d < {nd}; d++) ta[d * {C} + q] *= a; a *= xs[q]; }}")
        w("a = 1.0f;")
        w("#pragma unroll 1")
        w(f"for (int q = {C - 1}; q >= 0; q--) {{ for (int r = 0; r < {nr}; r++) tk[r * {C} + q] *= a; a *= xs[q]; }}")
        w("#pragma unroll 1")
        w.open(f"for (int i = 0; i < {C}; i++)")
        w("a = 1.0f;")
        w("#pragma unroll 1")
        w.open(f"for (int j = i + 1; j < {C}; j++)")
        w("#pragma unroll 1")
        w(f"for (int dr = 0; dr < {nd * nr}; dr++) {{ const int d = dr / {nr}, r = dr % {nr}; const float L = Lr[(d * {C} + j) * {LS} + r * {C} + i] * a; "
          f"ta[d * {C} + j] += L * ka[r * {C} + i]; tk[r * {C} + i] += L * aa[d * {C} + j]; }}")
        w("a *= xs[j];")
        w.close()
        w.close()
        w("#pragma unroll 1")
        w(f"for (int k = 0; k < {nA}; k++) sl[k * 128 + x128] = ta[k];")
        w("#pragma unroll 1")
        w(f"for (int k = 0; k < {nK}; k++) sl[({nA} + k) * 128 + x128] = tk[k];")
        w.close()
    if few:
        w.close()
    w.close()
    w("frnn_block_sync();")
    w("frnn_tmem_fence_after_sync();")
    w.close()


# ---------------------------------------------------------------------------
# planning
# ---------------------------------------------------------------------------

@dataclass
class ChunkPlan:
    """The chunked kernels of one specialisation."""
    problem: Problem
    nf: Normal
    bp: Optional[BackwardPlan]                # None: only calls without gradients are chunked
    dspec: List[TensorSpec]
    atomic: List[bool]
    C: int = CHUNK                            # timesteps per chunk of the training kernels
    short: bool = True                        # whether calls without gradients are chunked
    #: The state's update in one rolled loop (10 KB less code) where more than half of the SMs have a CTA.  A scan's code, 60 to 85 KB
    #: with all its warps' roles, does not fit an SM's instruction cache, and what lies behind that is shared: with every SM
    #: fetching, less code is faster, with few the unrolled loops are (us, unrolled and rolled: 256 heads T1024 Delta Rule
    #: 128x128 forward 324 and 284, backward 368 and 348, RWKV-7 650 and 581, 655 and 579, Mamba-2 64x128 295 and 260, 303 and
    #: 264; 32 heads RWKV-7 64x64 T2048 371 and 400; 16 heads Gated Delta 128x128 T1500 222 and 214, 279 and 280; 15 heads GLA
    #: 96x80 100 and 98, 103 and 108).
    compact: bool = False

    def scan(self, spec: ScanSpec, C: int, **kw) -> KernelSource:
        return emit_scan(self.problem, spec, C, rows_per_cta(self.problem.M), **{"compact": self.compact, **kw})

    def forward(self, **kw) -> KernelSource:
        p = self.problem
        return self.scan(forward_spec(p, self.nf, self.bp.saved, True, self.C), self.C, **kw)

    def infer(self, **kw) -> KernelSource:
        """Without checkpoints a chunk may be longer, which pays as long as its time less than doubles: the chain of a chunk takes
        a part that does not depend on its length and a substitution that grows with nd nr C^2.  64 heads, T1024, us with 16 and
        with 32 steps: Delta Rule (two pairs of vectors) 128x128 148 and 130, 64x64 111 and 113, 32x32 102 and 98; Gated Delta Rule
        128x128 177 and 141; Mamba-2 (one pair) 128x128 164 and 116, 64x64 134 and 99; GLA (one pair) 128x128 192 and 162; RWKV-7
        (four pairs) 64x64 229 and 391.  At 64 timesteps, two chunks, 15.9 and 15.5 us for the Delta Rule with 128x128."""
        p = self.problem
        if len(self.nf.alphas) * len(self.nf.kappas) <= 2 and p.T >= 4 * CHUNK:
            try:
                ks = self.scan(forward_spec(p, self.nf, [], False, 2 * CHUNK), 2 * CHUNK, **kw)
                if ks.smem_bytes <= SMEM_BYTES:
                    return ks
            except lower.LoweringError:
                pass
        return self.scan(forward_spec(p, self.nf, [], False, CHUNK), CHUNK, **kw)

    def backward_scan(self, **kw) -> KernelSource:
        p = self.problem
        return self.scan(backward_scan_spec(p, self.nf, self.bp, self.dspec, self.C), self.C, **kw)

    def vector_grads(self) -> KernelSource:
        return emit_vector_grads(self.problem, self.nf, self.bp, self.dspec, self.atomic, self.C)

    def variants(self) -> List[dict]:
        """Keyword arguments of the scans worth timing; member 0 is the default."""
        first = 1 if self.compact else 2
        return [dict(state_unroll=first), dict(state_unroll=3 - first), dict(state_unroll=4)]


def _fits(cp: ChunkPlan) -> bool:
    """Whether the training kernels fit an SM."""
    try:
        return all(ks.smem_bytes <= SMEM_BYTES for ks in (cp.forward(), cp.backward_scan(), cp.vector_grads()))
    except lower.LoweringError:
        return False


def chunk_plan(plan) -> Optional[ChunkPlan]:
    """The chunked form of a specialisation (a ``twopass.Plan``), where it applies and is the faster one.

    It applies to one state in the normal form, of at most 128 columns (a multiple of 8: one tf32 product takes 8) - the
    state, its rest and the products of a chunk then fit Tensor Memory; training also wants the rows of a head in one
    CTA.  The inputs have 16 bits; for fp32 inputs the recurrent kernels stay, whose sums are fp32 throughout.

    A chunk costs a CTA the same chain whatever the state's size, and only one CTA fits an SM; the recurrent kernels' time
    grows with the state and they share an SM.  So, in kernel time, forward + backward: where every SM has at most one CTA (T128
    Delta Rule: 16 heads of 128x128 62 us against 100 us, 128 heads of 64x64 67 us against 91 us), and beyond that for
    large states (256 heads T1024 128x128: 1.12 ms against 2.56 ms; 512 heads of 64x128, T128: 288 against 353 us, Mamba-2
    293 against 432 us; but with the kernels before their last rework 512 heads of 64x64 376 against 321 us).  Calls without
    gradients beyond one CTA per SM also want more than half of Tensor Memory's 128 lanes in use (512 heads of 64x128, Mamba-2,
    before that rework: 114 against 94 us).

    Long calls beyond these lines may be faster chunked (64x64, T256, forward + backward, chunked and recurrent: 160 heads, Delta
    Rule, 191 and 259 us; 1024 heads 835 and 884), but not as accurate: two tf32 terms in the place of fp32 operands.  Against
    fp64 at T128, recurrent and chunked, outputs and gradients of the initial state, in 1e-7: GLA 64x64 0.8 and 3.1, 0.5 and 1.3;
    Delta Rule 64x64 1.7 and 2.5, 2.9 and 1.8, 64x128 1.8 and 2.8, 3.4 and 1.8.  So they stay."""
    p = plan.problem
    if plan.n_st != 1 or p.N % 8 or not 16 <= p.N <= 128 or p.T < 2 * CHUNK or 0 in (p.B, p.T, p.H):
        return None
    if any(s.dt not in (lower.DT_BF16, lower.DT_F16) for s in p.inputs) or p.states[0].dt == lower.DT_F64:
        return None
    if p.M < 8 or rows_per_cta(p.M) is None:
        return None
    for s in p.inputs:
        cls = (int(s.shape[3] > 1), int(s.shape[4] > 1))
        if list(s.shape[:3]) != [p.B, p.T, p.H] and not (cls == S11 and s.shape[1] == 1):
            return None
    one_wave = p.B * p.H * (p.M // rows_per_cta(p.M)) <= plan.n_sm
    if not one_wave and p.M * p.N < 8192:
        return None
    nf = normal_form(plan.g_fw, p.in_names, p.st_names[0], plan.n_out)
    if nf is None or not all(nf_inputs(nf)):
        return None
    cp = ChunkPlan(p, nf, None, [g.spec for g in plan.whole_grads], [g.atomic for g in plan.whole_grads])
    cp.compact = 2 * p.B * p.H * (p.M // rows_per_cta(p.M)) > plan.n_sm
    try:
        cp.short = (one_wave or p.M > 64) and cp.infer().smem_bytes <= SMEM_BYTES
        if p.M <= 128 and p.M % 8 == 0:
            v = local_vjp(nf, p.M, p.N)
            cp.bp = backward_plan(p, nf, *v) if v is not None else None
    except lower.LoweringError:
        return None
    if cp.bp is not None:
        # 32 steps per chunk halve the traffic of the chunk boundaries and the chains of the scans, but not the
        # substitution: for large states and few pairs of vectors (kernels, forward + backward: B8 T1024 H32 128x128 Delta Rule
        # 1.12 ms against 1.54 ms, Mamba-2 1.16 ms against 1.73 ms, 64x128 0.96 against 1.32; 64x64, T512, 32 heads 147 against 166
        # us, 140 heads 251 against 277; 140 heads of 32x32 202 both)
        if len(nf.alphas) * len(nf.kappas) <= 2 and p.M * p.N >= (4096 if one_wave else 8192) and p.T >= 4 * CHUNK:
            cp.C = 2 * CHUNK
            if not _fits(cp):
                cp.C = CHUNK
        if not _fits(cp):
            cp.bp = None
    return cp if cp.short or cp.bp is not None else None
