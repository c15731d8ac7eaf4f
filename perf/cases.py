"""The block-sparse contraction work that programs built on this package run, as cases that
can be timed and checked: single block kernels, one contraction, the coupled-cluster
ladder, a doubles-residual iteration, an energy gradient, the streamed triples energy and
the memory-bound block operations between contractions.

    listed()             the named cases
    draw(rng)            one more case of the same ranges
    prepare(case, seed)  inputs, tensors and plans a program holds before the call
    run(state)           one pass through the public entry points; its outputs
    work(case)           bytes and FP64 operations a pass cannot do without
    exact(case, seed)    the outputs of a first pass in 64 bits, from torch alone

Spin-orbital spaces hold `oa` occupied and `va` virtual orbitals per spin (O = 2 oa, V =
2 va).  Tile lists are drawn from the case's own `tiles` seed, so that every input seed of
a case has the same block structure.  All tensors live in torch allocations attached to
the framework's tensors, all generated on the GPU from the seed.
"""
from __future__ import annotations

import ctypes as C
import itertools
import math

import numpy as np
import torch

import tamm_b200 as tb
from tamm_b200 import _capi as A
from tamm_b200 import ccsd, triples
from tamm_b200 import workloads as W

F64 = torch.float64
MODES = {"fp64": tb.Precision.FP64, "int8": tb.Precision.INT8, "bf16x3": tb.Precision.BF16X3}
ARENA_BYTES = 72 << 30
CACHE_BYTES = 60 << 30  # split digits of read-only integrals kept across contractions


# ---------------------------------------------------------------------------- the cases

def listed():
    return [
        # One tile triple of the ladder through the block kernel entry point: what an application
        # that keeps its own task loop calls per (A block, B block) pair.  The smallest call.
        {"name": "tile_fp64", "kind": "tile", "mode": "fp64", "a": 24, "b": 31, "c": 29, "d": 37, "i": 20, "j": 20},
        # One dense contraction C(a,b,i,j) += A(a,c,i,k) B(c,b,k,j) of uniform tiles through the
        # scheduler: a small system, where the host's share and the launches count.
        {"name": "dense_fp64", "kind": "dense", "mode": "fp64", "o": 10, "v": 40, "tile": 10},
        # The particle-particle ladder r2 += v t2 of a small molecule, split-INT8.
        {"name": "ladder_int8_small", "kind": "ladder", "mode": "int8", "oa": 6, "va": 33, "lo": 24, "hi": 48,
         "tiles": 1},
        # The ladder in plain FP64, the mode a program starts from.
        {"name": "ladder_fp64", "kind": "ladder", "mode": "fp64", "oa": 15, "va": 90, "lo": 24, "hi": 48, "tiles": 1},
        # The ladder in split-INT8 at the largest size whose integrals fit the card several times.
        {"name": "ladder_int8", "kind": "ladder", "mode": "int8", "oa": 20, "va": 130, "lo": 24, "hi": 48, "tiles": 1},
        # The ladder in the FP32-class mode, as early iterations of a solver use it.
        {"name": "ladder_bf16x3", "kind": "ladder", "mode": "bf16x3", "oa": 15, "va": 100, "lo": 24, "hi": 48,
         "tiles": 2},
        # A whole doubles-residual iteration replayed as a CUDA graph: ladders, rings, Fock terms,
        # integrals built on demand, permuted adds, energy, norm and amplitude update.
        {"name": "ccsd_fp64", "kind": "ccsd", "mode": "fp64", "oa": 10, "va": 50, "lo": 20, "hi": 64, "tiles": 2},
        {"name": "ccsd_int8", "kind": "ccsd", "mode": "int8", "oa": 20, "va": 80, "lo": 20, "hi": 64, "tiles": 2},
        # Energy and its gradient by the tape, forward and backward contraction, digits of v kept.
        {"name": "gradient_int8", "kind": "gradient", "mode": "int8", "oa": 15, "va": 120, "lo": 24, "hi": 48,
         "tiles": 3},
        # Steps of the streamed triples energy: much more output than arithmetic per contraction,
        # and a new output tensor, work list and denominator table for every step.
        {"name": "triples_int8", "kind": "triples", "mode": "int8", "oa": 25, "va": 120, "tile": 40, "jtile": 2,
         "steps": 3, "tiles": 4},
        # P(ab) P(ij) antisymmetrisation of a ring term: four adds with permuted labels.
        {"name": "permuted_adds", "kind": "adds", "oa": 20, "va": 180, "lo": 24, "hi": 48, "tiles": 1},
        # End of an iteration: energy, residual norm and the denominator update of the amplitudes.
        {"name": "update", "kind": "update", "oa": 20, "va": 180, "lo": 24, "hi": 48, "tiles": 1},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["tile", "dense", "ladder", "ladder", "ladder", "ccsd", "ccsd", "gradient", "triples", "adds",
                       "update"])
    seed = rng.randrange(1 << 16)
    if kind == "tile":
        case = {"kind": kind, "mode": rng.choice(["fp64", "fp64", "int8"])}
        case.update({x: _log(rng, 8, 64) for x in "abcd"})
        case.update({x: _log(rng, 4, 40) for x in "ij"})
        return case
    if kind == "dense":
        o = _log(rng, 6, 24)
        return {"kind": kind, "mode": "fp64", "o": o, "v": rng.randint(2 * o, 4 * o), "tile": rng.randint(5, 20)}
    lo, hi = rng.choice([(24, 48), (20, 64), (10, 30)])
    if kind == "triples":
        oa = _log(rng, 6, 22)
        return {"kind": kind, "mode": rng.choice(["fp64", "int8"]), "oa": oa, "va": rng.randint(2 * oa, 5 * oa),
                "tile": rng.choice([20, 32, 40]), "jtile": 2, "steps": rng.randint(1, 3), "tiles": seed}
    if kind in ("adds", "update"):
        oa = _log(rng, 4, 20)
        return {"kind": kind, "oa": oa, "va": rng.randint(4 * oa, 9 * oa), "lo": lo, "hi": hi, "tiles": seed}
    top, ratio = {"ladder": (16, 7), "ccsd": (17, 4), "gradient": (13, 7)}[kind]
    oa = _log(rng, 4, top)
    mode = rng.choice({"ladder": ["fp64", "int8", "int8", "bf16x3"], "ccsd": ["fp64", "int8", "int8", "bf16x3"],
                       "gradient": ["fp64", "int8"]}[kind])
    return {"kind": kind, "mode": mode, "oa": oa, "va": rng.randint(3 * oa, ratio * oa), "lo": lo, "hi": hi,
            "tiles": seed}


# ------------------------------------------------------------------ blocks and their order

class Side:
    """One mode of a block tensor: tile extents and their spins."""

    def __init__(self, sizes, spins=None):
        self.sizes = [int(x) for x in sizes]
        self.spins = list(spins) if spins is not None else [0] * len(self.sizes)
        self.starts = [0, *itertools.accumulate(self.sizes)]


def _of(tis):
    return Side(tis.tile_sizes, tis.tile_spins)


def _spin_side(tiles):
    return Side(list(tiles) + list(tiles), [1] * len(tiles) + [2] * len(tiles))


def _cuts(n, tile):
    """Tiles of `tile`, the last one cut."""
    return [min(tile, n - s) for s in range(0, n, tile)]


def _pack(dense, sides, upper=None, lower=None):
    """Admitted blocks of a dense tensor in row-major tile order, each row-major: a block is
    admitted where the spins of the `upper` modes and of the `lower` modes have equal sums."""
    out = []
    for bid in itertools.product(*(range(len(s.sizes)) for s in sides)):
        if upper is not None and (sum(sides[m].spins[bid[m]] for m in upper) !=
                                  sum(sides[m].spins[bid[m]] for m in lower)):
            continue
        cut = tuple(slice(s.starts[b], s.starts[b + 1]) for s, b in zip(sides, bid))
        out.append(dense[cut].reshape(-1))
    return torch.cat(out) if out else torch.zeros(0, dtype=F64, device="cuda")


def _spins(n):
    return torch.tensor([1] * n + [2] * n, device="cuda")


def _admit(*modes):
    """1 where the spins of the first half of the modes sum to those of the second half."""
    h = len(modes) // 2
    s = 0
    for m, sp in enumerate(modes):
        shape = [1] * len(modes)
        shape[m] = -1
        s = s + (1 if m < h else -1) * sp.view(shape)
    return (s == 0).to(F64)


# ---------------------------------------------------------------------- synthetic chemistry

def _gen(seed, salt):
    return torch.Generator(device="cuda").manual_seed((int(seed) * 1000003 + salt) % (1 << 62))


def _randn(seed, salt, *shape):
    return torch.randn(*shape, dtype=F64, device="cuda", generator=_gen(seed, salt))


def _energies(oa, va, seed):
    """Orbital energies over [occ alpha, occ beta, virt alpha, virt beta], equal for both spins."""
    r = np.random.default_rng(seed + 1000)
    eo, ev = r.uniform(-2.0, -0.3, size=oa), r.uniform(0.1, 5.0, size=va)
    return np.concatenate([eo, eo, ev, ev])


def _cholesky(seed, salt, q, n1, n2, o1, o2):
    """L(Q,p,q) ~ N(0,1)/sqrt(Q) exp(-|p-q|/50), zero between the spins: (q, 2 n1, 2 n2), the
    positions p, q counted from o1, o2 for alpha and n1, n2 further for beta."""
    out = torch.zeros(q, 2 * n1, 2 * n2, dtype=F64, device="cuda")
    p1 = torch.arange(n1, dtype=F64, device="cuda")
    p2 = torch.arange(n2, dtype=F64, device="cuda")
    for s in (0, 1):
        damp = torch.exp(-((o1 + s * n1 + p1)[:, None] - (o2 + s * n2 + p2)[None, :]).abs() / 50.0)
        out[:, s * n1:(s + 1) * n1, s * n2:(s + 1) * n2] = _randn(seed, salt + s, q, n1, n2) / math.sqrt(q) * damp
    return out


def _amplitudes(seed, oa, va, eps):
    """t2(a,b,i,j) ~ N(0, 0.1^2) / (e_a + e_b - e_i - e_j) on the spin-conserving blocks."""
    e = torch.from_numpy(eps).cuda()
    eo, ev = e[:2 * oa], e[2 * oa:]
    t = 0.1 * _randn(seed, 7, 2 * va, 2 * va, 2 * oa, 2 * oa)
    t /= ev[:, None, None, None] + ev[None, :, None, None] - eo[None, None, :, None] - eo[None, None, None, :]
    t *= _admit(_spins(va), _spins(va), _spins(oa), _spins(oa))
    return t


def _nchol(case):
    return 5 * (2 * case["oa"] + 2 * case["va"])


def _tile_lists(case):
    rng = np.random.default_rng(case["tiles"])
    occ = W.random_tiles(case["oa"], case["lo"], case["hi"], rng)
    return occ, W.random_tiles(case["va"], case["lo"], case["hi"], rng)


# -------------------------------------------------------------------- framework-side helpers

_shared = {}


def _context(mode, cache=0):
    """The process's execution context (one stream, one arena), in the given precision mode."""
    if "ec" not in _shared:
        _shared["ec"] = tb.ExecutionContext(0, ARENA_BYTES)
    _shared["ec"].set_precision(MODES[mode], 1e-11)
    return _shared["ec"].set_digit_cache(cache)


class _Store:
    """Tensors of a case over torch allocations, kept together."""

    def __init__(self, ec):
        self.ec, self.mem, self.T = ec, {}, {}

    def new(self, name, spaces, values=None, **kw):
        t = tb.Tensor(spaces, **kw)
        m = torch.zeros(max(t.nelems, 1), dtype=F64, device="cuda")
        if values is not None:
            m[:t.nelems].copy_(values)
        t.attach(self.ec, m.data_ptr(), m.numel() * 8)
        self.mem[name], self.T[name] = m, t
        return t

    def drop(self, name):
        self.T.pop(name).deallocate()
        self.mem.pop(name)

    def out(self, name):
        """The packed values of a tensor (its own storage)."""
        return self.mem[name][:self.T[name].nelems]


def _spin_spaces(case):
    occ, virt = _tile_lists(case)
    MO = W.mo_tiled(case["oa"], case["va"], occ, virt)
    return MO("occ"), MO("virt")


def _integrals(S, V, q, name, L):
    """v(a,b,c,d) = sum_Q L(Q,a,c) L(Q,b,d) as a read-only tensor, built by the framework."""
    ec = S.ec
    CI = tb.TiledIndexSpace(tb.IndexSpace(q), 1000)
    Lt = S.new("L", [CI, V, V], _pack(L, [Side(_cuts(q, 1000)), _of(V), _of(V)], [1], [2]), spin_mask=[2, 0, 1])
    v = S.new(name, [V, V, V, V], spin=(2, 2))
    torch.cuda.synchronize()
    mode = S.mode
    ec.set_precision(tb.Precision.FP64)
    a, b, c, d = V.labels(4)
    k = CI.label()
    sch = tb.Scheduler(ec)
    sch(v(a, b, c, d).assign(Lt(k, a, c) * Lt(k, b, d))).execute()
    ec.set_precision(mode, 1e-11)
    S.drop("L")
    v.set_read_only(True)
    return v


# ---------------------------------------------------------------------------------- prepare

def prepare(case, seed):
    return globals()["_prepare_" + case["kind"]](case, int(seed))


def run(state):
    return state["run"](state)


def _ints(v, t):
    return np.ascontiguousarray(np.asarray(v, dtype=t))


def _tile_inputs(case, seed):
    x = {c: case[c] for c in "abcdij"}
    return (2 * torch.rand(*(x[c] for c in "abcd"), dtype=F64, device="cuda", generator=_gen(seed, 1)) - 1,
            2 * torch.rand(*(x[c] for c in "cdij"), dtype=F64, device="cuda", generator=_gen(seed, 2)) - 1,
            2 * torch.rand(*(x[c] for c in "abij"), dtype=F64, device="cuda", generator=_gen(seed, 3)) - 1)


def _prepare_tile(case, seed):
    a, b, c = _tile_inputs(case, seed)
    dims = [_ints(t.shape, np.int64) for t in (a, b, c)]
    labels = [_ints([-ord(x) for x in names], np.int32) for names in ("abcd", "cdij", "abij")]
    arg = []
    for t, d, l in zip((a, b, c), dims, labels):
        arg.append((t.data_ptr(), d.ctypes.data_as(A.i64p), l.ctypes.data_as(A.ip), 4))
    return {"run": _run_tile, "t": (a, b, c), "arg": arg, "keep": (dims, labels), "mode": MODES[case["mode"]]}


def _run_tile(s):
    a, b, c = s["arg"]
    A.call("tb_block_multiply", 0.75, *a, *b, 1.0, *c, 0, s["mode"], C.c_void_p(torch.cuda.current_stream().cuda_stream))
    return s["t"][2]


def _dense_inputs(case, seed):
    o, v = case["o"], case["v"]
    return (2 * torch.rand(v, v, o, o, dtype=F64, device="cuda", generator=_gen(seed, 1)) - 1,
            2 * torch.rand(v, v, o, o, dtype=F64, device="cuda", generator=_gen(seed, 2)) - 1)


def _prepare_dense(case, seed):
    ec = _context(case["mode"])
    S = _Store(ec)
    O, V = (tb.TiledIndexSpace(tb.IndexSpace(case[x]), case["tile"]) for x in "ov")
    sides = [_of(V), _of(V), _of(O), _of(O)]
    for name, x in zip("AB", _dense_inputs(case, seed)):
        S.new(name, [V, V, O, O], _pack(x, sides))
    S.new("C", [V, V, O, O])
    a, b, c = V.labels(3)
    i, j, k = O.labels(3)
    T = S.T
    return {"run": _run_op, "S": S, "sch": tb.Scheduler(ec), "out": S.out("C"),
            "op": T["C"](a, b, i, j).iadd(T["A"](a, c, i, k) * T["B"](c, b, k, j))}


def _run_op(s):
    s["sch"](s["op"]).execute(tb.ExecutionHW.GPU)
    return s["out"]


def _ladder_inputs(case, seed):
    eps = _energies(case["oa"], case["va"], seed)
    L = _cholesky(seed, 11, _nchol(case), case["va"], case["va"], 0, 0)
    return eps, L, _amplitudes(seed, case["oa"], case["va"], eps)


def _ladder_store(case, seed, cache=0):
    S = _Store(_context(case["mode"], cache))
    S.mode = MODES[case["mode"]]
    O, V = _spin_spaces(case)
    _, L, t2 = _ladder_inputs(case, seed)
    S.new("t2", [V, V, O, O], _pack(t2, [_of(V), _of(V), _of(O), _of(O)], [0, 1], [2, 3]), spin=(2, 2))
    _integrals(S, V, _nchol(case), "v", L)
    return S, O, V


def _prepare_ladder(case, seed):
    S, O, V = _ladder_store(case, seed)
    S.new("r2", [V, V, O, O], spin=(2, 2))
    a, b, c, d = V.labels(4)
    i, j = O.labels(2)
    T = S.T
    return {"run": _run_op, "S": S, "sch": tb.Scheduler(S.ec), "out": S.out("r2"),
            "op": T["r2"](a, b, i, j).iadd(T["v"](a, b, c, d) * T["t2"](c, d, i, j))}


def _gradient_weights(case, seed):
    oa, va = case["oa"], case["va"]
    w = _randn(seed, 29, 2 * oa, 2 * oa, 2 * va, 2 * va) / math.sqrt(4 * oa * va)
    return w * _admit(_spins(oa), _spins(oa), _spins(va), _spins(va))


def _prepare_gradient(case, seed):
    S, O, V = _ladder_store(case, seed, CACHE_BYTES)
    S.new("w", [O, O, V, V], _pack(_gradient_weights(case, seed), [_of(O), _of(O), _of(V), _of(V)], [0, 1], [2, 3]),
          spin=(2, 2))
    # the tape may release and re-allocate the outputs it records: arena storage
    X = tb.Tensor([V, V, O, O], spin=(2, 2)).allocate(S.ec)
    S.new("g", [V, V, O, O], spin=(2, 2))
    torch.cuda.synchronize()
    return {"run": _run_gradient, "S": S, "X": X, "labels": (*V.labels(4), *O.labels(2)), "sch": tb.Scheduler(S.ec),
            "tape": tb.Tape(S.ec)}


def _run_gradient(s):
    T, X, (a, b, c, d, i, j), tape = s["S"].T, s["X"], s["labels"], s["tape"].reset()
    s["sch"](T["g"]().assign(0.0)).execute()
    tape.leaf(T["t2"], T["g"])
    tape.contract(X(a, b, i, j), T["v"](a, b, c, d) * T["t2"](c, d, i, j))
    e = tape.dot(T["w"](i, j, a, b), T["t2"](a, b, i, j))
    e += tape.dot(T["t2"](a, b, i, j), X(a, b, i, j), 0.25)
    tape.backward()
    return {"energy": e, "gradient": s["S"].out("g")}


def _ccsd_inputs(case, seed):
    oa, va, q = case["oa"], case["va"], _nchol(case)
    eps = _energies(oa, va, seed)
    e = torch.from_numpy(eps).cuda()
    x = {"L_vo": _cholesky(seed, 11, q, va, oa, 2 * oa, 0), "L_oo": _cholesky(seed, 13, q, oa, oa, 0, 0),
         "L_vv": _cholesky(seed, 15, q, va, va, 0, 0)}
    for name, n, part, salt in (("f_oo", oa, e[:2 * oa], 21), ("f_vv", va, e[2 * oa:], 22)):
        f = 1e-3 * _randn(seed, salt, 2 * n, 2 * n) * _admit(_spins(n), _spins(n))
        f.fill_diagonal_(0.0)
        x[name] = f + torch.diag(part)
    return eps, x, _amplitudes(seed, oa, va, eps)


def _prepare_ccsd(case, seed):
    oa, va, q = case["oa"], case["va"], _nchol(case)
    ec = _context(case["mode"])
    S = _Store(ec)
    O, V = _spin_spaces(case)
    CI = tb.TiledIndexSpace(tb.IndexSpace(q), 1000)
    so, sv, sq = _of(O), _of(V), Side(_cuts(q, 1000))
    eps, x, t2 = _ccsd_inputs(case, seed)
    for name, p, r in (("L_vo", V, O), ("L_oo", O, O), ("L_vv", V, V)):
        S.new(name, [CI, p, r], _pack(x[name], [sq, _of(p), _of(r)], [1], [2]), spin_mask=[2, 0, 1])
    S.new("f_oo", [O, O], _pack(x["f_oo"], [so, so], [0], [1]), spin=(1, 1))
    S.new("f_vv", [V, V], _pack(x["f_vv"], [sv, sv], [0], [1]), spin=(1, 1))
    S.new("t0", [V, V, O, O], _pack(t2, [sv, sv, so, so], [0, 1], [2, 3]), spin=(2, 2))
    del x, t2
    for name, sp in (("v_vvoo", [V, V, O, O]), ("t2", [V, V, O, O]), ("r2", [V, V, O, O]), ("X", [V, V, O, O]),
                     ("v_oooo", [O, O, O, O]), ("W_oo", [O, O, O, O]), ("v_ovvo", [O, V, V, O]),
                     ("W_ov", [O, V, V, O])):
        S.new(name, sp, spin=(2, 2))
    S.new("F_vv", [V, V], spin=(1, 1))
    S.new("F_oo", [O, O], spin=(1, 1))
    torch.cuda.synchronize()
    T = S.T
    k0 = CI.label()
    a, b, c, d = V.labels(4)
    i, j, k, l = O.labels(4)
    sch = tb.Scheduler(ec)
    ec.set_precision(tb.Precision.FP64)
    sch(T["v_vvoo"](a, b, i, j).assign(T["L_vo"](k0, a, i) * T["L_vo"](k0, b, j)))
    sch(T["v_oooo"](k, l, i, j).assign(T["L_oo"](k0, k, i) * T["L_oo"](k0, l, j)))
    sch(T["v_ovvo"](k, b, c, j).assign(T["L_vo"](k0, c, k) * T["L_vo"](k0, b, j)))
    sch.execute(tb.ExecutionHW.GPU)
    ec.set_precision(MODES[case["mode"]], 1e-11)
    q2 = CI.label()

    def build(batch, first, last, bsch):
        ap = batch.spaces[0].label()
        b2, c2, d2 = V.labels(3)
        bsch(batch(ap, b2, c2, d2).assign(T["L_vv"](q2, ap, c2) * T["L_vv"](q2, b2, d2)))

    # batches of one virtual tile: the largest tile's share of v
    T["v_vvvv"] = tb.Tensor.built([V, V, V, V], build, spin=(2, 2),
                                  batch_bytes=8 * max(sv.sizes) * 3 * va ** 3)
    for name in ("L_vo", "L_oo", "L_vv", "f_oo", "f_vv", "v_vvoo", "v_oooo", "v_ovvo"):
        T[name].set_read_only(True)
    P = ccsd.CCSDProblem(ec, None, O, V, CI, eps, T, 0)
    sch = tb.Scheduler(ec)
    sch(T["t2"](a, b, i, j).assign(T["t0"](a, b, i, j)))  # every iteration starts from the same amplitudes
    ccsd.queue_iteration(P, sch)
    return {"run": _run_ccsd, "S": S, "P": P, "sch": sch, "graph": sch.graph()}


def _run_ccsd(s):
    s["graph"].launch().sync()
    energy, norm = (float(x) for x in s["sch"].scalars(2))
    return {"energy": energy, "norm": norm, "r2": s["S"].out("r2"), "t2": s["S"].out("t2")}


def _triples_steps(case):
    """The sampled streaming steps: (occupied index i, block of j)."""
    rng = np.random.default_rng(case["tiles"])
    nj = 2 * len(_cuts(case["oa"], case["jtile"]))
    return [(int(x) // nj, int(x) % nj) for x in rng.choice(2 * case["oa"] * nj, size=case["steps"], replace=False)]


def _triples_inputs(case, seed):
    oa, va, q = case["oa"], case["va"], _nchol(case)
    eps = _energies(oa, va, seed)
    return (eps, _cholesky(seed, 13, q, va, va, 0, 0), _cholesky(seed, 11, q, va, oa, 2 * oa, 0),
            _cholesky(seed, 15, q, oa, oa, 0, 0), _amplitudes(seed, oa, va, eps))


def _prepare_triples(case, seed):
    oa, va, q = case["oa"], case["va"], _nchol(case)
    ec = _context("fp64", CACHE_BYTES)
    S = _Store(ec)
    is_ = W.mo_index_space(oa, va)
    MOb, MO1, MOj, MOd = (tb.TiledIndexSpace(is_, n) for n in (case["tile"], 1, case["jtile"], va))
    V, Ob, O1, Oj, Vd = MOb("virt"), MOb("occ"), MO1("occ"), MOj("occ"), MOd("virt")
    CI = tb.TiledIndexSpace(tb.IndexSpace(q), 1000)
    eps, lvv, lvo, loo, t2 = _triples_inputs(case, seed)
    for name, x, p, r in (("L_vv", lvv, V, Vd), ("L_vo", lvo, V, Ob), ("L_oo", loo, Ob, Oj)):
        S.new(name, [CI, p, r], _pack(x, [Side(_cuts(q, 1000)), _of(p), _of(r)], [1], [2]), spin_mask=[2, 0, 1])
    for name, sp in (("t2x", [V, Vd, O1, Oj]), ("t2y", [V, V, O1, Ob])):
        S.new(name, sp, _pack(t2, [_of(x) for x in sp], [0, 1], [2, 3]), spin=(2, 2))
    del lvv, lvo, loo, t2
    S.new("vx", [V, V, Ob, Vd], spin=(2, 2))
    S.new("vy", [Ob, V, Oj, Ob], spin=(2, 2))
    torch.cuda.synchronize()
    T = S.T
    k0 = CI.label()
    b, c = V.labels(2)
    (d,), (j,) = Vd.labels(1), Oj.labels(1)
    k, l = Ob.labels(2)
    sch = tb.Scheduler(ec)
    sch(T["vx"](b, c, k, d).assign(T["L_vv"](k0, b, d) * T["L_vo"](k0, c, k)))
    sch(T["vy"](l, c, j, k).assign(T["L_oo"](k0, l, j) * T["L_vo"](k0, c, k)))
    sch.execute(tb.ExecutionHW.GPU)
    for name in ("L_vv", "L_vo", "L_oo"):
        S.drop(name)
    for t in T.values():
        t.set_read_only(True)
    steps = _triples_steps(case)
    sizes = [tb.Tensor([V, V, V, O1.sub(i, i + 1), Oj.sub(jt, jt + 1), Ob], spin=(3, 3)).nelems for i, jt in steps]
    W_ = torch.zeros(max(max(sizes), 1), dtype=F64, device="cuda")
    ec.set_precision(MODES[case["mode"]], 1e-11)
    torch.cuda.synchronize()
    P = triples.TriplesProblem(ec, V, Ob, O1, Oj, Vd, eps, T, W_.data_ptr(), W_.numel())
    return {"run": _run_triples, "S": S, "P": P, "W": W_, "steps": steps, "sch": tb.Scheduler(ec), "last": sizes[-1]}


def _run_triples(s):
    e, _, _ = triples.energy(s["P"], s["steps"], s["sch"])
    return {"energy": e, "W": s["W"][:s["last"]]}


def _adds_input(case, seed):
    oa, va = case["oa"], case["va"]
    return _randn(seed, 3, 2 * va, 2 * va, 2 * oa, 2 * oa)


def _prepare_adds(case, seed):
    ec = _context("fp64")
    S = _Store(ec)
    O, V = _spin_spaces(case)
    S.new("X", [V, V, O, O], _pack(_adds_input(case, seed), [_of(V), _of(V), _of(O), _of(O)], [0, 1], [2, 3]),
          spin=(2, 2))
    S.new("r2", [V, V, O, O], spin=(2, 2))
    return {"run": _run_adds, "S": S, "sch": tb.Scheduler(ec), "labels": (*V.labels(2), *O.labels(2))}


def _run_adds(s):
    (a, b, i, j), sch, r, X = s["labels"], s["sch"], s["S"].T["r2"], s["S"].T["X"]
    sch(r(a, b, i, j).assign(X(a, b, i, j)))
    sch(r(a, b, i, j).isub(X(b, a, i, j)))
    sch(r(a, b, i, j).isub(X(a, b, j, i)))
    sch(r(a, b, i, j).iadd(X(b, a, j, i)))
    sch.execute(tb.ExecutionHW.GPU)
    return s["S"].out("r2")


def _update_inputs(case, seed):
    oa, va = case["oa"], case["va"]
    eps = _energies(oa, va, seed)
    m = _admit(_spins(va), _spins(va), _spins(oa), _spins(oa))
    shape = (2 * va, 2 * va, 2 * oa, 2 * oa)
    return eps, _amplitudes(seed, oa, va, eps), 1e-3 * _randn(seed, 4, *shape) * m, 0.1 * _randn(seed, 5, *shape) * m


def _prepare_update(case, seed):
    ec = _context("fp64")
    S = _Store(ec)
    O, V = _spin_spaces(case)
    eps, t2, r2, v = _update_inputs(case, seed)
    for name, x in (("t2", t2), ("r2", r2), ("v", v)):
        S.new(name, [V, V, O, O], _pack(x, [_of(V), _of(V), _of(O), _of(O)], [0, 1], [2, 3]), spin=(2, 2))
    return {"run": _run_update, "S": S, "sch": tb.Scheduler(ec), "labels": (*V.labels(2), *O.labels(2)), "eps": eps}


def _run_update(s):
    lab, sch, T = s["labels"], s["sch"], s["S"].T
    sch.dot(0, T["v"](*lab), T["t2"](*lab), 0.25)
    sch.norm(1, T["r2"](*lab))
    sch.denom(T["t2"](*lab), -1.0, T["r2"](*lab), s["eps"], [1, 1, -1, -1])
    sch.execute(tb.ExecutionHW.GPU)
    energy, norm = (float(x) for x in sch.scalars(2))
    return {"energy": energy, "norm": norm, "t2": s["S"].out("t2")}


# ------------------------------------------------------------------------------------- work

# Operands of the iteration's contractions: letters a-h virtual, i-p occupied, Q Cholesky.
_CCSD_TERMS = ["cdkl,bdkl", "cdkl,cdjl", "cdkl,cdij", "cdkl,dblj", "bc,acij", "ac,bcij", "kj,abik", "ki,abjk",
               "klij,abkl", "acik,kbcj", "abcd,cdij", "Qac,Qbd"]


def _spin_flops(term, oa, va, q, paired):
    """FP64 operations of a contraction over the spin combinations with nonzero operands: a
    4-index operand conserves spin between its first and last two labels; integral operands
    (`paired`) also pairwise (first with third, second with fourth)."""
    ops = term.split(",")
    labels = sorted(set("".join(ops)) - {"Q"})
    n = 0
    for s in itertools.product((0, 1), repeat=len(labels)):
        sp = dict(zip(labels, s))
        ok = True
        for k, x in enumerate(ops):
            x = x.replace("Q", "")
            h = len(x) // 2
            ok &= sum(sp[c] for c in x[:h]) == sum(sp[c] for c in x[h:])
            if k in paired and len(x) == 4:
                ok &= sp[x[0]] == sp[x[2]]
        n += ok
    size = 1.0
    for c in labels:
        size *= va if c in "abcdefgh" else oa
    return 2.0 * n * size * (q if "Q" in term else 1)


def work(case):
    k = case["kind"]
    if k == "tile":
        a, b, c, d, i, j = (case[x] for x in "abcdij")
        return {"bytes": 8.0 * (a * b * c * d + c * d * i * j + 2 * a * b * i * j), "flops": 2.0 * a * b * c * d * i * j}
    if k == "dense":
        n = (case["o"] * case["v"]) ** 2
        return {"bytes": 8.0 * 4 * n, "flops": 2.0 * (case["o"] * case["v"]) ** 3}
    oa, va, q = case["oa"], case["va"], _nchol(case)
    t2 = 6.0 * va ** 2 * oa ** 2  # stored elements of t2, r2 (the spin-conserving quarter-and-a-half)
    if k == "adds":
        return {"bytes": 8.0 * 2 * t2, "flops": 0.0}
    if k == "update":
        return {"bytes": 8.0 * 4 * t2, "flops": 8.0 * t2}
    if k == "ladder":
        return {"bytes": 8.0 * (4.0 * va ** 4 + 3 * t2), "flops": _spin_flops("abcd,cdij", oa, va, q, {0})}
    if k == "gradient":
        return {"bytes": 8.0 * (4.0 * va ** 4 + 3 * t2), "flops": 2 * _spin_flops("abcd,cdij", oa, va, q, {0})}
    if k == "ccsd":
        flops = sum(_spin_flops(t, oa, va, q, {0} if t[:4] in ("cdkl", "abcd") else set()) for t in _CCSD_TERMS)
        nbytes = 8.0 * (2 * q * (va * va + va * oa + oa * oa) + 3 * t2 + 4.0 * (va * oa) ** 2 * 2 + 4.0 * oa ** 4)
        return {"bytes": nbytes, "flops": flops}
    flops, out, last = 0.0, 0.0, 0.0
    cuts = _cuts(oa, case["jtile"])
    for i, jt in _triples_steps(case):
        nj, si, sj = cuts[jt % len(cuts)], i // oa, jt // len(cuts)
        n1 = n2 = n = 0
        for a, b, c, kk in itertools.product((0, 1), repeat=4):
            if a + b + c != si + sj + kk:
                continue
            n += 1
            n1 += c == kk and a + b == si + sj  # d carries b's spin, v(b,c,d,k) pairs c with k
            n2 += c == kk and a + b == si + sj  # l carries j's spin, v(l,c,j,k) pairs c with k
        last = float(n) * va ** 3 * oa * nj
        flops += 2.0 * va ** 3 * oa * nj * (n1 * va + n2 * oa) + 3 * last
        out += last
    return {"bytes": 8.0 * (4.0 * va ** 3 * oa + 4.0 * va * oa ** 3 + last), "flops": flops}


# ------------------------------------------------------------------------------------ exact

def exact(case, seed):
    return globals()["_exact_" + case["kind"]](case, int(seed))


def _exact_tile(case, seed):
    a, b, c = _tile_inputs(case, seed)
    return c + 0.75 * torch.einsum("abcd,cdij->abij", a, b)


def _exact_dense(case, seed):
    x, y = _dense_inputs(case, seed)
    v, o = Side(_cuts(case["v"], case["tile"])), Side(_cuts(case["o"], case["tile"]))
    return _pack(torch.einsum("acik,cbkj->abij", x, y), [v, v, o, o])


def _vt(L, t2, chunk_bytes=4 << 30, transpose=False):
    """sum_cd v(a,b,c,d) t2(c,d,i,j), or sum_ab v(a,b,c,d) t2(a,b,i,j), v = sum_Q L(Q,a,c) L(Q,b,d)
    formed for a few first indices at a time."""
    if transpose:
        L = L.transpose(1, 2)
    q, n = L.shape[0], L.shape[1]
    o2 = t2.shape[2] * t2.shape[3]
    out = torch.empty(n, n, t2.shape[2], t2.shape[3], dtype=F64, device="cuda")
    right = L.reshape(q, n * n)
    tm = t2.reshape(n * n, o2)
    step = max(1, int(chunk_bytes // (8 * n ** 3)))
    for a0 in range(0, n, step):
        a1 = min(n, a0 + step)
        v = (L[:, a0:a1].reshape(q, -1).T @ right).reshape(a1 - a0, n, n, n)  # (a, c, b, d)
        out[a0:a1] = (v.permute(0, 2, 1, 3).reshape((a1 - a0) * n, n * n) @ tm).reshape(out[a0:a1].shape)
    return out


def _spin_sides(case):
    occ, virt = _tile_lists(case)
    return _spin_side(occ), _spin_side(virt)


def _exact_ladder(case, seed):
    _, L, t2 = _ladder_inputs(case, seed)
    o, v = _spin_sides(case)
    return _pack(_vt(L, t2), [v, v, o, o], [0, 1], [2, 3])


def _exact_gradient(case, seed):
    _, L, t2 = _ladder_inputs(case, seed)
    w = _gradient_weights(case, seed).permute(2, 3, 0, 1)
    o, v = _spin_sides(case)
    X = _vt(L, t2)
    energy = float((w * t2).sum() + 0.25 * (t2 * X).sum())
    g = w + 0.25 * X + 0.25 * _vt(L, t2, transpose=True)
    return {"energy": energy, "gradient": _pack(g, [v, v, o, o], [0, 1], [2, 3])}


def _exact_ccsd(case, seed):
    eps, x, t = _ccsd_inputs(case, seed)
    E = torch.einsum
    Lvo, Loo = x["L_vo"], x["L_oo"]
    v = E("qai,qbj->abij", Lvo, Lvo)
    F_vv = x["f_vv"] - 0.5 * E("cdkl,bdkl->bc", v, t)
    F_oo = x["f_oo"] + 0.5 * E("cdkl,cdjl->kj", v, t)
    W_oo = 0.5 * E("qki,qlj->klij", Loo, Loo) + 0.25 * E("cdkl,cdij->klij", v, t)
    W_ov = E("qck,qbj->kbcj", Lvo, Lvo) + 0.5 * E("cdkl,dblj->kbcj", v, t)
    r = v + E("bc,acij->abij", F_vv, t) - E("ac,bcij->abij", F_vv, t) - E("kj,abik->abij", F_oo, t)
    r += E("ki,abjk->abij", F_oo, t)
    r += E("klij,abkl->abij", W_oo, t)
    X = E("acik,kbcj->abij", t, W_ov)
    r += X - X.permute(1, 0, 2, 3) - X.permute(0, 1, 3, 2) + X.permute(1, 0, 3, 2)
    r += 0.5 * _vt(x["L_vv"], t)
    e = torch.from_numpy(eps).cuda()
    no = 2 * case["oa"]
    eo, ev = e[:no], e[no:]
    D = ev[:, None, None, None] + ev[None, :, None, None] - eo[None, None, :, None] - eo[None, None, None, :]
    o, vv = _spin_sides(case)
    sides = [vv, vv, o, o]
    rp = _pack(r, sides, [0, 1], [2, 3])
    return {"energy": float(0.25 * (v * t).sum()), "norm": float(rp.norm()), "r2": rp,
            "t2": _pack(t - r / D, sides, [0, 1], [2, 3])}


def _exact_triples(case, seed):
    oa, va = case["oa"], case["va"]
    eps, lvv, lvo, loo, t2 = _triples_inputs(case, seed)
    e = torch.from_numpy(eps).cuda()
    eo, ev = e[:2 * oa], e[2 * oa:]
    so, sv = _spins(oa), _spins(va)
    vb = _spin_side(_cuts(va, case["tile"]))
    ob = _spin_side(_cuts(oa, case["tile"]))
    cuts = _cuts(oa, case["jtile"])
    starts = [0, *itertools.accumulate(cuts + cuts)]
    energy, packed = 0.0, None
    steps = _triples_steps(case)
    vx = torch.einsum("qbd,qck->dbck", lvv, lvo).reshape(2 * va, -1)  # (d, b c k)
    for n, (i, jt) in enumerate(steps):
        j = slice(starts[jt], starts[jt + 1])
        nj = j.stop - j.start
        x = t2[:, :, i, j].permute(0, 2, 1)  # (a, j, d)
        vy = torch.einsum("qlj,qck->lcjk", loo[:, :, j], lvo)
        dense = torch.empty(2 * va, 2 * va, 2 * va, 1, nj, 2 * oa, dtype=F64, device="cuda")
        ok = _admit(sv, sv, sv, so[i:i + 1], so[j], so)
        for a in range(2 * va):
            w = (x[a] @ vx).reshape(nj, 2 * va, 2 * va, 2 * oa).permute(1, 2, 0, 3)
            w = w - torch.einsum("bl,lcjk->bcjk", t2[a, :, i, :], vy)
            w = w * ok[a, :, :, 0]
            D = (eo[i] + eo[j][None, None, :, None] + eo[None, None, None, :] - ev[a] - ev[:, None, None, None] -
                 ev[None, :, None, None])
            energy += float((w * w / D).sum())
            dense[a, :, :, 0] = w
        del ok
        if n == len(steps) - 1:
            sides = [vb, vb, vb, Side([1], [int(so[i])]), Side([nj], [int(so[j.start])]), ob]
            packed = _pack(dense, sides, [0, 1, 2], [3, 4, 5])
        del dense
    return {"energy": energy, "W": packed}


def _exact_adds(case, seed):
    x = _adds_input(case, seed)
    o, v = _spin_sides(case)
    r = x - x.permute(1, 0, 2, 3) - x.permute(0, 1, 3, 2) + x.permute(1, 0, 3, 2)
    return _pack(r, [v, v, o, o], [0, 1], [2, 3])


def _exact_update(case, seed):
    eps, t2, r2, v = _update_inputs(case, seed)
    e = torch.from_numpy(eps).cuda()
    no = 2 * case["oa"]
    eo, ev = e[:no], e[no:]
    D = ev[:, None, None, None] + ev[None, :, None, None] - eo[None, None, :, None] - eo[None, None, None, :]
    o, vs = _spin_sides(case)
    return {"energy": 0.25 * float((v * t2).sum()), "norm": float(r2.norm()),
            "t2": _pack(t2 - r2 / D, [vs, vs, o, o], [0, 1], [2, 3])}
