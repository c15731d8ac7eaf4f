"""The FP64 contraction kernel repeated: a particle ladder r2(a,b,i,j) = v(a,b,c,d) t2(c,d,i,j) of
30 spin-orbital occupied and 180 virtual, whose launch has all the kernel does at once - more
items than CTAs, ragged tiles, tiles of several K segments that run whole and others spread
over CTAs.  Every pass over alternating inputs gives the bits of the first pass over the same
inputs, rebuilt integrals the bits of the first ones, and that first pass agrees with torch in
64 bits.

The bound: r2 = sum over 16200 (c,d) of sums over Q = 1050 products, so any two orders of
summation differ by at most 2 (16200 + 1050 + 2) 2^-53 of the same sums of magnitudes."""
import itertools

import pytest

import tamm_b200 as tb
from tamm_b200 import workloads as W

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

OA, VA, Q, PASSES = 15, 90, 1050, 360
OCC, VIRT = [15], [35, 36, 19]
F64 = torch.float64


def _spin(n):
    return torch.tensor([0] * n + [1] * n, device="cuda")


def _attached(ec, spaces, **kw):
    t = tb.Tensor(spaces, **kw)
    m = torch.zeros(t.nelems, dtype=F64, device="cuda")
    t.attach(ec, m.data_ptr(), m.numel() * 8)
    return t, m


def _blocks(dense, tiles, admit):
    """Packed blocks of a dense tensor, row-major over the admitted tile combinations."""
    cuts, out = [], []
    for sizes in tiles:
        starts = [0]
        for n in sizes + sizes:
            starts.append(starts[-1] + n)
        cuts.append(starts)
    for bid in itertools.product(*(range(len(c) - 1) for c in cuts)):
        spins = [b >= len(t) for b, t in zip(bid, tiles)]
        if admit(spins):
            out.append(dense[tuple(slice(c[b], c[b + 1]) for c, b in zip(cuts, bid))].reshape(-1))
    return torch.cat(out)


def _ladder(L, t2):
    """sum_cd (sum_Q L(Q,a,c) L(Q,b,d)) t2(c,d,i,j), a few a at a time."""
    n, out = L.shape[1], []
    for a in range(0, n, 20):
        v = torch.einsum("qac,qbd->abcd", L[:, a:a + 20], L)
        out.append(torch.einsum("abcd,cdij->abij", v, t2))
    return torch.cat(out)


def _pairs():
    """Slices of the spin-conserving tile pairs of two virtual modes, in tile order."""
    cut, p = [], 0
    for n in VIRT + VIRT:
        cut.append(slice(p, p + n))
        p += n
    h = len(VIRT)
    return [(cut[x], cut[y]) for x in range(2 * h) for y in range(2 * h) if (x < h) == (y < h)]


def test_every_pass_has_the_first_ones_bits():
    ec = tb.ExecutionContext(0, 1 << 30)
    MO = W.mo_tiled(OA, VA, OCC, VIRT)
    O, V = MO("occ"), MO("virt")
    CI = tb.TiledIndexSpace(tb.IndexSpace(Q), 1000)
    a, b, c, d = V.labels(4)
    i, j = O.labels(2)
    k = CI.label()
    r2, rm = _attached(ec, [V, V, O, O], spin=(2, 2))
    states = []
    for seed in (1, 2):
        g = torch.Generator(device="cuda").manual_seed(seed)
        sv, so = _spin(VA), _spin(OA)
        L = torch.randn(Q, 2 * VA, 2 * VA, dtype=F64, device="cuda", generator=g) / Q ** 0.5
        L *= sv[:, None] == sv[None, :]
        t2 = torch.randn(2 * VA, 2 * VA, 2 * OA, 2 * OA, dtype=F64, device="cuda", generator=g)
        t2 *= (sv[:, None, None, None] + sv[None, :, None, None]) == (so[None, None, :, None] + so[None, None, None, :])
        Lt, lm = _attached(ec, [CI, V, V], spin_mask=[2, 0, 1])
        lm.copy_(torch.cat([x[:, p, q].reshape(-1) for x in (L[:1000], L[1000:]) for p, q in _pairs()]))
        tt, tm = _attached(ec, [V, V, O, O], spin=(2, 2))
        tm.copy_(_blocks(t2, [VIRT, VIRT, OCC, OCC], lambda s: s[0] + s[1] == s[2] + s[3]))
        v, vm = _attached(ec, [V, V, V, V], spin=(2, 2))
        states.append({"L": L, "t2": t2, "Lt": Lt, "lm": lm, "tt": tt, "tm": tm, "v": v, "vm": vm})
    torch.cuda.synchronize()
    for s in states:
        build = tb.Scheduler(ec)
        build(s["v"](a, b, c, d).assign(s["Lt"](k, a, c) * s["Lt"](k, b, d))).execute(tb.ExecutionHW.GPU)
        first = s["vm"].clone()
        for _ in range(10):
            s["vm"].fill_(-1.0)
            torch.cuda.synchronize()
            build(s["v"](a, b, c, d).assign(s["Lt"](k, a, c) * s["Lt"](k, b, d))).execute(tb.ExecutionHW.GPU)
            assert torch.equal(s["vm"], first)
        del first
        s["v"].set_read_only(True)  # (its zero blocks are found: half the tasks of the mixed spins are skipped)
        s["sch"], s["first"] = tb.Scheduler(ec), None
    wrong = []
    for n in range(PASSES):
        s = states[n % 2]
        rm.zero_()
        torch.cuda.synchronize()
        s["sch"](r2(a, b, i, j).iadd(s["v"](a, b, c, d) * s["tt"](c, d, i, j))).execute(tb.ExecutionHW.GPU)
        if s["first"] is None:
            s["first"] = rm.clone()
        elif not torch.equal(rm, s["first"]):
            wrong.append((n, int((rm != s["first"]).sum())))
    assert wrong == []
    for s in states:
        eps = 2 * (4 * VA * VA // 2 + Q + 2) * 2.0 ** -53
        pack = lambda x: _blocks(x, [VIRT, VIRT, OCC, OCC], lambda p: p[0] + p[1] == p[2] + p[3])  # noqa: E731
        want, mag = pack(_ladder(s["L"], s["t2"])), pack(_ladder(s["L"].abs(), s["t2"].abs()))
        assert bool(((s["first"] - want).abs() <= eps * mag).all())
        s["v"].set_read_only(False)
    ec.close()
