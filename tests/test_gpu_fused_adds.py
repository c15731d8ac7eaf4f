"""Runs of AddOps of one destination and one source that the scheduler executes in one pass,
bit for bit against the same ops executed one by one (a profiled execute times every op, so
it runs them apart): the P(ab) P(ij) terms and other permutations, with spin blocks, tiles
below, at and above the sub-tile's extents (64 and 32), one-element modes, partial label
spaces, and runs that cannot share a pass (two transposing modes) or only in part."""
import numpy as np
import pytest

import tamm_b200 as tb
from tamm_b200 import workloads as W

pytestmark = pytest.mark.gpu


def _run(ec, R, X, r0, ops, apart):
    R.write(r0)
    sch = tb.Scheduler(ec)
    for f in ops:
        sch(f(R, X))
    sch.execute(tb.ExecutionHW.GPU, apart)
    return R.read()


def _check(ec, R, X, seed, ops):
    rng = np.random.default_rng(seed)
    X.write(rng.normal(size=X.nelems))
    r0 = rng.normal(size=R.nelems)
    assert np.array_equal(_run(ec, R, X, r0, ops, False), _run(ec, R, X, r0, ops, True))


@pytest.mark.parametrize("assign", [True, False])
@pytest.mark.parametrize("occ,virt", [([3, 2], [5, 4, 1]), ([8, 7], [9, 12]), ([20], [33, 7]), ([65, 2], [3, 2]),
                                      ([33, 31], [2, 3]), ([1, 9], [6])])
def test_antisymmetrisation(ec, occ, virt, assign):
    MO = W.mo_tiled(sum(occ), sum(virt), occ, virt)
    O, V = MO("occ"), MO("virt")
    R, X = (tb.Tensor([V, V, O, O], spin=(2, 2)).allocate(ec) for _ in range(2))
    (a, b), (i, j) = V.labels(2), O.labels(2)
    first = (lambda R, X: R(a, b, i, j).assign(0.3 * X(a, b, i, j))) if assign else (
        lambda R, X: R(a, b, i, j).iadd(0.3 * X(a, b, i, j)))
    _check(ec, R, X, 1, [first, lambda R, X: R(a, b, i, j).isub(1.7 * X(b, a, i, j)),
                         lambda R, X: R(a, b, i, j).isub(0.9 * X(a, b, j, i)),
                         lambda R, X: R(a, b, i, j).iadd(X(b, a, j, i)),
                         lambda R, X: R(a, b, i, j).iadd(0.1 * X(b, a, i, j))])  # (a fifth: a pass of its own)
    av, io = V.sub(0, 1).label(), O.sub(0, 1).label()  # the first tiles only
    a2, i2 = V.sub(0, 1).label(), O.sub(0, 1).label()
    _check(ec, R, X, 2, [lambda R, X: R(av, a2, io, i2).iadd(0.3 * X(a2, av, io, i2)),
                         lambda R, X: R(av, a2, io, i2).iadd(0.6 * X(av, a2, i2, io))])
    for t in (R, X):
        t.deallocate()


@pytest.mark.parametrize("perms", [("ijk", "jik"), ("kij", "kji"), ("jik", "kij"), ("ikj", "kji"), ("ijk", "kji")])
@pytest.mark.parametrize("tiles", [[70, 9], [3, 1, 40], [64, 32]])
def test_three_modes(ec, tiles, perms):
    S = tb.TiledIndexSpace(tb.IndexSpace(sum(tiles)), tiles)
    R, X = (tb.Tensor([S, S, S]).allocate(ec) for _ in range(2))
    lab = dict(zip("ijk", S.labels(3)))
    ops = [lambda R, X, p=p, n=n: R(*(lab[c] for c in "ijk")).iadd((0.7 - n) * X(*(lab[c] for c in p)))
           for n, p in enumerate(perms)]
    _check(ec, R, X, 3, ops)
    for t in (R, X):
        t.deallocate()


def test_captured(ec):
    """A run inside a captured graph: the replay repeats the eager result."""
    S = tb.TiledIndexSpace(tb.IndexSpace(50), [20, 30])
    R, X = (tb.Tensor([S, S]).allocate(ec) for _ in range(2))
    rng = np.random.default_rng(4)
    X.write(rng.normal(size=X.nelems))
    i, j = S.labels(2)
    sch = tb.Scheduler(ec)
    sch(R(i, j).assign(X(i, j)))(R(i, j).isub(0.5 * X(j, i)))
    g = sch.graph()
    eager = R.read()
    R.write(np.zeros(R.nelems))
    g.launch().sync()
    assert np.array_equal(R.read(), eager)
    del g
    for t in (R, X):
        t.deallocate()
