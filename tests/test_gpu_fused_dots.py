"""Dots that the scheduler runs in the kernel of the denominator update behind them: the same
updated bits as one op at a time (a profiled execute runs the ops apart), and scalars within
the rounding of a differently ordered sum, for every choice of operands, one and two dots,
units of few and many rows and long last modes; ops that cannot share the pass stay apart."""
import numpy as np
import pytest

import tamm_b200 as tb
from tamm_b200 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("occ,virt", [([3, 2], [5, 4, 1]), ([20], [33, 7]), ([1, 9], [6]), ([300], [2, 3])])
def test_dots_and_update(ec, occ, virt):
    MO = W.mo_tiled(sum(occ), sum(virt), occ, virt)
    O, V = MO("occ"), MO("virt")
    modes = [V, V, O, O] if sum(occ) < 100 else [V, O]
    spin = (2, 2) if len(modes) == 4 else (1, 1)
    t, r, x, y = (tb.Tensor(modes, spin=spin).allocate(ec) for _ in range(4))
    lab = (*V.labels(2), *O.labels(2)) if len(modes) == 4 else (V.label(), O.label())
    rng = np.random.default_rng(7)
    val = {n: rng.normal(size=t.nelems) for n in "trxy"}
    for u, n in ((r, "r"), (x, "x"), (y, "y")):
        u.write(val[n])
    n = 2 * (sum(occ) + sum(virt))
    eps = np.concatenate([-1.0 - rng.random(n // 2), 1.0 + rng.random(n - n // 2)])
    signs = [1, 1, -1, -1] if len(modes) == 4 else [1, -1]
    T = {"t": t, "r": r, "x": x, "y": y}
    for pairs in ([("x", "t"), ("r", None)], [("t", "r")], [("t", None), ("x", "r")], [("x", "x"), ("x", None)],
                  [("x", "t"), ("y", "t")], [("x", "y")], [("x", "t"), ("r", "r"), ("t", "t")]):
        got = []
        for apart in (False, True):
            t.write(val["t"])
            sch = tb.Scheduler(ec)
            for k, (p, q) in enumerate(pairs):
                if q is None:
                    sch.norm(k, T[p](*lab))
                else:
                    sch.dot(k, T[p](*lab), T[q](*lab), 0.25)
            sch.denom(t(*lab), -1.0, r(*lab), eps, signs)
            sch.execute(tb.ExecutionHW.GPU, apart)
            got.append((t.read(), np.array([float(v) for v in sch.scalars(len(pairs))])))
        assert np.array_equal(got[0][0], got[1][0])
        for k, (p, q) in enumerate(pairs):
            # either order of summation is off by at most nelems * 2^-53 of the sum of magnitudes
            mag = np.abs(val[p] * val[q or p]).sum() * t.nelems * 2.0 ** -52
            a, b = got[0][1][k], got[1][1][k]
            if q is None:
                assert abs(a * a - b * b) <= mag + 4 * 2.0 ** -52 * b * b
            else:
                assert abs(a - b) <= 0.25 * mag
    for u in (t, r, x, y):
        u.deallocate()
