"""Device tables of short-lived schedulers (work lists, split layouts, segment, add and
denominator lists): made and dropped in the order of the context's stream without waiting
for the device, so a table's memory may be handed on while the work that reads it is still
queued, and the pinned buffer they are filled through (8 MB) is reused.  Every scheduler must
give the first one's bits, before and after a graph captured in between, also when the
schedulers outlive one another."""
import numpy as np
import pytest

import tamm_b200 as tb
from tamm_b200 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", ["FP64", "INT8"])
def test_short_lived_schedulers(mode):
    ec = tb.ExecutionContext(0, 1 << 31)
    ec.set_precision(getattr(tb.Precision, mode), 1e-11)
    MO = W.mo_tiled(24, 36, [8] * 3, [9] * 4)
    O, V = MO("occ"), MO("virt")
    R, X, Y = (tb.Tensor([V, V, O, O], spin=(2, 2)).allocate(ec) for _ in range(3))
    Z = tb.Tensor([O, O, O, O], spin=(2, 2)).allocate(ec)
    rng = np.random.default_rng(3)
    X.write(rng.normal(size=X.nelems))
    Z.write(rng.normal(size=Z.nelems))
    (a, b), (i, j, k, l) = V.labels(2), O.labels(4)

    def queue(sch):
        sch(R(a, b, i, j).assign(0.5 * X(a, b, k, l) * Z(k, l, i, j)))
        sch(Y(a, b, i, j).assign(R(a, b, i, j)))
        sch(Y(a, b, i, j).isub(R(b, a, i, j)))
        return sch

    first, kept, graph = None, [], None
    for n in range(60):
        sch = queue(tb.Scheduler(ec))
        if n == 20:
            graph = (sch, sch.graph())
            graph[1].launch()
        else:
            sch.execute(tb.ExecutionHW.GPU)
        if n % 7 == 0:
            kept.append(sch)
        if n in (0, 1, 19, 20, 21, 40, 59):
            got = Y.read()
            first = got if first is None else first
            assert np.array_equal(got, first)
    X.write(2.0 * X.read())
    del kept
    graph[1].launch().sync()
    assert np.array_equal(Y.read(), 2.0 * first)
