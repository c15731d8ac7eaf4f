"""A captured graph keeps the device tables its kernels read: its replays give the eager run's bits
after the scheduler has released its caches, run other ops, and other schedulers have made and
dropped tables of the same sizes."""
import numpy as np
import pytest

import tamm_b200 as tb
from tamm_b200 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", ["FP64", "INT8"])
def test_replay_after_release(mode):
    ec = tb.ExecutionContext(0, 1 << 30)
    ec.set_precision(getattr(tb.Precision, mode), 1e-11)
    MO = W.mo_tiled(12, 20, [5, 7], [9, 4, 7])
    O, V = MO("occ"), MO("virt")
    spin = dict(spin=(2, 2))
    X, R, Y, D = (tb.Tensor([V, V, O, O], **spin).allocate(ec) for _ in range(4))
    Z = tb.Tensor([O, O, O, O], **spin).allocate(ec)
    F = tb.Tensor([O, O], spin=(1, 1)).allocate(ec)
    G = tb.Tensor([V, V, V, V], **spin).allocate(ec)
    rng = np.random.default_rng(3)
    start = {t: rng.normal(size=t.nelems) for t in (X, Z, Y)}
    eps = np.concatenate([-1.0 - rng.random(24), 1.0 + rng.random(40)])
    (a, b, c, d), (i, j, k, l) = V.labels(4), O.labels(4)
    av = V.sub(0, 2).label()

    def reset():
        for t, v in start.items():
            t.write(v)
        for t in (R, D, F):
            t.write(np.full(t.nelems, 3.0))

    def queue(sch):
        sch(R(a, b, i, j).assign(0.5 * X(a, b, k, l) * Z(k, l, i, j)))  # store, and the fill of blocks without tasks
        sch(F(i, j).assign(X(a, b, i, k) * X(a, b, j, k)))              # K in segments
        sch(D(a, b, i, j).assign(R(a, b, i, j)))                        # a run of adds
        sch(D(a, b, i, j).isub(R(b, a, i, j)))
        sch(D(av, b, i, j).iadd(2.0 * X(b, av, i, j)))                  # a permuted add, over some tiles
        sch(D(av, b, i, j).iadd(0.25))                                  # a fill of some blocks
        sch.dot(0, X(a, b, i, j), Y(a, b, i, j), 0.25)                  # dots and an update in one kernel
        sch.norm(1, D(a, b, i, j))
        sch.denom(Y(a, b, i, j), -1.0, D(a, b, i, j), eps, [1, 1, -1, -1])
        sch.set_scalar(2, 0.0)
        sch.denom_energy(2, 1.0, R(a, b, i, j), eps, [1, 1, -1, -1])
        sch.mult_energy(2, 1.0, R(a, b, i, j).iadd(0.5 * X(a, b, k, l) * Z(k, l, i, j)), eps, [1, 1, -1, -1])
        return sch

    def state(sch):
        return [t.read() for t in (R, F, D, Y)] + [np.array([float(x) for x in sch.scalars(3)])]

    sch = queue(tb.Scheduler(ec))
    reset()
    graph = sch.graph()
    reset()
    graph.launch().sync()
    want = state(sch)
    G.fill_random(5, 0, -1.0, 1.0)
    for n in range(12):
        if n % 3 == 0:
            sch.release()
        other = queue(tb.Scheduler(ec)) if n % 2 else tb.Scheduler(ec)
        other(G(a, b, c, d).iadd(0.1 * G(b, a, c, d)))(G(a, b, c, d).isub(0.1 * G(a, b, d, c)))
        other(G(av, b, c, d).assign(1.0 * n))
        other.execute(tb.ExecutionHW.GPU)
        if n % 4 == 1:  # other ops on the graph's own scheduler
            sch(G(a, b, c, d).assign(0.5 * G(a, b, c, d))).execute(tb.ExecutionHW.GPU)
        del other
        reset()
        graph.launch().sync()
        for got, w in zip(state(sch), want):
            assert np.array_equal(got, w)
    del graph
    for t in (X, R, Y, D, Z, F, G):
        t.deallocate()
    del sch
    ec.close()
