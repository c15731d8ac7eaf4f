"""Statistics of split-INT8 requests that run on the FP64 kernel: its mode and its time, no
digits, for a stored and for a built operand."""
import pytest

import tamm_b200 as tb

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("built", [False, True])
@pytest.mark.parametrize("n,mode", [(24, tb.Precision.FP64), (400, tb.Precision.INT8)])
def test_mode_that_ran(built, n, mode):
    ec = tb.ExecutionContext(0, 1 << 30)
    ec.set_precision(tb.Precision.INT8, 1e-11)
    M, K, N = (tb.TiledIndexSpace(tb.IndexSpace(x), y) for x, y in ((4000, 2000), (300, 300), (n, n)))
    X, F, C = (tb.Tensor(s).allocate(ec) for s in ([M, K], [K, N], [M, N]))
    X.fill_random(1, 0, -1.0, 1.0)
    F.fill_random(2, 0, -1.0, 1.0)
    m, k, p = M.label(), K.label(), N.label()

    def build(batch, first, last, sch):
        mp, kp = batch.spaces[0].label(), K.label()
        sch(batch(mp, kp).assign(X(mp, kp)))

    L = tb.Tensor.built([M, K], build, batch_bytes=8 * 2000 * 300) if built else X
    sch = tb.Scheduler(ec)
    sch(C(m, p).iadd(L(m, k) * F(k, p))).execute(tb.ExecutionHW.GPU, True)
    st = sch.op_stats(-1)
    assert st["mode"] == mode and st["gemm_ms"] > 0
    assert (st["slices_max"] == 0 and st["split_ms"] == 0) == (mode == tb.Precision.FP64)
    for t in (X, F, C):
        t.deallocate()
    ec.close()
