"""Which kernel a split-INT8 contraction over a built tensor runs on follows the whole tensor, not
its batches: any batch size gives the bits of one batch, and those are an FP64 request's where
the contraction uses its operands only a few times."""
import numpy as np
import pytest

import tamm_b200 as tb

pytestmark = pytest.mark.gpu


# a tensor of 2^20 elements and more whose batches have fewer, times 24 columns (few uses); 160
# rows by 400 columns, not few, in batches of 8 rows, which would be
@pytest.mark.parametrize("rows,tile,k,n,fp64", [(32400, 8100, 33, 24, True), (160, 8, 3000, 400, False)])
def test_batches_run_on_the_kernel_of_the_whole(rows, tile, k, n, fp64):
    ec = tb.ExecutionContext(0, 1 << 30)
    M, K, N = (tb.TiledIndexSpace(tb.IndexSpace(x), y) for x, y in ((rows, tile), (k, k), (n, n)))
    X, F, C = (tb.Tensor(s).allocate(ec) for s in ([M, K], [K, N], [M, N]))
    rng = np.random.default_rng(2)
    for t in (X, F):
        t.write(rng.normal(size=t.nelems))
    m, q, p = M.label(), K.label(), N.label()

    def build(batch, first, last, sch):
        mp, qp = batch.spaces[0].label(), K.label()
        sch(batch(mp, qp).assign(X(mp, qp)))

    def run(mode, batch_bytes):
        ec.set_precision(mode, 1e-11)
        L = tb.Tensor.built([M, K], build, batch_bytes=batch_bytes)
        sch = tb.Scheduler(ec)
        sch(C(m, p).assign(L(m, q) * F(q, p))).execute(tb.ExecutionHW.GPU)
        return C.read()

    whole, one = (run(tb.Precision.INT8, b) for b in (8 * rows * k, 8 * tile * k))
    assert np.array_equal(whole, one)
    assert np.array_equal(whole, run(tb.Precision.FP64, 8 * rows * k)) == fp64
    for t in (X, F, C):
        t.deallocate()
    ec.close()
