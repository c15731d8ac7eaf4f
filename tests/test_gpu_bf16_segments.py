"""BF16x3 contractions whose output block is a few tiles with a long K are cut between tasks
only: rows of a small block (which is cut) have the bits of the same rows in a block of more
tiles (which is not), for one task of a long K and for several."""
import numpy as np
import pytest

import tamm_b200 as tb

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ktiles", [[20000], [9000, 9100, 33], [8192, 8192]])
def test_rows_do_not_depend_on_the_cut(ktiles):
    ec = tb.ExecutionContext(0, 1 << 31)
    ec.set_precision(tb.Precision.BF16X3)
    K, N = tb.TiledIndexSpace(tb.IndexSpace(sum(ktiles)), ktiles), tb.TiledIndexSpace(tb.IndexSpace(48), 48)
    rng = np.random.default_rng(5)
    a, b = rng.normal(size=(1152, sum(ktiles))), rng.normal(size=(sum(ktiles), 48))
    cuts = np.cumsum([0] + ktiles)
    k, n = K.label(), N.label()
    B = tb.Tensor([K, N]).allocate(ec)
    B.write(np.concatenate([b[p:q].ravel() for p, q in zip(cuts, cuts[1:])]))
    got = {}
    for rows in (128, 1152):
        M = tb.TiledIndexSpace(tb.IndexSpace(rows), rows)
        m = M.label()
        A, C = tb.Tensor([M, K]).allocate(ec), tb.Tensor([M, N]).allocate(ec)
        A.write(np.concatenate([a[:rows, p:q].ravel() for p, q in zip(cuts, cuts[1:])]))
        sch = tb.Scheduler(ec)
        sch(C(m, n).assign(A(m, k) * B(k, n)))
        sch.execute(tb.ExecutionHW.GPU)
        got[rows] = C.read().reshape(rows, 48)
    # one task: the same sums; several: only the order of the FP64 sums over tasks differs
    mag = np.abs(a[:128]) @ np.abs(b)
    bound = 0.0 if len(ktiles) == 1 else len(ktiles) * 2.0 ** -52 * mag.max()
    assert np.max(np.abs(got[128] - got[1152][:128])) <= bound
