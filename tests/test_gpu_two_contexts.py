"""A scheduler of one context over tensors of another: the device tables of its contractions
belong to the scheduler's stream and do not wait behind, or race with, what the tensors' own
context has queued."""
import numpy as np
import pytest

import tamm_b200 as tb

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", ["FP64", "INT8"])
def test_tables_on_the_schedulers_stream(mode):
    mine, other = tb.ExecutionContext(0, 1 << 29), tb.ExecutionContext(0, 1 << 28)
    other.set_precision(getattr(tb.Precision, mode), 1e-11)
    big, S = tb.TiledIndexSpace(tb.IndexSpace(2000), 500), tb.TiledIndexSpace(tb.IndexSpace(150), [70, 80])
    P, Q, R = (tb.Tensor([big, big]).allocate(mine) for _ in range(3))
    A, B, C = (tb.Tensor([S, S]).allocate(mine) for _ in range(3))
    rng = np.random.default_rng(1)
    P.fill_random(1, 0, -1.0, 1.0)
    Q.fill_random(2, 0, -1.0, 1.0)
    a, b = rng.normal(size=(150, 150)), rng.normal(size=(150, 150))
    cut = [slice(0, 70), slice(70, 150)]
    pack = lambda x: np.concatenate([x[p, q].ravel() for p in cut for q in cut])  # noqa: E731
    A.write(pack(a))
    B.write(pack(b))
    i, j, k = S.labels(3)
    x, y, z = big.labels(3)
    busy = tb.Scheduler(mine)
    for _ in range(30):
        busy(R(x, y).iadd(P(x, z) * Q(z, y)))
    busy.execute_async()  # about 15 ms on the tensors' own stream
    got = []
    for _ in range(3):
        sch = tb.Scheduler(other)
        sch(C(i, j).assign(A(i, k) * B(k, j))).execute(tb.ExecutionHW.GPU)
        got.append(sch)
    busy.wait()
    assert np.max(np.abs(C.read() - pack(a @ b))) <= 1e-11 * np.abs(a).max() * np.abs(b).max() * 150
    del got
    for t in (P, Q, R, A, B, C):
        t.deallocate()
    other.close()
    mine.close()
