"""Ops that the scheduler must not run in one pass although they look alike: adds over tensors
attached to one buffer, where each op reads what the one before it wrote."""
import numpy as np
import pytest

import tamm_b200 as tb

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("labels", ["ab", "ba"])
def test_adds_over_one_buffer(labels):
    """R += p X, R += q X with R and X in the same memory: (1 + p)(1 + q) x."""
    torch = pytest.importorskip("torch")
    ec = tb.ExecutionContext(0, 1 << 28)
    S = tb.TiledIndexSpace(tb.IndexSpace(60), [20, 30, 10])
    R, X = tb.Tensor([S, S]), tb.Tensor([S, S])
    rng = np.random.default_rng(3)
    x0 = rng.normal(size=R.nelems)
    buf = torch.from_numpy(x0).cuda()
    for t in (R, X):
        t.attach(ec, buf.data_ptr(), buf.numel() * 8)
    torch.cuda.synchronize()
    a, b = S.labels(2)
    l, m = (a, b) if labels == "ab" else (b, a)  # the same order on both sides: element by element
    for profile in (False, True):
        buf.copy_(torch.from_numpy(x0))
        torch.cuda.synchronize()
        sch = tb.Scheduler(ec)
        sch(R(l, m).iadd(0.5 * X(l, m)))(R(l, m).iadd(0.25 * X(l, m)))(R(l, m).isub(2.0 * X(l, m)))
        sch.execute(tb.ExecutionHW.GPU, profile)
        assert np.array_equal(buf.cpu().numpy(), ((x0 * 1.5) * 1.25) * -1.0)
    for t in (R, X):
        t.deallocate()
    ec.close()


def test_dots_before_a_refused_update():
    """The update of a read-only tensor is refused; the dots queued before it have run."""
    ec = tb.ExecutionContext(0, 1 << 28)
    S = tb.TiledIndexSpace(tb.IndexSpace(50), [20, 30])
    t, r = (tb.Tensor([S, S]).allocate(ec) for _ in range(2))
    rng = np.random.default_rng(4)
    tv, rv = rng.integers(-8, 8, size=(2, t.nelems)).astype(float)
    t.write(tv)
    r.write(rv)
    t.set_read_only(True)
    lab = S.labels(2)
    sch = tb.Scheduler(ec)
    sch.dot(0, t(*lab), r(*lab))
    sch.dot(1, r(*lab), r(*lab), 0.5)
    sch.denom(t(*lab), -1.0, r(*lab), np.ones(50), [1, 1])
    with pytest.raises(tb.TambError):
        sch.execute(tb.ExecutionHW.GPU)
    assert [float(x) for x in sch.scalars(2)] == [tv @ rv, 0.5 * (rv @ rv)]  # sums of small integers: exact
    t.set_read_only(False)
    sch.execute(tb.ExecutionHW.GPU)  # the ops are still queued
    assert np.max(np.abs(t.read() - (tv - rv / 2.0))) <= 1e-14
    for x in (t, r):
        x.deallocate()
    ec.close()
