"""Split-INT8 contractions that use each element of the larger operand only a few times run
on the FP64 kernel: the bits of an FP64 request on one side of every condition of that
rule, other bits on the other side, and within the split mode's error bound throughout."""
import numpy as np
import pytest

import tamm_b200 as tb

pytestmark = pytest.mark.gpu


def _space(n, t):
    return tb.TiledIndexSpace(tb.IndexSpace(n), t)


@pytest.mark.parametrize("kind,n,target,slices,read_only,fp64", [
    ("dress", 24, 1e-11, 0, False, True), ("dress", 24, 1e-11, 0, True, False), ("dress", 24, 1e-6, 0, False, False),
    ("dress", 24, 1e-11, 6, False, False), ("dress", 80, 1e-11, 0, False, True), ("dress", 88, 1e-11, 0, False, False),
    ("small", 24, 1e-11, 0, False, False), ("strided", 24, 1e-11, 0, False, False)])
def test_route(kind, n, target, slices, read_only, fp64):
    ec = tb.ExecutionContext(0, 1 << 31).set_digit_cache(1 << 29)
    N, K, V = _space(n, 24), _space(33, 33), _space(170 if kind == "small" else 180, 45)
    (p, k), (a, b) = (N.label(), K.label()), V.labels(2)
    C = tb.Tensor([V, V, N]).allocate(ec)
    X = tb.Tensor([V, V, K]).allocate(ec)
    F = tb.Tensor([K, N]).allocate(ec)
    rhs = X(a, b, k) * F(k, p)
    if kind == "strided":  # B = [N, k, q] with the K order (k, q) of A as (q, k): k is last in B, first in A
        Q = _space(2, 2)
        q = Q.label()
        X, F = tb.Tensor([V, V, K, Q]).allocate(ec), tb.Tensor([N, Q, K]).allocate(ec)
        rhs = X(a, b, k, q) * F(p, q, k)
    rng = np.random.default_rng(1)
    for t in (X, F):
        t.write(rng.normal(size=t.nelems))
    X.set_read_only(read_only)
    got = {}
    for mode in (tb.Precision.INT8, tb.Precision.FP64):
        ec.set_precision(mode, target, slices)
        sch = tb.Scheduler(ec)
        sch(C(a, b, p).assign(rhs))
        sch.execute(tb.ExecutionHW.GPU)
        got[mode] = C.read()
    i8, f8 = got[tb.Precision.INT8], got[tb.Precision.FP64]
    assert np.array_equal(i8, f8) == fp64
    assert np.max(np.abs(i8 - f8)) <= 10 * target * np.max(np.abs(f8))
    X.set_read_only(False)
