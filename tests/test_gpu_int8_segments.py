"""Split-INT8 and BF16x3 contractions whose K runs as segments over CTAs, the last of which to
arrive adds them up: every pass over alternating inputs gives the bits of the first pass over
the same inputs."""
import numpy as np
import pytest

import tamm_b200 as tb

pytestmark = pytest.mark.gpu


def _space(sizes):
    return tb.TiledIndexSpace(tb.IndexSpace(sum(sizes)), sizes)


@pytest.mark.parametrize("mode", ["INT8", "BF16X3"])
@pytest.mark.parametrize("rows,cols,ktiles", [([20, 33], [20], [20000, 9000, 300]), ([200], [150, 7], [4096] * 9)])
def test_every_pass_has_the_first_ones_bits(mode, rows, cols, ktiles):
    ec = tb.ExecutionContext(0, 1 << 30)
    ec.set_precision(getattr(tb.Precision, mode), 1e-11)
    M, N, K = _space(rows), _space(cols), _space(ktiles)
    m, n, k = M.label(), N.label(), K.label()
    rng = np.random.default_rng(7)
    C = tb.Tensor([M, N]).allocate(ec)
    ops = []
    for _ in range(2):
        A, B = tb.Tensor([M, K]).allocate(ec), tb.Tensor([K, N]).allocate(ec)
        A.write(rng.normal(size=A.nelems))
        B.write(rng.normal(size=B.nelems))
        ops.append((tb.Scheduler(ec), C(m, n).assign(A(m, k) * B(k, n)), A, B))
    first = [None, None]
    for i in range(200):
        sch, op, A, B = ops[i % 2]
        sch(op).execute(tb.ExecutionHW.GPU)
        got = C.read()
        if first[i % 2] is None:
            first[i % 2] = got
        assert np.array_equal(got, first[i % 2])
    for (_, _, A, B), got in zip(ops, first):  # and they are the products
        at = [0, *np.cumsum(ktiles)]
        a, b = A.read(), B.read()
        nr, nc, blocks, p = sum(rows), sum(cols), [], 0
        ad, bd = np.zeros((nr, sum(ktiles))), np.zeros((sum(ktiles), nc))
        for r0, r in zip(np.cumsum([0] + rows), rows):
            for k0, kn in zip(at, ktiles):
                ad[r0:r0 + r, k0:k0 + kn] = a[p:p + r * kn].reshape(r, kn)
                p += r * kn
        p = 0
        for k0, kn in zip(at, ktiles):
            for c0, c in zip(np.cumsum([0] + cols), cols):
                bd[k0:k0 + kn, c0:c0 + c] = b[p:p + kn * c].reshape(kn, c)
                p += kn * c
        want = ad @ bd
        for r0, r in zip(np.cumsum([0] + rows), rows):
            for c0, c in zip(np.cumsum([0] + cols), cols):
                blocks.append(want[r0:r0 + r, c0:c0 + c].ravel())
        bar = 1e-11 if mode == "INT8" else 5e-5  # the modes' stated bars, of max |a| max |b| K
        assert np.max(np.abs(got - np.concatenate(blocks))) <= bar * np.abs(a).max() * np.abs(b).max() * sum(ktiles)
    ec.close()
