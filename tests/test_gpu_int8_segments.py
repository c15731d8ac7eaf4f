"""Split-INT8 and BF16x3 contractions whose K runs as segments over CTAs, the last of which to
arrive adds them up: every pass over alternating inputs gives the bits of the first pass over
the same inputs, and the segments' sums stay bounded and are no reason to fail."""
import numpy as np
import pytest

import tamm_b200 as tb

pytestmark = pytest.mark.gpu


def _space(sizes):
    return tb.TiledIndexSpace(tb.IndexSpace(sum(sizes)), sizes)


def _dense(flat, rows, cols):
    """A matrix from its packed blocks."""
    out, p = np.zeros((sum(rows), sum(cols))), 0
    for r0, r in zip(np.cumsum([0] + rows), rows):
        for c0, c in zip(np.cumsum([0] + cols), cols):
            out[r0:r0 + r, c0:c0 + c] = flat[p:p + r * c].reshape(r, c)
            p += r * c
    return out


def _check(mode, got, a, b, rows, cols, ktiles):
    """Within the modes' stated bars of max |a| max |b| K."""
    bar = {"INT8": 1e-11, "BF16X3": 5e-5}[mode] * np.abs(a).max() * np.abs(b).max() * sum(ktiles)
    assert np.max(np.abs(_dense(got, rows, cols) - _dense(a, rows, ktiles) @ _dense(b, ktiles, cols))) <= bar


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
        _check(mode, got, A.read(), B.read(), rows, cols, ktiles)
    ec.close()


def _product(mode, arena, tiles, kt, target=1e-11):
    """C(m,n) = A(m,k) B(k,n) over torch storage, so that the arena holds the launch's scratch
    alone; its values and the digits' bytes."""
    torch = pytest.importorskip("torch")
    ec = tb.ExecutionContext(0, arena)
    ec.set_precision(getattr(tb.Precision, mode), target, 6 if mode == "INT8" else 0)
    M, N, K = _space(tiles), _space(tiles), _space(kt)
    m, n, k = M.label(), N.label(), K.label()
    keep, T = [], []
    for seed, sp in ((1, [M, K]), (2, [K, N]), (None, [M, N])):
        t = tb.Tensor(sp)
        x = torch.zeros(t.nelems, dtype=torch.float64, device="cuda")
        if seed is not None:
            x.normal_(generator=torch.Generator(device="cuda").manual_seed(seed))
        t.attach(ec, x.data_ptr(), x.numel() * 8)
        keep.append(x)
        T.append(t)
    torch.cuda.synchronize()
    sch = tb.Scheduler(ec)
    sch(T[2](m, n).assign(T[0](m, k) * T[1](k, n))).execute(tb.ExecutionHW.GPU, True)
    out, scratch = keep[2].cpu().numpy(), sch.op_stats()["scratch_bytes"]
    for t in T:
        t.deallocate()
    ec.close()
    return out, scratch, keep


@pytest.mark.parametrize("mode,kt", [("INT8", [8200]), ("BF16X3", [4100, 4100])])
def test_many_small_blocks_need_no_more_than_their_digits(mode, kt):
    """10000 output blocks of one tile each and a K of 8200: enough tiles for every SM, so none is
    cut (cut in two, their sums alone took 1.6 GB)."""
    out, scratch, (a, b, _) = _product(mode, 3 << 29, [2] * 100, kt)
    assert scratch < 3 << 29
    _check(mode, out, a.cpu().numpy(), b.cpu().numpy(), [2] * 100, [2] * 100, kt)


@pytest.mark.parametrize("mode,kt", [("INT8", [200000]), ("BF16X3", [9000] * 22)])
def test_an_arena_without_room_for_the_segments(mode, kt):
    """Cut tiles' sums that the arena cannot hold beside the digits come from elsewhere: same bits."""
    want, scratch, _ = _product(mode, 1 << 30, [20], kt)
    got, again, _ = _product(mode, scratch + (1 << 18), [20], kt)
    assert again == scratch and np.array_equal(got, want)
