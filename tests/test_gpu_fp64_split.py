"""The FP64 contraction kernel where its work is cut: tiles at the edges of both tile
shapes, K at the edges of a chunk (32) and of a segment (64 chunks), operands contiguous
along K or along their outer label, one block triple split over CTAs, and groups whose
segments run in one CTA or in several.

Against numpy's matmul within 1e-12 of max |C| (the plain FP64 bar; the products of K <=
9000 uniform numbers summed in any order differ by less than K eps of sum |a b|, 2e-12 of
which is 1e-12 of max |C| for these positive operands).  Whole and split tiles: bit for
bit, since both sum the same segments in the same order."""
import ctypes as C

import numpy as np
import pytest

import tamm_b200 as tb
from tamm_b200 import _capi as A

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(1, 1, 1), (64, 32, 32), (65, 33, 33), (63, 31, 31), (128, 80, 2048), (129, 81, 2049),
                                   (127, 65, 2047), (16, 16, 9000), (300, 600, 65), (744, 400, 1073)])
@pytest.mark.parametrize("al,bl", [("mk", "kn"), ("km", "nk"), ("mk", "nk"), ("km", "kn")])
def test_block_edges(shape, al, bl):
    ext = dict(zip("mnk", shape))
    lab = {c: -ord(c) for c in "mnk"}
    rng = np.random.default_rng(sum(shape))
    a, b = (rng.uniform(0.5, 1.0, size=[ext[c] for c in x]) for x in (al, bl))
    c = rng.uniform(0.5, 1.0, size=shape[:2])
    want = c + 0.5 * (a if al == "mk" else a.T) @ (b if bl == "kn" else b.T)
    keep, arg = [], []
    for x, names in ((a, al), (b, bl), (c, "mn")):
        t = torch.from_numpy(x).cuda()
        d = np.asarray(x.shape, dtype=np.int64)
        l = np.asarray([lab[y] for y in names], dtype=np.int32)
        keep.append((t, d, l))
        arg.append((t.data_ptr(), d.ctypes.data_as(A.i64p), l.ctypes.data_as(A.ip), 2))
    A.call("tb_block_multiply", 0.5, *arg[0], *arg[1], 1.0, *arg[2], 0, A.TB_MODE_FP64,
           C.c_void_p(torch.cuda.current_stream().cuda_stream))
    got = keep[2][0].cpu().numpy()
    assert np.max(np.abs(got - want)) <= 1e-12 * np.max(np.abs(want))


@pytest.mark.parametrize("ti,tj", [(130, 90), (40, 20)])
def test_segments_whole_and_split(ec, ti, tj):
    """C(i,j) += A(i,k) B(k,j) over three k tiles of 1500 (141 chunks: three segments): the
    whole output, whose first tiles run whole, and one row of blocks, spread over the SMs."""
    ni, nj = (24, 12) if ti == 130 else (40, 30)
    I, J, K = (tb.TiledIndexSpace(tb.IndexSpace(n * t), t) for n, t in ((ni, ti), (nj, tj), (3, 1500)))
    x, y, z, r = (tb.Tensor(s).allocate(ec) for s in ([I, K], [K, J], [I, J], [I, J]))
    x.fill_random(1, 0, 0.5, 1.0)
    y.fill_random(2, 0, 0.5, 1.0)
    (k,), (i,), (j,) = K.labels(1), I.labels(1), J.labels(1)
    sch = tb.Scheduler(ec)
    sch(z().assign(0.0))(z(i, j).iadd(x(i, k) * y(k, j))).execute(tb.ExecutionHW.GPU)
    row = I.sub(2, 3).label()
    sch(r().assign(0.0))(r(row, j).iadd(x(row, k) * y(k, j))).execute(tb.ExecutionHW.GPU)
    xd = np.concatenate([x.get([2, n]) for n in range(3)], axis=1)
    for n in range(nj):
        yd = np.concatenate([y.get([m, n]) for m in range(3)], axis=0)
        want = xd @ yd
        assert np.max(np.abs(z.get([2, n]) - want)) <= 1e-12 * np.max(want)
        assert np.array_equal(r.get([2, n]), z.get([2, n]))
    for t in (x, y, z, r):
        t.deallocate()
