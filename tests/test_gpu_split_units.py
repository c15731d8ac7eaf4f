"""The digit split of the tensor-core modes over operand layouts and sizes where its work
units end: K contiguous, rows contiguous, neither (a middle label), K at the edges of a
16-element core matrix, a 32-byte step, the staged kernel's shortest row (128) and the
longest row of a unit (beyond it: segments), row counts at the edges of 8-row groups and of
the 80- and 128-row tiles, rows of zeros and rows scaled far from one.

One block triple through tb_block_multiply against numpy, per row of C: split-INT8 within
1e-11 and BF16x3 within 5e-5 of the row's max |A| max |B| K (the modes' stated bars; each
row of A has a scale of its own, so a row is its own unit of error)."""
import ctypes as C

import numpy as np
import pytest

from tamm_b200 import _capi as A

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

LAYOUTS = [("amkl", "klnb"), ("klam", "nbkl"), ("kalm", "nkbl"), ("alkm", "nlkb")]
SHAPES = [  # a, m, n, b, k, l
    (1, 1, 1, 1, 1, 1), (1, 7, 9, 1, 3, 5), (3, 43, 8, 10, 4, 8), (2, 64, 9, 9, 3, 11), (1, 129, 81, 1, 127, 1),
    (5, 26, 4, 20, 16, 8), (1, 40, 2, 41, 43, 3), (2, 17, 3, 27, 31, 33), (1, 16, 1, 24, 61, 53), (1, 9, 17, 1, 70, 90)]


@pytest.mark.parametrize("mode,tol", [(A.TB_MODE_INT8, 1e-11), (A.TB_MODE_BF16X3, 5e-5)])
@pytest.mark.parametrize("al,bl", LAYOUTS)
@pytest.mark.parametrize("shape", SHAPES)
def test_layouts_and_edges(mode, tol, al, bl, shape):
    ext = dict(zip("amnbkl", shape))
    lab = {c: -ord(c) for c in "amnbkl"}
    rng = np.random.default_rng(sum(shape) + len(al))
    a = rng.normal(size=[ext[c] for c in "amkl"])
    b = rng.normal(size=[ext[c] for c in "nbkl"])
    scale = 2.0 ** rng.integers(-60, 60, size=shape[:2])
    scale[rng.uniform(size=scale.shape) < 0.1] = 0.0
    a *= scale[:, :, None, None]
    want = np.einsum("amkl,nbkl->amnb", a, b)
    x = np.ascontiguousarray(np.transpose(a, ["amkl".index(c) for c in al]))
    y = np.ascontiguousarray(np.transpose(b, ["nbkl".index(c) for c in bl]))
    keep, arg = [], []
    for v, names in ((x, al), (y, bl), (np.zeros_like(want), "amnb")):
        t = torch.from_numpy(v).cuda()
        d = np.asarray(v.shape, dtype=np.int64)
        l = np.asarray([lab[c] for c in names], dtype=np.int32)
        keep.append((t, d, l))
        arg.append((t.data_ptr(), d.ctypes.data_as(A.i64p), l.ctypes.data_as(A.ip), 4))
    A.call("tb_block_multiply", 1.0, *arg[0], *arg[1], 1.0, *arg[2], 0, mode,
           C.c_void_p(torch.cuda.current_stream().cuda_stream))
    got = keep[2][0].cpu().numpy()
    bound = tol * np.max(np.abs(a), axis=(2, 3)) * np.max(np.abs(b)) * ext["k"] * ext["l"]
    assert np.all(np.abs(got - want) <= bound[:, :, None, None])
