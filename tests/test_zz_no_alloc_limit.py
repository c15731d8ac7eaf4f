"""The largest scratch that tb_block_multiply_int8_noalloc accepts: a block triple that needs the
64 MiB but for a few hundred bytes runs, and the next K step more is refused with its size."""
import ctypes as C

import numpy as np
import pytest

from tamm_b200 import _capi as A

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def _call(a, b, c):
    m, k, n = -1, -2, -3
    arg, keep = [], []
    for t, l in ((a, (m, k)), (b, (k, n)), (c, (m, n))):
        d, x = np.asarray(t.shape, dtype=np.int64), np.asarray(l, dtype=np.int32)
        keep.append((d, x))
        arg.append((t.data_ptr(), d.ctypes.data_as(A.i64p), x.ctypes.data_as(A.ip), 2))
    A.call("tb_block_multiply_int8_noalloc", 1.0, *arg[0], *arg[1], *arg[2], 0,
           C.c_void_p(torch.cuda.current_stream().cuda_stream))
    torch.cuda.synchronize()


def test_limit():
    # 1280 + 16 bytes per 128 x 80 tile, the unit tables, 4 bytes and 6 K bytes per row and column
    M, N, K = 128, 3200, 3360
    assert (64 << 20) - 1024 < 1280 + 16 * 40 + 512 + (4 + 6 * K) * (M + N) <= 64 << 20
    g = torch.Generator(device="cuda").manual_seed(1)
    a, b = (torch.randn(*s, dtype=torch.float64, device="cuda", generator=g) for s in ((M, K), (K, N)))
    c = torch.zeros(M, N, dtype=torch.float64, device="cuda")
    _call(a, b, c)
    assert float((c - a @ b).abs().max()) <= 1e-11 * float(a.abs().max() * b.abs().max()) * K
    a, b = (torch.zeros(*s, dtype=torch.float64, device="cuda") for s in ((M, K + 1), (K + 1, N)))
    with pytest.raises(A.TambError):
        _call(a, b, c)
