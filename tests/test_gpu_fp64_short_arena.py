"""FP64 contractions in an arena that cannot hold the accumulators of tiles spread over CTAs: the
tiles run whole and close their K segments, with the bits of the spread ones - a few tiles, and
more items than CTAs, where a CTA passes over the items it has nothing to do for."""
import pytest

import tamm_b200 as tb

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def _run(arena, ni, nj, kt, graph):
    ec = tb.ExecutionContext(0, arena)
    I, J, K = (tb.TiledIndexSpace(tb.IndexSpace(n * t), t) for n, t in ((ni, 130), (nj, 90), kt))
    i, j, k = I.label(), J.label(), K.label()
    mem, T = [], []
    for seed, sp in ((1, [I, K]), (2, [K, J]), (None, [I, J])):
        t = tb.Tensor(sp)
        x = torch.zeros(t.nelems, dtype=torch.float64, device="cuda")
        if seed is not None:
            x.normal_(generator=torch.Generator(device="cuda").manual_seed(seed))
        t.attach(ec, x.data_ptr(), x.numel() * 8)
        mem.append(x)
        T.append(t)
    torch.cuda.synchronize()
    sch = tb.Scheduler(ec)
    sch(T[2](i, j).assign(T[0](i, k) * T[1](k, j)))
    if graph:
        g = sch.graph()
        mem[2].fill_(7.0)
        torch.cuda.synchronize()
        g.launch().sync()
        del g
    else:
        sch.execute(tb.ExecutionHW.GPU)
    for t in T:
        t.deallocate()
    del sch
    ec.close()
    return mem


@pytest.mark.parametrize("graph", [False, True])
@pytest.mark.parametrize("ni,nj,kt", [(1, 1, (3, 6000)), (2, 3, (5, 1111)), (24, 12, (3, 1500)), (12, 11, (2, 2100))])
def test_same_bits(ni, nj, kt, graph):
    a, b, want = _run(1 << 29, ni, nj, kt, graph)
    *_, got = _run(1 << 12, ni, nj, kt, graph)
    assert torch.equal(got, want)
    K, n = kt[0] * kt[1], kt[1]
    first = sum(a[p * 130 * n:(p + 1) * 130 * n].view(130, n) @ b[p * nj * 90 * n:][:90 * n].view(n, 90)
                for p in range(kt[0]))  # the first output block, in 64 bits
    mag = sum(a[p * 130 * n:(p + 1) * 130 * n].view(130, n).abs() @ b[p * nj * 90 * n:][:90 * n].view(n, 90).abs()
              for p in range(kt[0]))
    assert bool(((want[:130 * 90].view(130, 90) - first).abs() <= 2 * K * 2.0 ** -53 * mag).all())
