"""Large query batches, which are sorted by position before they run: every
answer equals the one the same queries get in batches too small to be sorted
(the plain route, checked against the oracle in test_gpu_tree.py and
test_gpu_range.py).  Positions at and past the ends of the sequence included."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

N, L, NQ, SMALL = (1 << 26) + 3, 20, (5 << 19) + 5, 1 << 19  # 168 MB of bits; SMALL is never sorted


@pytest.fixture(scope="module")
def setup(wtg):
    torch = pytest.importorskip("torch")
    g = torch.Generator(device="cuda")
    g.manual_seed(11)
    x = torch.empty(N, device="cuda").exponential_(2.0 ** -14, generator=g).floor_().clamp_(max=2 ** 20 - 1)
    seq = x.to(torch.int32)
    t = wtg.WaveletTree.from_device(seq.data_ptr(), N, 4, L, wtg.ALL, torch.cuda.current_stream().cuda_stream)
    t.sync()
    idx = torch.randint(0, N, (NQ,), device="cuda", generator=g)
    idx[:6] = torch.tensor([0, N - 1, N, N + 1, 1 << 40, -1], device="cuda")  # -1: 2^64 - 1
    sym = seq[torch.randint(0, N, (NQ,), device="cuda", generator=g)].long()
    sym[6:10] = torch.tensor([0, 2 ** 20 - 1, 2 ** 20, 1 << 40], device="cuda")
    end = torch.where((idx >= 0) & (idx < N), torch.clamp(idx + 5000, max=N), idx)
    return torch, t, seq, idx, sym, end


def _both(torch, nout, call):
    """call(at, m, outs) over the whole batch and over small pieces of it."""
    got = [torch.empty(NQ, dtype=torch.int64, device="cuda") for _ in range(nout)]
    exp = [torch.empty(NQ, dtype=torch.int64, device="cuda") for _ in range(nout)]
    call(0, NQ, [o.data_ptr() for o in got])
    for at in range(0, NQ, SMALL):
        call(at, min(SMALL, NQ - at), [o.data_ptr() + 8 * at for o in exp])
    torch.cuda.synchronize()
    for a, b in zip(got, exp):
        assert torch.equal(a, b)
    return got


def test_access(setup):
    torch, t, seq, idx, sym, end = setup
    st = torch.cuda.current_stream().cuda_stream
    got = _both(torch, 1, lambda at, m, o: t.access_device(idx.data_ptr() + 8 * at, m, o[0], st))[0]
    ok = (idx >= 0) & (idx < N)
    assert torch.equal(got[ok], seq[idx[ok]].long()) and bool((got[~ok] == -1).all())


def test_rank(setup):
    torch, t, seq, idx, sym, end = setup
    st = torch.cuda.current_stream().cuda_stream
    _both(torch, 1, lambda at, m, o: t.rank_device(idx.data_ptr() + 8 * at, sym.data_ptr() + 8 * at, m, o[0], st))


def test_lex_count_and_range_count(setup):
    torch, t, seq, idx, sym, end = setup
    st = torch.cuda.current_stream().cuda_stream
    p = [x.data_ptr() for x in (idx, end, sym)]
    _both(torch, 3, lambda at, m, o: t.lex_count_device(p[0] + 8 * at, p[1] + 8 * at, p[2] + 8 * at, m, *o, st))
    last, hi = torch.clamp(end - 1, min=0), sym + 100
    r = [x.data_ptr() for x in (idx, last, sym, hi)]
    _both(torch, 1, lambda at, m, o: t.range_count_device(r[0] + 8 * at, r[1] + 8 * at, r[2] + 8 * at, r[3] + 8 * at,
                                                          m, o[0], st))


def test_inverse_select_from_host_arrays(setup):
    torch, t, seq, idx, sym, end = setup
    i = idx.cpu().numpy().view(np.uint64)
    r, c = t.inverse_select(i)
    parts = [t.inverse_select(i[a:a + SMALL]) for a in range(0, NQ, SMALL)]
    assert np.array_equal(r, np.concatenate([p[0] for p in parts]))
    assert np.array_equal(c, np.concatenate([p[1] for p in parts]))


@pytest.mark.parametrize("m", [(1 << 20) + 1, NQ])  # sorted over the two tables, and over the blocks
def test_batches_with_and_without_blocks(setup, m):
    torch, t, seq, idx, sym, end = setup
    st = torch.cuda.current_stream().cuda_stream
    i, c = idx[-m:], sym[-m:]
    got = torch.empty((2, m), dtype=torch.int64, device="cuda")
    exp = torch.empty((2, m), dtype=torch.int64, device="cuda")
    for out, piece in ((got, m), (exp, SMALL)):
        for at in range(0, m, piece):
            k = min(piece, m - at)
            t.access_device(i.data_ptr() + 8 * at, k, out[0].data_ptr() + 8 * at, st)
            t.rank_device(i.data_ptr() + 8 * at, c.data_ptr() + 8 * at, k, out[1].data_ptr() + 8 * at, st)
    torch.cuda.synchronize()
    assert torch.equal(got, exp)
