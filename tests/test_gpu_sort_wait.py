"""A look-back wait that runs out inside the sort of a query batch (tile 0 of its
first pass is never taken): the batch ends, nothing outside the caller's arrays
is written, the next check reports the timeout, and after a rebuild the same
batch is right.  Made on the host: no kernel waits without a limit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

N, L, NQ, PAD, MARK = (1 << 25) + 3, 20, (1 << 21) + 5, 1 << 16, -77


class _Setup:
    def __init__(self, wtg, torch):
        self.wtg, self.torch = wtg, torch
        g = torch.Generator(device="cuda")
        g.manual_seed(3)
        self.st = torch.cuda.current_stream().cuda_stream
        self.seq = torch.randint(0, 1 << L, (N,), device="cuda", generator=g, dtype=torch.int32)
        self.idx = torch.randint(0, N, (NQ,), device="cuda", generator=g)
        self.sym = self.seq[torch.randint(0, N, (NQ,), device="cuda", generator=g)].long()
        self.end = torch.clamp(self.idx + 1000, max=N - 1)
        self.bytes = torch.randint(1, 200, (1 << 18,), device="cuda", generator=g).to(torch.uint8)
        self.C = torch.zeros(256, dtype=torch.int64, device="cuda")
        self.C[1:] = torch.cumsum(torch.bincount(self.bytes.int(), minlength=256), 0)[:-1]
        self.off = torch.zeros(NQ + 1, dtype=torch.int64, device="cuda")  # lengths that are worth sorting
        self.off[1:] = torch.cumsum(torch.randint(1, 14, (NQ,), device="cuda", generator=g), 0)
        self.pat = self.bytes[torch.randint(0, 1 << 18, (int(self.off[-1]),), device="cuda", generator=g)].contiguous()
        torch.cuda.synchronize()


@pytest.fixture(scope="module")
def s(wtg):
    return _Setup(wtg, pytest.importorskip("torch"))


def _tree(s, old=None):
    t = s.wtg.WaveletTree.from_device(s.seq.data_ptr(), N, 4, L, s.wtg.ALL, s.st, tree=old)
    t.sync()
    return t


def _fm(s, old=None):
    t = s.wtg.WaveletTree.from_device(s.bytes.data_ptr(), s.bytes.numel(), 1, 8, s.wtg.ALL, s.st, tree=old)
    t.sync()
    return t


def _run(s, what, t, o):
    d = [x.data_ptr() for x in (s.idx, s.sym, s.end)]
    if what == "access":
        t.access_device(d[0], NQ, o[0], s.st)
    elif what == "rank":
        t.rank_device(d[0], d[1], NQ, o[0], s.st)
    elif what == "lex_count":
        t.lex_count_device(d[0], d[2], d[1], NQ, *o, s.st)
    elif what == "range_count":
        t.range_count_device(d[0], d[2], d[1], d[1], NQ, o[0], s.st)
    else:
        s.wtg._ck(s.wtg.lib().wtg_fm_count_device(t.h, s.C.data_ptr(), 200, s.pat.data_ptr(), s.off.data_ptr(), NQ,
                                                  o[0], s.st))


def _outputs(s, k):
    return [s.torch.full((NQ + 2 * PAD,), MARK, dtype=s.torch.int64, device="cuda") for _ in range(k)]


@pytest.mark.parametrize("what", ["access", "rank", "lex_count", "range_count", "fm_count"])
def test_batch(s, what):
    torch, wtg = s.torch, s.wtg
    make, k = (_fm if what == "fm_count" else _tree), 3 if what == "lex_count" else 1
    t = make(s)
    exp = _outputs(s, k)
    _run(s, what, t, [o.data_ptr() + 8 * PAD for o in exp])
    t.sync()
    got = _outputs(s, k)
    torch.cuda.synchronize()
    wtg.set_wait_limits(lookback_spins=2000)
    try:
        wtg.inject_lookback_stall(True)
        _run(s, what, t, [o.data_ptr() + 8 * PAD for o in got])
        for _ in range(2):
            with pytest.raises(wtg.WtgError) as e:
                t.sync()
            assert e.value.code == wtg.ERR_TIMEOUT
    finally:
        wtg.inject_lookback_stall(False)
        wtg.set_wait_limits(0, 0)
    for o in got:
        assert bool((o[:PAD] == MARK).all()) and bool((o[NQ + PAD:] == MARK).all())
    t = make(s, t)
    got = _outputs(s, k)
    _run(s, what, t, [o.data_ptr() + 8 * PAD for o in got])
    t.sync()
    for a, b in zip(got, exp):
        assert torch.equal(a, b)
    t.free()


def test_host_query_and_huffman_counts(s):
    torch, wtg = s.torch, s.wtg
    idx = s.idx.cpu().numpy().astype(np.uint64)
    t = _tree(s)
    exp = t.inverse_select(idx)
    h = wtg.HuffmanTree.from_device(s.bytes.data_ptr(), s.bytes.numel(), wtg.ALL, s.st)
    C, pat, off = (x.cpu().numpy() for x in (s.C, s.pat, s.off))
    counts = h.fm_count(C, pat, off)
    wtg.set_wait_limits(lookback_spins=2000)
    try:
        for call in (lambda: t.inverse_select(idx), lambda: h.fm_count(C, pat, off)):
            wtg.inject_lookback_stall(True)
            with pytest.raises(wtg.WtgError) as e:
                call()
            assert e.value.code == wtg.ERR_TIMEOUT
    finally:
        wtg.inject_lookback_stall(False)
        wtg.set_wait_limits(0, 0)
    h.free()
    t = _tree(s, t)
    assert all(np.array_equal(a, b) for a, b in zip(t.inverse_select(idx), exp))
    h = wtg.HuffmanTree.from_device(s.bytes.data_ptr(), s.bytes.numel(), wtg.ALL, s.st)
    assert np.array_equal(h.fm_count(C, pat, off), counts)
    h.free()
    t.free()
