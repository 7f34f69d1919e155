"""Large batches whose scratch has no room (allocation failures injected one after
the other: the sort's pairs, the blocks, the interval table, the step table):
the call goes on without it and the answers are the same, or it reports
WTG_ERR_OOM and works the next time."""
import pytest

pytestmark = pytest.mark.gpu

N, L, NQ = (1 << 26) + 3, 20, (5 << 19) + 5


def _each_failure(wtg, torch, call, out):
    """call() with its k-th allocation failing, for every k that it gets to."""
    call()
    torch.cuda.synchronize()
    exp = out.clone()
    refused = went_on = 0
    for k in range(1, 12):
        out.fill_(-5)
        torch.cuda.synchronize()
        wtg.inject_alloc_failure(k)
        try:
            call()
            torch.cuda.synchronize()
            went_on += 1
            assert torch.equal(out, exp)
        except wtg.WtgError as e:
            refused += 1
            assert e.code == wtg.ERR_OOM
        finally:
            wtg.inject_alloc_failure(0)
    out.fill_(-5)
    call()
    torch.cuda.synchronize()
    assert torch.equal(out, exp)
    return refused, went_on


def test_sorted_batches(wtg):
    torch = pytest.importorskip("torch")
    g = torch.Generator(device="cuda")
    g.manual_seed(1)
    st = torch.cuda.current_stream().cuda_stream
    seq = torch.randint(0, 1 << L, (N,), device="cuda", generator=g, dtype=torch.int32)
    idx = torch.randint(0, N, (NQ,), device="cuda", generator=g)
    out = torch.empty(NQ, dtype=torch.int64, device="cuda")
    torch.cuda.synchronize()
    t = wtg.WaveletTree.from_device(seq.data_ptr(), N, 4, L, wtg.RANK, st)
    t.sync()
    refused, went_on = _each_failure(wtg, torch, lambda: t.access_device(idx.data_ptr(), NQ, out.data_ptr(), st), out)
    assert refused == 0 and went_on == 11  # (the node tables were there)
    assert torch.equal(out, seq[idx].long())
    t.free()


@pytest.mark.parametrize("huff", [False, True])
def test_pattern_counts(wtg, huff):
    torch = pytest.importorskip("torch")
    g = torch.Generator(device="cuda")
    g.manual_seed(2)
    n, npat = 1 << 20, 1 << 19
    st = torch.cuda.current_stream().cuda_stream
    text = torch.randint(1, 6, (n,), device="cuda", generator=g).to(torch.uint8)
    text[-1] = 0
    bwt = torch.empty_like(text)
    torch.cuda.synchronize()
    wtg.suffix_array_device(text.data_ptr(), n, 0, bwt.data_ptr(), st)
    C = torch.zeros(256, dtype=torch.int64, device="cuda")
    C[1:] = torch.cumsum(torch.bincount(text.int(), minlength=256), 0)[:-1]
    lens = torch.randint(3, 20, (npat,), device="cuda", generator=g)
    off = torch.zeros(npat + 1, dtype=torch.int64, device="cuda")
    off[1:] = torch.cumsum(lens, 0)
    at = torch.randint(0, n - 32, (npat,), device="cuda", generator=g)
    pat = text[torch.repeat_interleave(at - off[:-1], lens) + torch.arange(int(off[-1]), device="cuda")]
    out = torch.empty(npat, dtype=torch.int64, device="cuda")
    torch.cuda.synchronize()
    h = wtg.HuffmanTree.from_device(bwt.data_ptr(), n, wtg.ALL, st) if huff else \
        wtg.FMIndex.from_device(bwt.data_ptr(), n, 6, st)
    count = h.fm_count_device if huff else h.count_device
    refused, went_on = _each_failure(
        wtg, torch, lambda: count(C.data_ptr(), pat.data_ptr(), off.data_ptr(), npat, out.data_ptr(), st), out)
    assert refused == 0 and went_on == 11  # (the step constants were there)
    assert bool((out > 0).all())
