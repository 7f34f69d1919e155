"""Backward-search counts on several streams over one tree at once: a count leaves
nothing in the handle that another one reads or writes, on whatever stream it
runs and however late, and a count captured into a graph keeps nothing there."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

N, NPAT = 20001, 500


@pytest.fixture(scope="module")
def text(wtg):
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(3)
    s = np.minimum(rng.geometric(0.3, N), 5).astype(np.uint8)
    s[-1] = 0
    C = np.zeros(256, dtype=np.uint64)
    C[1:] = np.cumsum(np.bincount(s, minlength=256))[:-1]
    off = (np.arange(NPAT + 1) * 4).astype(np.uint64)
    start = rng.integers(0, N - 5, NPAT)
    pat = np.concatenate([s[a:a + 4] for a in start]).astype(np.uint8)
    b = s.tobytes()
    exp = np.array([sum(b.startswith(bytes(pat[4 * k:4 * k + 4]), i) for i in range(N)) for k in range(20)])
    return torch, wtg.bwt(s), C, pat, off, exp


def _huff(wtg, bwt, st):
    h = wtg.HuffmanTree.from_device(bwt.data_ptr(), N, wtg.ALL, st)
    return h, h.fm_count_device


def _balanced(wtg, bwt, st):
    f = wtg.FMIndex.from_device(bwt.data_ptr(), N, 6, st)
    return f.tree, f.count_device


def _device(torch, arrays):
    return [torch.from_numpy(a.view(np.int64) if a.dtype == np.uint64 else a.copy()).cuda() for a in arrays]


@pytest.mark.parametrize("make", [_huff, _balanced])
def test_counts_on_two_streams(wtg, text, make):
    torch, bwt, C, pat, off, exp = text
    d_bwt, d_C, d_pat, d_off = _device(torch, (bwt, C, pat, off))
    out = [torch.zeros(NPAT, dtype=torch.int64, device="cuda") for _ in range(2)]
    slow, st = torch.cuda.Stream(), torch.cuda.current_stream()
    torch.cuda.synchronize()
    h, count = make(wtg, d_bwt, st.cuda_stream)
    torch.cuda.synchronize()
    with torch.cuda.stream(slow):
        torch.cuda._sleep(400_000_000)
    count(d_C.data_ptr(), d_pat.data_ptr(), d_off.data_ptr(), NPAT, out[0].data_ptr(), slow.cuda_stream)
    count(d_C.data_ptr(), d_pat.data_ptr(), d_off.data_ptr(), NPAT, out[1].data_ptr(), st.cuda_stream)
    st.synchronize()
    got = out[1].cpu().numpy()
    assert np.array_equal(got[:20], exp)
    torch.cuda.synchronize()
    assert torch.equal(out[0], out[1])
    h.free()


def test_counts_with_different_C_on_two_streams(wtg, text):
    """A call's C and number of symbols are its own."""
    torch, bwt, C, pat, off, exp = text
    d_bwt, d_C, d_pat, d_off = _device(torch, (bwt, C, pat, off))
    d_zero = torch.zeros_like(d_C)
    slow, st = torch.cuda.Stream(), torch.cuda.current_stream()
    t = wtg.FMIndex.from_device(d_bwt.data_ptr(), N, 6, st.cuda_stream).tree

    def count(d_c, sigma, stream, out):
        wtg._ck(wtg.lib().wtg_fm_count_device(t.h, d_c.data_ptr(), sigma, d_pat.data_ptr(), d_off.data_ptr(), NPAT,
                                              out.data_ptr(), stream.cuda_stream))

    calls = [(d_C, 4), (d_zero, 6), (d_C, 6), (d_zero, 4)]
    alone = [torch.zeros(NPAT, dtype=torch.int64, device="cuda") for _ in calls]
    got = [torch.zeros(NPAT, dtype=torch.int64, device="cuda") for _ in calls]
    for (c, sigma), out in zip(calls, alone):
        count(c, sigma, st, out)
        torch.cuda.synchronize()
    with torch.cuda.stream(slow):
        torch.cuda._sleep(400_000_000)
    for k, ((c, sigma), out) in enumerate(zip(calls, got)):
        count(c, sigma, (slow, st)[k % 2], out)
    torch.cuda.synchronize()
    for a, b in zip(got, alone):
        assert torch.equal(a, b)
    assert np.array_equal(got[2].cpu().numpy()[:20], exp)


@pytest.mark.parametrize("make", [_huff, _balanced])
def test_captured_count(wtg, text, make):
    torch, bwt, C, pat, off, exp = text
    d_bwt, d_C, d_pat, d_off = _device(torch, (bwt, C, pat, off))
    out = torch.zeros(NPAT, dtype=torch.int64, device="cuda")
    torch.cuda.synchronize()
    h, count = make(wtg, d_bwt, torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()

    def call():
        count(d_C.data_ptr(), d_pat.data_ptr(), d_off.data_ptr(), NPAT, out.data_ptr(),
              torch.cuda.current_stream().cuda_stream)

    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        call()
    call()  # before the graph has run
    torch.cuda.synchronize()
    first = out.cpu().numpy().copy()
    assert np.array_equal(first[:20], exp)
    out.zero_()
    g.replay()
    torch.cuda.synchronize()
    assert np.array_equal(out.cpu().numpy(), first)
    del g
    torch.cuda.synchronize()
    out.zero_()
    call()
    torch.cuda.synchronize()
    assert np.array_equal(out.cpu().numpy(), first)
    h.free()
