"""Backward-search counts of large pattern batches -- interval table, 192-bit
blocks, patterns by length -- equal the counts of the same patterns in batches
too small for any of them (checked against the oracle in test_gpu_fm.py and
test_gpu_huff.py), over the balanced and the Huffman-shaped tree, at pattern
buffers that do not start on an 8-byte boundary."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

NPAT, SMALL = (1 << 19) + 9, 1 << 13


def _setup(wtg, torch, sigma, n, seed):
    rng = np.random.default_rng(seed)
    text = np.minimum(rng.geometric(0.35 if sigma < 10 else 0.05, n), sigma - 1).astype(np.uint8)
    text[-1] = 0  # unique smallest symbol: counts are occurrences
    b = wtg.bwt(text)
    C = np.zeros(256, dtype=np.uint64)
    C[1:] = np.cumsum(np.bincount(text, minlength=256))[:-1]
    lens = rng.integers(0, 40, NPAT)
    lens[:4] = [0, 1, 300, 2]
    start = rng.integers(0, n - 301, NPAT)
    off = np.concatenate([[0], np.cumsum(lens)]).astype(np.uint64)
    pat = text[np.repeat(start - off[:-1].astype(np.int64), lens) + np.arange(int(off[-1]))]
    pat[::997] = 255 if sigma < 255 else 0  # a symbol the text does not have (or has once)
    return b, C, pat, off


@pytest.mark.parametrize("sigma,n,shift", [(6, 1 << 20, 0), (6, 300001, 3), (200, 1 << 18, 5)])
def test_balanced_and_huffman(wtg, sigma, n, shift):
    torch = pytest.importorskip("torch")
    b, C, pat, off = _setup(wtg, torch, sigma, n, sigma + n)
    st = torch.cuda.current_stream().cuda_stream
    d_b, d_C = torch.from_numpy(b).cuda(), torch.from_numpy(C.view(np.int64)).cuda()
    buf = torch.zeros(pat.size + shift, dtype=torch.uint8, device="cuda")
    buf[shift:] = torch.from_numpy(pat).cuda()
    d_pat, d_off = buf.data_ptr() + shift, torch.from_numpy(off.view(np.int64)).cuda()
    fm = wtg.FMIndex.from_device(d_b.data_ptr(), n, sigma, st)
    hf = wtg.HuffmanTree.from_device(d_b.data_ptr(), n, wtg.ALL, st)
    res = {}
    for name, f in (("balanced", fm.count_device), ("huff", hf.fm_count_device)):
        whole = torch.empty(NPAT, dtype=torch.int64, device="cuda")
        parts = torch.empty_like(whole)
        f(d_C.data_ptr(), d_pat, d_off.data_ptr(), NPAT, whole.data_ptr(), st)
        for at in range(0, NPAT, SMALL):
            f(d_C.data_ptr(), d_pat, d_off.data_ptr() + 8 * at, min(SMALL, NPAT - at), parts.data_ptr() + 8 * at, st)
        torch.cuda.synchronize()
        assert torch.equal(whole, parts), name
        res[name] = whole
    assert torch.equal(res["balanced"], res["huff"])
    assert int(res["huff"][0]) == n


@pytest.mark.parametrize("npat", [1000, 1 << 19])  # without and with the interval table
def test_offsets_that_decrease_are_empty_patterns(wtg, npat):
    """A device batch's offsets are not checked; nothing outside the patterns is read."""
    torch = pytest.importorskip("torch")
    n, st = 1 << 16, torch.cuda.current_stream().cuda_stream
    rng = np.random.default_rng(npat)
    text = rng.integers(1, 6, n).astype(np.uint8)
    text[-1] = 0
    C = np.zeros(256, dtype=np.uint64)
    C[1:] = np.cumsum(np.bincount(text, minlength=256))[:-1]
    off = np.zeros(npat + 1, dtype=np.uint64)
    off[1::2] = 12  # 0, 12, 0, 12, ..: every second pattern's offsets decrease to 0
    d_b, d_C, d_off = (torch.from_numpy(x).cuda() for x in (wtg.bwt(text), C.view(np.int64), off.view(np.int64)))
    d_pat = torch.from_numpy(text[:12].copy()).cuda()
    torch.cuda.synchronize()
    fm = wtg.FMIndex.from_device(d_b.data_ptr(), n, 6, st)
    hf = wtg.HuffmanTree.from_device(d_b.data_ptr(), n, wtg.ALL, st)
    for f in (fm.count_device, hf.fm_count_device):
        out = torch.empty(npat, dtype=torch.int64, device="cuda")
        f(d_C.data_ptr(), d_pat.data_ptr(), d_off.data_ptr(), npat, out.data_ptr(), st)
        torch.cuda.synchronize()
        assert bool((out[1::2] == n).all()) and bool((out[::2] >= 1).all()) and bool((out[::2] < n).all())
