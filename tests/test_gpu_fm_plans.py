"""Large pattern batches whose preparation depends on their lengths (interval table
of fewer symbols than it could have, blocks or none, by length or as they come):
counts equal those of the same patterns in batches too small to be prepared, over
trees that L1 holds and larger ones, of 2 to 200 symbols."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SMALL = 1 << 11


def _lengths(kind, npat, rng):
    if kind == "mixed":
        return rng.integers(0, 60, npat)
    if kind == "few_long":
        return np.where(rng.random(npat) < 0.01, 250, 2)
    return np.full(npat, kind)


@pytest.mark.parametrize("sigma,n", [(2, 5000), (4, 40001), (6, 1 << 21), (200, 1 << 17)])
@pytest.mark.parametrize("kind", [0, 1, 2, 5, 9, 30, "mixed", "few_long"])
def test_counts(wtg, sigma, n, kind):
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(n)
    npat = ((3 << 18) + 77) // max(1, sigma.bit_length() - 1) + SMALL
    text = rng.integers(1, sigma, n).astype(np.uint8) if sigma > 2 else np.ones(n, dtype=np.uint8)
    if sigma == 2:
        text[rng.integers(0, n, n // 3)] = 0
    text[-1] = 0
    C = np.zeros(256, dtype=np.uint64)
    C[1:] = np.cumsum(np.bincount(text, minlength=256))[:-1]
    lens = _lengths(kind, npat, rng).astype(np.int64)
    off = np.concatenate([[0], np.cumsum(lens)])
    at = rng.integers(0, n - 260, npat)
    pat = text[np.repeat(at - off[:-1], lens) + np.arange(int(off[-1]))] if off[-1] else np.zeros(1, dtype=np.uint8)
    pat[::1009] = 255
    st = torch.cuda.current_stream().cuda_stream
    d_b, d_C, d_pat, d_off = (torch.from_numpy(x).cuda() for x in (wtg.bwt(text), C.view(np.int64), pat, off))
    torch.cuda.synchronize()
    fm = wtg.FMIndex.from_device(d_b.data_ptr(), n, sigma, st)
    hf = wtg.HuffmanTree.from_device(d_b.data_ptr(), n, wtg.ALL, st)
    res = []
    for f in (fm.count_device, hf.fm_count_device):
        whole = torch.full((npat,), -3, dtype=torch.int64, device="cuda")
        f(d_C.data_ptr(), d_pat.data_ptr(), d_off.data_ptr(), npat, whole.data_ptr(), st)
        m = min(60, npat // SMALL) * SMALL  # (enough of them)
        parts = torch.full((m,), -4, dtype=torch.int64, device="cuda")
        for k in range(0, m, SMALL):
            f(d_C.data_ptr(), d_pat.data_ptr(), d_off.data_ptr() + 8 * k, SMALL, parts.data_ptr() + 8 * k, st)
        torch.cuda.synchronize()
        assert torch.equal(whole[:m], parts)
        res.append(whole)
    assert torch.equal(*res)
    if kind == 0:
        assert bool((res[0] == n).all())
    elif kind != "mixed" and sigma > 2:  # (two letters: 0 is not the last symbol alone)
        assert int((res[0] > 0).sum()) > npat // 2
