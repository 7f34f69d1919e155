"""wt_huff over texts beyond 32-bit positions, which take one pass per depth: just
past the group passes' limit, and with more than 2^32 zeros at one depth.
Checked against the text itself (access, counts, ranks)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,values", [(0xFFFF0000 + 1001, 11), ((1 << 33) + (1 << 24) + 5, 4)])
def test_beyond_32_bits(wtg, n, values):
    torch = pytest.importorskip("torch")
    if torch.cuda.mem_get_info()[0] < 64 << 30:
        pytest.skip("needs 64 GB")
    g = torch.Generator(device="cuda")
    g.manual_seed(n)
    text = torch.empty(n, dtype=torch.uint8, device="cuda")
    counts = torch.zeros(values, dtype=torch.int64, device="cuda")
    step = 1 << 28
    for o in range(0, n, step):
        part = torch.randint(0, values, (min(step, n - o),), device="cuda", generator=g, dtype=torch.uint8)
        text[o:o + part.numel()] = part
        counts += torch.stack([(part == c).sum() for c in range(values)])
    half = n // 2 + 3
    below = torch.zeros(values, dtype=torch.int64, device="cuda")
    for o in range(0, half, step):
        part = text[o:min(o + step, half)]
        below += torch.stack([(part == c).sum() for c in range(values)])
    torch.cuda.synchronize()
    h = wtg.HuffmanTree.from_device(text.data_ptr(), n, wtg.RANK, torch.cuda.current_stream().cuda_stream)
    assert (h.n, h.sigma) == (n, values)
    idx = torch.cat([torch.randint(0, n, (1 << 16,), device="cuda", generator=g),
                     torch.arange(n - 2048, n, device="cuda"), torch.arange(0, 2048, device="cuda")])
    assert np.array_equal(h.access(idx.cpu().numpy().astype(np.uint64)), text[idx].cpu().numpy())
    c = np.arange(values, dtype=np.uint64)
    for at, exp in ((n, counts), (half, below)):
        assert np.array_equal(h.rank(np.full(values, at, dtype=np.uint64), c), exp.cpu().numpy().astype(np.uint64))
    h.free()
