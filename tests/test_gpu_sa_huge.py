"""A suffix array of more than 2^30 symbols, whose sorts keep 64-bit status words:
checked as a permutation in the order of (first byte, rank of the rest)."""
import pytest

pytestmark = pytest.mark.gpu


def test_beyond_2p30_symbols(wtg):
    torch = pytest.importorskip("torch")
    n = (1 << 30) + 12345
    if torch.cuda.mem_get_info()[0] < 100 << 30:
        pytest.skip("needs 100 GB")
    g = torch.Generator(device="cuda")
    g.manual_seed(30)
    text = torch.empty(n, dtype=torch.uint8, device="cuda")
    for o in range(0, n, 1 << 28):
        text[o:o + (1 << 28)] = torch.randint(0, 4, (min(1 << 28, n - o),), device="cuda", generator=g).to(torch.uint8)
    text[n // 2:n // 2 + (1 << 20)] = text[:1 << 20]  # a long repeat
    sa = torch.empty(n, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    wtg.suffix_array_device(text.data_ptr(), n, sa.data_ptr(), 0, torch.cuda.current_stream().cuda_stream)
    rank = torch.full((n + 1,), -1, dtype=torch.int32, device="cuda")  # past the end: first
    step = 1 << 27
    for o in range(0, n, step):
        part = sa[o:o + step].long()
        rank[part] = torch.arange(o, o + part.numel(), device="cuda", dtype=torch.int32)
    assert int(rank[:n].min()) == 0  # every suffix has its place
    last = None
    for o in range(0, n, step):
        part = sa[o:o + step].long()
        key = text[part].long() * (n + 1) + rank[part + 1].long() + 1
        assert bool((key[1:] > key[:-1]).all())
        assert last is None or int(key[0]) > last
        last = int(key[-1])
