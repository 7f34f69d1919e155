"""Suffix arrays of texts whose groups of equal suffixes span many settling tiles:
one letter throughout, one long run, a run between other text, two letters with
a long run each."""
import pytest

pytestmark = pytest.mark.gpu


def _texts(torch, n):
    g = torch.Generator(device="cuda")
    g.manual_seed(n)
    noise = torch.randint(0, 4, (n,), device="cuda", generator=g).to(torch.uint8)
    same = torch.full_like(noise, 2)
    end, middle, two = noise.clone(), noise.clone(), same.clone()
    end[n // 3:] = 1
    middle[n // 4:n // 2] = 3
    two[n // 2:] = 0
    return {"same": same, "end": end, "middle": middle, "two": two}


@pytest.mark.parametrize("kind", ["same", "end", "middle", "two"])
@pytest.mark.parametrize("n", [4096, 3 * 4096 + 1, (1 << 20) + 3, (1 << 24) + 5])
def test_runs(wtg, kind, n):
    torch = pytest.importorskip("torch")
    text = _texts(torch, n)[kind]
    sa = torch.empty(n, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    wtg.suffix_array_device(text.data_ptr(), n, sa.data_ptr(), 0, torch.cuda.current_stream().cuda_stream)
    sa = sa.long()
    if kind == "same":
        assert torch.equal(sa, torch.arange(n - 1, -1, -1, device="cuda"))
    rank = torch.full((n + 1,), -1, dtype=torch.int64, device="cuda")  # past the end: first
    rank[sa] = torch.arange(n, device="cuda")
    key = text[sa].long() * (n + 1) + rank[sa + 1] + 1
    assert int(rank[:n].min()) == 0 and bool((key[1:] > key[:-1]).all())
