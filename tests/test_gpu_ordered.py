"""Query batches that come in the order of their positions, which are not sorted
again, and batches that only nearly do: every answer equals the one that the
same queries get in batches too small to be sorted.  Batches of more than 2^26
queries, which run in parts, with parts in order and parts not."""
import pytest

pytestmark = pytest.mark.gpu

N, L, SMALL = (1 << 26) + 3, 20, 1 << 18


@pytest.fixture(scope="module")
def s(wtg):
    torch = pytest.importorskip("torch")
    g = torch.Generator(device="cuda")
    g.manual_seed(21)
    x = torch.empty(N, device="cuda").exponential_(2.0 ** -14, generator=g).floor_().clamp_(max=2 ** L - 1)
    seq = x.to(torch.int32)
    torch.cuda.synchronize()
    t = wtg.WaveletTree.from_device(seq.data_ptr(), N, 4, L, wtg.RANK, torch.cuda.current_stream().cuda_stream)
    t.sync()
    yield torch, t, seq, g
    t.free()


def _positions(torch, g, kind, nq):
    r = torch.randint(0, N, (nq,), device="cuda", generator=g)
    if kind == "random":
        return r
    if kind == "same":
        return torch.full((nq,), N // 3, dtype=torch.int64, device="cuda")
    if kind == "consecutive":  # past the end of the sequence, too
        return torch.arange(nq, device="cuda") + (N - nq + 5)
    up = torch.sort(r).values
    if kind == "down":
        return torch.flip(up, [0])
    if kind == "runs":
        return torch.sort(r[:nq // 100 * 100].view(100, -1), dim=1).values.reshape(-1)
    if kind == "one_out":  # not in order by one query, which the check need not see
        up[nq // 2], up[nq // 2 + 1] = N - 1, 0
    return up


def _check(torch, t, seq, idx, nq):
    st = torch.cuda.current_stream().cuda_stream
    at = torch.randint(0, N, (nq,), device="cuda")
    sym = seq[at].long()
    end = torch.clamp(idx + 3000, max=N)
    p = [x.data_ptr() for x in (idx, end, sym)]
    got, exp = ([torch.empty(nq, dtype=torch.int64, device="cuda") for _ in range(6)] for _ in range(2))
    for outs, part in ((got, nq), (exp, SMALL)):
        for k in range(0, nq, part):
            m, o = min(part, nq - k), [x.data_ptr() + 8 * k for x in outs]
            a, b, c = (x + 8 * k for x in p)
            t.access_device(a, m, o[0], st)
            t.rank_device(a, c, m, o[1], st)
            t.lex_count_device(a, b, c, m, *o[2:5], st)
            t.range_count_device(a, b, c, c, m, o[5], st)
    torch.cuda.synchronize()
    for a, b in zip(got, exp):
        assert torch.equal(a, b)
    ok = (idx >= 0) & (idx < N)
    assert torch.equal(got[0][ok], seq[idx[ok]].long()) and bool((got[0][~ok] == -1).all())


# sorted over the two tables, and over the blocks
@pytest.mark.parametrize("nq", [(1 << 20) + 1, (5 << 19) + 5])
@pytest.mark.parametrize("kind", ["random", "same", "consecutive", "up", "down", "runs", "one_out"])
def test_orders(s, kind, nq):
    torch, t, seq, g = s
    idx = _positions(torch, g, kind, nq)
    _check(torch, t, seq, idx, idx.numel())


@pytest.mark.parametrize("kinds", [("random", "up"), ("up", "random"), ("up", "up")])
def test_parts(s, kinds):
    torch, t, seq, g = s
    nq, st = (1 << 26) + 100003, torch.cuda.current_stream().cuda_stream
    idx = torch.cat([_positions(torch, g, kinds[0], 1 << 26), _positions(torch, g, kinds[1], nq - (1 << 26))])
    sym = seq[torch.randint(0, N, (nq,), device="cuda", generator=g)].long()
    out = torch.full((2, nq), -9, dtype=torch.int64, device="cuda")
    torch.cuda.synchronize()
    t.access_device(idx.data_ptr(), nq, out[0].data_ptr(), st)
    t.rank_device(idx.data_ptr(), sym.data_ptr(), nq, out[1].data_ptr(), st)
    torch.cuda.synchronize()
    assert torch.equal(out[0], seq[idx].long())
    for k in [0, (1 << 26) - SMALL, 1 << 26, nq - 7]:  # pieces on both sides of the parts' edge
        m = min(SMALL, nq - k)
        exp = torch.empty(m, dtype=torch.int64, device="cuda")
        t.rank_device(idx.data_ptr() + 8 * k, sym.data_ptr() + 8 * k, m, exp.data_ptr(), st)
        torch.cuda.synchronize()
        assert torch.equal(out[1][k:k + m], exp)


def test_a_last_part_of_a_few_queries(s):
    torch, t, seq, g = s
    nq, st = (1 << 26) + 3, torch.cuda.current_stream().cuda_stream
    idx = _positions(torch, g, "random", nq)
    out = torch.full((nq,), -9, dtype=torch.int64, device="cuda")
    torch.cuda.synchronize()
    t.access_device(idx.data_ptr(), nq, out.data_ptr(), st)
    torch.cuda.synchronize()
    assert torch.equal(out, seq[idx].long())
