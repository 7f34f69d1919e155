"""The node tables that queries share, made by the first query after a build:
a query on another stream than the one that is still filling them waits for
them, and a query captured into a graph leaves nothing to the calls after it
that exists only once the graph has run."""
import numpy as np
import pytest

import datagen

pytestmark = pytest.mark.gpu

N, L, NQ = 300001, 20, 2000


@pytest.fixture()
def tree(wtg):
    torch = pytest.importorskip("torch")
    seq = datagen.exp_u32(N, seed=5)
    d = torch.from_numpy(seq.view(np.int32).copy()).cuda()
    torch.cuda.synchronize()
    t = wtg.WaveletTree.from_device(d.data_ptr(), N, 4, L, wtg.ALL, torch.cuda.current_stream().cuda_stream)
    t.sync()
    rng = np.random.default_rng(1)
    idx = rng.integers(0, N, NQ)
    order = np.argsort(seq, kind="stable")
    first = np.searchsorted(seq[order], seq[idx], side="left")
    yield torch, t, seq, idx, order[first]  # position of the first occurrence of each query's symbol
    torch.cuda.synchronize()
    t.free()


def test_queries_on_other_streams_wait_for_the_table(tree):
    torch, t, seq, idx, first = tree
    d_idx = torch.from_numpy(idx).cuda()
    outs = [torch.zeros(NQ, dtype=torch.int64, device="cuda") for _ in range(3)]
    streams = [torch.cuda.Stream() for _ in range(2)]
    ones, sym = np.ones(NQ, dtype=np.uint64), seq[idx].astype(np.uint64)
    d_sym = torch.from_numpy(seq[idx].astype(np.int64)).cuda()
    torch.cuda.synchronize()
    with torch.cuda.stream(streams[0]):
        torch.cuda._sleep(400_000_000)  # a few tenths of a second before the table is filled
    t.access_device(d_idx.data_ptr(), NQ, outs[0].data_ptr(), streams[0].cuda_stream)
    t.rank_device(d_idx.data_ptr(), d_sym.data_ptr(), NQ, outs[1].data_ptr(), streams[1].cuda_stream)
    assert np.array_equal(t.select(ones, sym), first.astype(np.uint64))  # on the tree's own stream
    assert np.array_equal(t.access(idx.astype(np.uint64)), sym)
    torch.cuda.synchronize()
    assert np.array_equal(outs[0].cpu().numpy(), seq[idx])
    rank = np.array([np.count_nonzero(seq[:i] == c) for i, c in zip(idx[:50], seq[idx[:50]])])
    assert np.array_equal(outs[1].cpu().numpy()[:50], rank)


@pytest.mark.parametrize("table_first", [False, True])
def test_captured_queries(tree, table_first):
    torch, t, seq, idx, first = tree
    if table_first:
        t.access(np.zeros(1, dtype=np.uint64))
    d_idx = torch.from_numpy(idx).cuda()
    out = torch.zeros(NQ, dtype=torch.int64, device="cuda")
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        t.access_device(d_idx.data_ptr(), NQ, out.data_ptr(), torch.cuda.current_stream().cuda_stream)
    # a call before the graph has run
    sym = seq[idx].astype(np.uint64)
    assert np.array_equal(t.access(idx.astype(np.uint64)), sym)
    assert np.array_equal(t.select(np.ones(NQ, dtype=np.uint64), sym), first.astype(np.uint64))
    for _ in range(2):
        out.zero_()
        g.replay()
        torch.cuda.synchronize()
        assert np.array_equal(out.cpu().numpy(), seq[idx])
    del g
    torch.cuda.synchronize()
    assert np.array_equal(t.access(idx.astype(np.uint64)), sym)


def test_level_selects_on_other_streams_wait_for_the_level_table(tree):
    torch, t, seq, idx, first = tree
    level, k = np.full(NQ, L - 1, dtype=np.uint64), np.arange(1, NQ + 1, dtype=np.uint64)
    d_level, d_k = (torch.from_numpy(x.view(np.int64)).cuda() for x in (level, k))
    out = torch.zeros(NQ, dtype=torch.int64, device="cuda")
    slow = torch.cuda.Stream()
    torch.cuda.synchronize()
    with torch.cuda.stream(slow):
        torch.cuda._sleep(400_000_000)
    t.level_select_device(1, d_level.data_ptr(), d_k.data_ptr(), NQ, out.data_ptr(), slow.cuda_stream)
    got = t.level_select(level, k)  # on the tree's own stream
    order = np.argsort(seq >> 1, kind="stable")  # the last level's order
    assert np.array_equal(got, np.flatnonzero(seq[order] & 1)[:NQ].astype(np.uint64))
    torch.cuda.synchronize()
    assert np.array_equal(out.cpu().numpy().view(np.uint64), got)
