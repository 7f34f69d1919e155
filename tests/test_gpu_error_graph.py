"""A sorted batch captured into a graph on the handle's own stream: a wait that
runs out when the graph is launched, after the handle's error word was found
clear, is reported by the check that follows."""
import pytest

pytestmark = pytest.mark.gpu

N, L, NQ = (1 << 25) + 3, 20, (1 << 21) + 5


def test_launched_graph_reports(wtg):
    torch = pytest.importorskip("torch")
    own = torch.cuda.Stream()
    seq = torch.randint(0, 1 << L, (N,), device="cuda", dtype=torch.int32)
    idx = torch.randint(0, N, (NQ,), device="cuda")
    out = torch.empty(NQ, dtype=torch.int64, device="cuda")
    torch.cuda.synchronize()
    t = wtg.WaveletTree.from_device(seq.data_ptr(), N, 4, L, wtg.RANK, own.cuda_stream)
    t.access_device(idx.data_ptr(), NQ, out.data_ptr(), own.cuda_stream)
    t.sync()
    assert torch.equal(out, seq[idx].long())
    graphs = []
    for stall in (False, True):
        g = torch.cuda.CUDAGraph()
        wtg.inject_lookback_stall(stall)
        with torch.cuda.graph(g, stream=own):
            t.access_device(idx.data_ptr(), NQ, out.data_ptr(), own.cuda_stream)
        graphs.append(g)
    wtg.inject_lookback_stall(False)
    t.sync()  # nothing has run: clear
    out.zero_()
    torch.cuda.synchronize()
    with torch.cuda.stream(own):
        graphs[0].replay()
    t.sync()
    assert torch.equal(out, seq[idx].long())
    wtg.set_wait_limits(lookback_spins=2000)
    try:
        with torch.cuda.stream(own):
            graphs[1].replay()
        with pytest.raises(wtg.WtgError) as e:
            t.sync()
        assert e.value.code == wtg.ERR_TIMEOUT
    finally:
        wtg.set_wait_limits(0, 0)
    torch.cuda.synchronize()
    del graphs, g
    t.free()
