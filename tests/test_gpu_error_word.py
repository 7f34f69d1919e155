"""The device error word of a handle: an error that a build's kernels report is
seen by the first call that waits, stays for the calls after it, and is gone
with the next build."""
import numpy as np
import pytest

import datagen

pytestmark = pytest.mark.gpu


def test_error_stays_until_the_next_build(wtg, oracle):
    torch = pytest.importorskip("torch")
    n, L = 1 << 20, 8
    sym = (datagen.exp_u32(n, seed=3) & 255).astype(np.uint8)
    d = torch.from_numpy(sym).cuda()
    st = torch.cuda.current_stream().cuda_stream
    torch.cuda.synchronize()
    good = wtg.WaveletTree.from_device(d.data_ptr(), n, 1, L, wtg.RANK, st)
    bits = good.bits()
    assert np.array_equal(bits, oracle.wt_build(sym, L)[0])
    assert np.array_equal(good.bits(), bits)  # found clear: not read again
    wtg.set_wait_limits(lookback_spins=2000)
    try:
        wtg.inject_lookback_stall(True)
        t = wtg.WaveletTree.from_device(d.data_ptr(), n, 1, L, wtg.RANK, st)
        for call in (t.bits, t.rank_table, t.bits, t.sync):
            with pytest.raises(wtg.WtgError) as e:
                call()
            assert e.value.code == wtg.ERR_TIMEOUT
    finally:
        wtg.inject_lookback_stall(False)
        wtg.set_wait_limits(0, 0)
    wtg.WaveletTree.from_device(d.data_ptr(), n, 1, L, wtg.RANK, st, tree=t)
    assert np.array_equal(t.bits(), bits)
    assert np.array_equal(t.rank_table(), good.rank_table())
    # a device call on another stream may still report: every check reads
    s2 = torch.cuda.Stream()
    idx = torch.zeros(4, dtype=torch.int64, device="cuda")
    out = torch.empty_like(idx)
    torch.cuda.synchronize()
    t.access_device(idx.data_ptr(), 4, out.data_ptr(), s2.cuda_stream)
    torch.cuda.synchronize()
    assert int(out[0]) == int(sym[0]) and np.array_equal(t.bits(), bits)
    t.free()
    good.free()
