"""Look-back waits that run out while a suffix array is made: the call reports the
timeout (or is right, where no wait ran out), and the next one is right."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _text(torch, n, period, seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    t = torch.randint(0, 4, (n,), device="cuda", generator=g).to(torch.uint8)
    if period:  # long repeats: many rounds over a long active list
        t[n // 2:] = t[:period].repeat(n // period + 1)[:n - n // 2]
    return t


def _check(torch, text, sa):
    """sa is a permutation in the order of (first byte, rank of the rest)."""
    n = text.numel()
    sa = sa.long()
    rank = torch.full((n + 1,), -1, dtype=torch.int64, device="cuda")  # past the end: first
    rank[sa] = torch.arange(n, device="cuda")
    assert int(rank[:n].min()) == 0
    key = text[sa].long() * (n + 1) + rank[sa + 1] + 1
    assert bool((key[1:] > key[:-1]).all())


# below and from the size whose ranks are binned on
@pytest.mark.parametrize("n,period", [(300001, 0), (300001, 1000), ((1 << 24) + 5, 0), ((1 << 24) + 5, 1 << 16)])
def test_waits_that_run_out(wtg, n, period):
    torch = pytest.importorskip("torch")
    text = _text(torch, n, period, n)
    sa = torch.empty(n, dtype=torch.int32, device="cuda")
    st = torch.cuda.current_stream().cuda_stream
    torch.cuda.synchronize()
    wtg.set_wait_limits(lookback_spins=2000)
    try:
        wtg.inject_lookback_stall(True)  # tile 0 of the first sort
        with pytest.raises(wtg.WtgError) as e:
            wtg.suffix_array_device(text.data_ptr(), n, sa.data_ptr(), 0, st)
        assert e.value.code == wtg.ERR_TIMEOUT
    finally:
        wtg.inject_lookback_stall(False)
        wtg.set_wait_limits(0, 0)
    wtg.set_wait_limits(lookback_spins=1)  # any wait, of sorts and of settling, may run out
    try:
        for _ in range(3):
            try:
                wtg.suffix_array_device(text.data_ptr(), n, sa.data_ptr(), 0, st)
                _check(torch, text, sa)
            except wtg.WtgError as err:
                assert err.code == wtg.ERR_TIMEOUT
    finally:
        wtg.set_wait_limits(0, 0)
    wtg.suffix_array_device(text.data_ptr(), n, sa.data_ptr(), 0, st)
    _check(torch, text, sa)
