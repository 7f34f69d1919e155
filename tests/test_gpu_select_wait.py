"""A look-back wait of the rank pass that runs out under a build of the select
supports: the finishing kernels leave its starts and offsets alone, the build
reports the timeout, and the next one is right.  Bitvectors dense and sparse
(long blocks), alone and under a tree."""
import numpy as np
import pytest

import datagen

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("density", [0.5, 0.0002])
def test_bitvector(wtg, oracle, density):
    size = (1 << 25) + 123
    words = datagen.random_bits(size, density, seed=5)
    wtg.set_wait_limits(lookback_spins=2000)
    try:
        for _ in range(2):
            wtg.inject_lookback_stall(True)
            with pytest.raises(wtg.WtgError) as e:
                wtg.BitVectorSupport(words, size, wtg.ALL)
            assert e.value.code in (wtg.ERR_TIMEOUT, wtg.ERR_OOM)
    finally:
        wtg.inject_lookback_stall(False)
        wtg.set_wait_limits(0, 0)
    b = wtg.BitVectorSupport(words, size, wtg.ALL)
    s = oracle.Select(np.concatenate([words, np.zeros(1, np.uint64)]), size, 1)
    assert np.array_equal(b.select_tables(1).pool, s.pool)
    b.free()


def test_tree(wtg, oracle):
    sym = datagen.exp_u32(1 << 20, seed=4)
    wtg.set_wait_limits(lookback_spins=2000)
    try:
        wtg.inject_lookback_stall(True)
        with pytest.raises(wtg.WtgError) as e:
            wtg.WaveletTree(sym, levels=20, flags=wtg.ALL)
        assert e.value.code in (wtg.ERR_TIMEOUT, wtg.ERR_OOM)
    finally:
        wtg.inject_lookback_stall(False)
        wtg.set_wait_limits(0, 0)
    t = wtg.WaveletTree(sym, levels=20, flags=wtg.ALL)
    assert np.array_equal(t.bits(), oracle.wt_build(sym, 20)[0])
    idx = np.arange(0, sym.size, 1001, dtype=np.uint64)
    c = sym[idx.astype(np.int64)].astype(np.uint64)
    assert np.array_equal(t.select(t.rank(idx, c) + np.uint64(1), c), idx)
    t.free()
