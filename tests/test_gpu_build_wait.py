"""Tree builds under a look-back limit of one spin, so that any wait of a count or
rank pass may run out: a build reports the timeout or is right, and the next
one with the usual limit is right.  Chunks over many small nodes among them,
whose nodes are then not in order."""
import numpy as np
import pytest

import datagen

pytestmark = pytest.mark.gpu

SHAPES = [("exp", np.uint32, 20, 400001), ("u16", np.uint16, 13, 300001), ("exp", np.uint32, 20, 5_000_000),
          ("u8", np.uint8, 8, (1 << 22) + 3)]


@pytest.mark.parametrize("kind,dtype,L,n", SHAPES)
def test_builds(wtg, oracle, kind, dtype, L, n):
    sym = datagen.exp_u32(n, seed=n) if kind == "exp" else \
        np.random.default_rng(n).integers(0, 1 << L, n).astype(dtype)
    exp = oracle.wt_build(sym, L)[0]
    wtg.set_wait_limits(lookback_spins=1)
    try:
        for _ in range(6):
            try:
                t = wtg.WaveletTree(sym, levels=L, flags=wtg.RANK)
                assert np.array_equal(t.bits(), exp)
                t.free()
            except wtg.WtgError as e:
                assert e.code in (wtg.ERR_TIMEOUT, wtg.ERR_CUDA)  # (a bad index, found after the wait)
    finally:
        wtg.set_wait_limits(0, 0)
    t = wtg.WaveletTree(sym, levels=L, flags=wtg.RANK)
    assert np.array_equal(t.bits(), exp)
    t.free()


def test_huffman_builds(wtg, oracle):
    text = np.minimum(np.random.default_rng(2).zipf(1.3, 600001) - 1, 255).astype(np.uint8)
    exp = oracle.HuffOracle(text).words[:-1]
    wtg.set_wait_limits(lookback_spins=1)
    try:
        for _ in range(6):
            try:
                t = wtg.HuffmanTree(text, flags=wtg.RANK)
                assert np.array_equal(t.bits(), exp)
                t.free()
            except wtg.WtgError as e:
                assert e.code in (wtg.ERR_TIMEOUT, wtg.ERR_CUDA)
    finally:
        wtg.set_wait_limits(0, 0)
    t = wtg.HuffmanTree(text, flags=wtg.RANK)
    assert np.array_equal(t.bits(), exp)
    t.free()
