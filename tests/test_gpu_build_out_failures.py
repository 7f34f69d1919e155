"""wtg_tree_build_out that fails (every device allocation of it in turn): once it has
returned nothing is written to the caller's arrays any more, and the handle
builds again."""
import numpy as np
import pytest

import datagen

pytestmark = pytest.mark.gpu


def test_no_copy_after_the_return(wtg, oracle):
    torch = pytest.importorskip("torch")
    n, L = (1 << 23) + 77, 20
    seq = torch.empty(n, dtype=torch.int32, pin_memory=True)
    sym = seq.numpy().view(np.uint32)
    sym[:] = datagen.exp_u32(n, seed=6)
    words = (n * L + 63) // 64
    rank_words = 2 * (words // 8 + 1)
    bits = torch.zeros(words, dtype=torch.int64, pin_memory=True)
    rank = torch.zeros(rank_words, dtype=torch.int64, pin_memory=True)
    small = wtg.WaveletTree.build_out(sym[:5000].copy(), L, wtg.ALL, bits.data_ptr(), rank.data_ptr())
    failed = 0
    try:
        for k in range(1, 60):
            wtg.inject_alloc_failure(k)
            try:
                t = wtg.WaveletTree.build_out(sym, L, wtg.ALL, bits.data_ptr(), rank.data_ptr(), tree=small)
            except wtg.WtgError as e:
                assert e.code == wtg.ERR_OOM
                failed += 1
                bits.fill_(-3)
                rank.fill_(-3)
                torch.cuda.synchronize()
                assert bool((bits == -3).all()) and bool((rank == -3).all())
                small = wtg.WaveletTree.build_out(sym[:5000].copy(), L, wtg.ALL, bits.data_ptr(), rank.data_ptr())
                continue
            break
    finally:
        wtg.inject_alloc_failure(0)
    assert failed >= 5
    exp = oracle.wt_build(sym, L)[0]
    assert np.array_equal(bits.numpy().view(np.uint64), exp)
    assert np.array_equal(t.bits(), exp)
    t.free()
