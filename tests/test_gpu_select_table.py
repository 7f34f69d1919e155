"""Selects by the node table (after an access made it, or in a batch that is
worth it) equal the selects that walk down the tree, at occurrences that exist
and one past them, absent symbols and symbols above the alphabet."""
import numpy as np
import pytest

import datagen

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,L", [(1, 1), (1000, 1), (1025, 3), (5000, 8), (70001, 20)])
def test_table_equals_walk(wtg, n, L):
    seq = datagen.exp_u32(n, seed=n) >> (20 - L) if L > 8 else \
        np.random.default_rng(n).integers(0, max(1, (1 << L) - 1), n).astype(np.uint32)
    rng = np.random.default_rng(n + 1)
    sym = np.concatenate([seq[rng.integers(0, n, 40)], [0, (1 << L) - 1, 1 << L, 1 << 40]]).astype(np.uint64)
    occ = np.array([np.count_nonzero(seq == c) for c in sym], dtype=np.uint64)
    q = np.concatenate([np.ones_like(occ), np.maximum(occ, 1), occ + 1, np.zeros_like(occ)]).astype(np.uint64)
    c = np.concatenate([sym] * 4)
    exp = np.full(q.size, np.iinfo(np.uint64).max, dtype=np.uint64)
    for k in range(q.size):
        if 1 <= q[k] <= np.count_nonzero(seq == c[k]):
            exp[k] = np.flatnonzero(seq == c[k])[int(q[k]) - 1]
    t = wtg.WaveletTree(seq, levels=L, flags=wtg.ALL)
    walk = np.concatenate([t.select(q[k:k + 1], c[k:k + 1]) for k in range(q.size)]) if L > 3 else t.select(q, c)
    assert np.array_equal(walk, exp)
    t.access(np.zeros(1, dtype=np.uint64))  # makes the table
    assert np.array_equal(t.select(q, c), exp)
    t.free()
