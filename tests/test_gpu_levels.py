"""The level passes at the sizes where their paths change, against the oracle:
chunks of 1024 symbols and tiles of 8 chunks, one to six groups of levels,
chunks inside one node, over a few nodes and over many small ones, one symbol
only, symbols that do not start on a 32-byte boundary and 8-byte symbols."""
import numpy as np
import pytest

from helpers import words_with_tail

pytestmark = pytest.mark.gpu

KINDS = {  # dtype, levels, values
    "u8_3": (np.uint8, 3, lambda r, n: r.integers(0, 5, n)),
    "u8_5": (np.uint8, 5, lambda r, n: r.integers(0, 32, n)),
    "u8_8_same": (np.uint8, 8, lambda r, n: np.full(n, 0xB7)),
    "u8_8_runs": (np.uint8, 8, lambda r, n: np.repeat(r.integers(0, 256, n // 300 + 1), 300)[:n]),
    "u16_13": (np.uint16, 13, lambda r, n: r.integers(0, 1 << 13, n)),
    "u32_17_skew": (np.uint32, 17, lambda r, n: np.minimum(r.exponential(900, n), (1 << 17) - 1)),
    "u32_24": (np.uint32, 24, lambda r, n: r.integers(0, 1 << 24, n)),
    "u64_9": (np.uint64, 9, lambda r, n: r.integers(0, 1 << 60, n)),
}
SIZES = [1, 33, 1023, 1024, 1025, 3 * 1024, 8191, 8192 + 1, 70001, (1 << 18) + 511]


def _check(wtg, oracle, t, sym, L):
    bits, nodes = oracle.wt_build(sym, L, n_nodes=1 << min(L, 17))
    assert np.array_equal(t.bits(), bits)
    assert np.array_equal(t.nodes(1 << min(L, 17), index_bytes=8), nodes)
    assert np.array_equal(t.rank_table(), oracle.rank_build(words_with_tail(bits), sym.size * L))


@pytest.mark.parametrize("kind", list(KINDS))
@pytest.mark.parametrize("n", SIZES)
def test_sizes(wtg, oracle, kind, n):
    dtype, L, gen = KINDS[kind]
    sym = gen(np.random.default_rng(n), n).astype(dtype)
    _check(wtg, oracle, wtg.WaveletTree(sym, levels=L, flags=wtg.RANK), sym, L)


@pytest.mark.parametrize("kind", ["u8_5", "u16_13", "u32_17_skew"])
@pytest.mark.parametrize("shift", [1, 3, 16])
def test_unaligned_device_sequence(wtg, oracle, kind, shift):
    torch = pytest.importorskip("torch")
    dtype, L, gen = KINDS[kind]
    sym = gen(np.random.default_rng(shift), 50000).astype(dtype)
    d = torch.from_numpy(sym.view(f"i{sym.itemsize}").copy()).cuda()
    part = np.ascontiguousarray(sym[shift:])
    t = wtg.WaveletTree.from_device(d.data_ptr() + shift * sym.itemsize, part.size, sym.itemsize, L, wtg.RANK,
                                    torch.cuda.current_stream().cuda_stream)
    t.sync()
    _check(wtg, oracle, t, part, L)


def test_rebuild_over_larger_and_smaller(wtg, oracle):
    """A handle rebuilt with other sizes, widths and levels gives that build alone."""
    torch = pytest.importorskip("torch")
    st = torch.cuda.current_stream().cuda_stream
    t = None
    for kind, n in (("u32_24", 30000), ("u8_3", 200001), ("u16_13", 5000), ("u8_8_runs", 100000), ("u64_9", 3000)):
        dtype, L, gen = KINDS[kind]
        sym = gen(np.random.default_rng(n), n).astype(dtype)
        d = torch.from_numpy(sym.view(f"i{sym.itemsize}").copy()).cuda()
        t = wtg.WaveletTree.from_device(d.data_ptr(), n, sym.itemsize, L, wtg.ALL, st, tree=t)
        t.sync()
        _check(wtg, oracle, t, sym, L)
