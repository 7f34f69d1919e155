"""Trees with more levels than a symbol of the sequence has bits: the levels above
it are zeros.  Against the oracle, at the sizes around a chunk of 1024 symbols,
from host arrays and from device sequences that do not start on a 32-byte
boundary."""
import numpy as np
import pytest

from helpers import words_with_tail

pytestmark = pytest.mark.gpu

SHAPES = [(np.uint8, 9), (np.uint8, 12), (np.uint8, 16), (np.uint8, 17), (np.uint8, 24), (np.uint16, 17),
          (np.uint16, 20), (np.uint16, 24)]


def _symbols(dtype, n):
    return np.random.default_rng(n).integers(0, np.iinfo(dtype).max + 1, n).astype(dtype)


def _check(wtg, oracle, t, sym, L):
    bits, nodes = oracle.wt_build(sym.astype(np.uint32), L, n_nodes=1 << min(L, 17))
    assert np.array_equal(t.bits(), bits)
    assert np.array_equal(t.nodes(1 << min(L, 17), index_bytes=8), nodes)
    assert np.array_equal(t.rank_table(), oracle.rank_build(words_with_tail(bits), sym.size * L))
    idx = np.arange(0, sym.size, 7, dtype=np.uint64)
    assert np.array_equal(t.access(idx), sym[::7].astype(np.uint64))


@pytest.mark.parametrize("dtype,L", SHAPES)
@pytest.mark.parametrize("n", [1, 33, 1023, 1024, 1025, 9001, 70001])
def test_sizes(wtg, oracle, dtype, L, n):
    sym = _symbols(dtype, n)
    _check(wtg, oracle, wtg.WaveletTree(sym, levels=L, flags=wtg.ALL), sym, L)


@pytest.mark.parametrize("dtype,L", SHAPES)
@pytest.mark.parametrize("shift", [1, 16])
def test_unaligned_device_sequence(wtg, oracle, dtype, L, shift):
    torch = pytest.importorskip("torch")
    sym = _symbols(dtype, 30000)
    d = torch.from_numpy(sym.view(f"i{sym.itemsize}").copy()).cuda()
    part = np.ascontiguousarray(sym[shift:])
    torch.cuda.synchronize()
    t = wtg.WaveletTree.from_device(d.data_ptr() + shift * sym.itemsize, part.size, sym.itemsize, L, wtg.ALL,
                                    torch.cuda.current_stream().cuda_stream)
    t.sync()
    _check(wtg, oracle, t, part, L)


def test_wt_of_bytes_with_an_alphabet_above_256(wtg, oracle):
    sym = _symbols(np.uint8, 5000)
    nodes, bits = wtg.WT(sym, 257)  # 9 levels
    exp_bits, exp_nodes = oracle.wt_build(sym.astype(np.uint32), 9, n_nodes=len(nodes))
    assert np.array_equal(np.asarray(bits), exp_bits)
    assert len(nodes) == len(exp_nodes)


def test_pieces_of_a_page_locked_input(wtg, oracle):
    """build_out copies a page-locked input in pieces; the widening waits for all of them."""
    torch = pytest.importorskip("torch")
    n, L = (1 << 22) + 5, 9
    pinned = torch.empty(n, dtype=torch.uint8, pin_memory=True)
    sym = pinned.numpy()
    sym[:] = _symbols(np.uint8, n)
    bits = np.zeros((n * L + 63) // 64, dtype=np.uint64)
    wtg.WaveletTree.build_out(sym, L, wtg.RANK, bits.ctypes.data, 0).free()
    assert np.array_equal(bits, oracle.wt_build(sym.astype(np.uint32), L)[0])
