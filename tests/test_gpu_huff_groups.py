"""The Huffman-shaped tree's group passes (four depths at a time) where they
can go wrong: codes that end on every depth of a group, sequences that shrink
to a few symbols, chunk edges, several nodes in a chunk, and texts that do not
start on a row boundary.  Bit-exact against the oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _fibonacci(depth, seed):
    """A text whose codes have every length up to depth (Fibonacci counts)."""
    f = [1, 1]
    while len(f) <= depth:
        f.append(f[-1] + f[-2])
    text = np.repeat(np.arange(len(f), dtype=np.uint8) * 3, f)
    np.random.default_rng(seed).shuffle(text)
    return text


def _check(t, o):
    assert (t.n, t.sigma, t.size) == (o.n, o.shape.sigma, o.shape.bv_size)
    assert np.array_equal(t.bits(), o.words[:-1])
    assert np.array_equal(t.tree()[0][:, 1], o.node_rank)


@pytest.mark.parametrize("depth", [1, 3, 4, 5, 8, 9, 12, 13, 20])
def test_code_lengths(wtg, oracle, depth):
    text = _fibonacci(depth, depth)
    o = oracle.HuffOracle(text)
    assert int(o.shape.plen.max()) == depth
    t = wtg.HuffmanTree(text)
    _check(t, o)
    t.free()


@pytest.mark.parametrize("sigma", [2, 5, 16, 17, 60, 256])
@pytest.mark.parametrize("n", [1, 31, 33, 1023, 1024, 1025, 8191, 8193, 40000])
def test_chunk_edges(wtg, oracle, sigma, n):
    rng = np.random.default_rng(n * 257 + sigma)
    text = rng.integers(0, sigma, n).astype(np.uint8) if n % 2 else \
        np.minimum(rng.zipf(1.3, n) - 1, sigma - 1).astype(np.uint8)
    t = wtg.HuffmanTree(text)
    _check(t, oracle.HuffOracle(text))
    t.free()


@pytest.mark.parametrize("shift", [1, 16, 31])
def test_text_off_a_row(wtg, oracle, shift):
    torch = pytest.importorskip("torch")
    text = _fibonacci(16, shift)[:5000]
    dev = torch.zeros(text.size + 64, dtype=torch.uint8, device="cuda")
    dev[shift:shift + text.size] = torch.from_numpy(text).cuda()
    torch.cuda.synchronize()
    t = wtg.HuffmanTree.from_device(dev.data_ptr() + shift, text.size)
    _check(t, oracle.HuffOracle(text))
    t.free()
