"""The workloads this framework's speed is measured on: what its users call,
from the smallest calls to the largest, through the public entry points
(wtg.py and the C ABI of include/wtg.h).

  wt        WT(s, sigma) on a host array: the drop-in for levelWT's WT(), the
            smallest and most frequent call (latency and launches count)
  wt_int    WaveletTree(seq) on a host array with every table read back: the
            drop-in for building an sdsl::wt_int and storing it
  tree      a tree (re)built from device memory, outputs left on the device:
            byte texts, DNA codes, 16- and 32-bit integers, 3 to 20 levels, n
            a multiple of 512 or not; with the select supports, a batch of
            per-level selects is asked of it (the tables' own sizes follow
            from the data)
  bv        rank_support_v and select_support_mcl built over a device
            bit_vector, then select1 / select0 queries through them
  query     batches of wt_int queries on device arrays over a built tree
  ask       a few wt_int queries from host arrays (an interactive caller)
  sa        suffix array and BWT of a device text
  fm_build  the reference FM-index's own tree, wt_huff over the bytes of a
            text's BWT, built and asked for a batch of pattern counts
  fm_count  backward-search counts over the balanced tree of a BWT

Every output is made of whole numbers: they are exact, there is no rounding.
"""
import ctypes
import math
import os
import sys

import numpy as np
import torch

HERE = os.path.dirname(os.path.abspath(__file__))
PKG = os.path.join(os.path.dirname(HERE), "wavelet-suffix-fm-index_gb300")
if PKG not in sys.path:
    sys.path.insert(0, PKG)

import wtg  # noqa: E402

DEV = "cuda"

# data: symbols, their bytes and the tree's levels
#   zipf   byte text, Zipf(1.0) over 256 values under a random permutation
#   dna    order-2 Markov over ACGT codes with runs of N, 5 codes
#   u12    uniform 12-bit values in 16-bit symbols
#   exp    32-bit values, exponential with mean 2^14 below 2^20
DATA = {"zipf": (1, 8), "dna": (1, 3), "u12": (2, 12), "exp": (4, 20)}


def listed():
    return [
        # WT() of one short byte text: a caller that builds a tree per document
        {"name": "wt_1000", "kind": "wt", "data": "zipf", "n": 1000},
        # an integer sequence of some tens of thousands, every table stored
        {"name": "wt_int_70001", "kind": "wt_int", "data": "u12", "n": 70001},
        # byte text of 2^24 symbols, tree and rank table
        {"name": "tree_bytes_2p24", "kind": "tree", "data": "zipf", "n": 1 << 24, "flags": 1},
        # integers of a database column, 10^7 of them, all supports
        {"name": "tree_exp_1e7", "kind": "tree", "data": "exp", "n": 10_000_000, "flags": 7},
        # a genome's codes: 404 million symbols, an odd number of 512-blocks
        {"name": "tree_dna_404m", "kind": "tree", "data": "dna", "n": 403_927_746, "flags": 7},
        # the large integer tree: 2^30 symbols, 20 levels, all supports
        {"name": "tree_exp_2p30", "kind": "tree", "data": "exp", "n": 1 << 30, "flags": 7},
        # supports over a text-sized bit_vector, then a batch of selects
        {"name": "bv_842m", "kind": "bv", "size": 842_215_217, "density": 0.5, "nq": 1 << 20},
        # 2^26 random access queries on the large integer tree
        {"name": "access_2p26", "kind": "query", "op": "access", "data": "exp", "n": 1 << 30, "nq": 1 << 26},
        # a thousand access, rank and select queries from host arrays
        {"name": "ask_1000", "kind": "ask", "data": "zipf", "n": 1 << 24, "nq": 1000},
        # suffix array and BWT of 128 million DNA symbols
        {"name": "sa_dna_134m", "kind": "sa", "data": "dna", "n": (1 << 27) + 13},
        # wt_huff over the BWT of a byte text, and 2^20 counts
        {"name": "fm_build_67m", "kind": "fm_build", "data": "zipf", "n": (1 << 26) + 77, "nq": 1 << 20},
        # 2^24 pattern counts over a 2^28-symbol DNA BWT
        {"name": "fm_count_2p24", "kind": "fm_count", "data": "dna", "n": 1 << 28, "nq": 1 << 24},
    ]


def _log(rng, lo, hi):
    """A whole number spread over the logarithm of [2^lo, 2^hi]; every other one odd."""
    v = int(2.0 ** rng.uniform(lo, hi))
    return v | 1 if rng.random() < 0.5 else max(1, v)


def draw(rng):
    kind = rng.choice(["wt", "wt_int", "tree", "tree", "tree", "bv", "query", "query", "ask", "sa", "fm_build",
                       "fm_count"])
    if kind == "wt":
        return {"kind": kind, "data": rng.choice(["zipf", "dna", "u12"]), "n": _log(rng, 5, 18)}
    if kind == "wt_int":
        return {"kind": kind, "data": rng.choice(["zipf", "dna", "u12", "exp"]), "n": _log(rng, 8, 20)}
    if kind == "tree":
        n = _log(rng, 18, 28.5)
        if rng.random() < 0.3:
            n = max(512, n // 512 * 512)
        return {"kind": kind, "data": rng.choice(sorted(DATA)), "n": n, "flags": rng.choice([0, 1, 7, 7])}
    if kind == "bv":
        return {"kind": kind, "size": _log(rng, 20, 31), "density": rng.choice([0.5, 0.2, 0.03]),
                "nq": _log(rng, 14, 22)}
    if kind == "query":
        return {"kind": kind, "op": rng.choice(["access", "rank", "lex_count", "range_count"]),
                "data": rng.choice(["zipf", "u12", "exp"]), "n": _log(rng, 22, 28), "nq": _log(rng, 14, 24)}
    if kind == "ask":
        return {"kind": kind, "data": rng.choice(["zipf", "dna", "exp"]), "n": _log(rng, 16, 24),
                "nq": _log(rng, 0, 13)}
    if kind == "sa":
        return {"kind": kind, "data": rng.choice(["dna", "dna", "zipf"]), "n": _log(rng, 16, 26.5)}
    if kind == "fm_build":
        return {"kind": kind, "data": rng.choice(["zipf", "dna"]), "n": _log(rng, 18, 26), "nq": _log(rng, 10, 20)}
    return {"kind": kind, "data": rng.choice(["dna", "zipf"]), "n": _log(rng, 20, 26), "nq": _log(rng, 14, 22)}


# ------------------------------------------------------------------ inputs

def _gen(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed))
    return g


def _symbols(data, n, seed):
    """n symbols on the device (uint8, int16 or int32 storage)."""
    g = _gen(seed)
    if data == "dna":
        return _dna(n, g)
    out = torch.empty(n, dtype={"zipf": torch.uint8, "u12": torch.int16, "exp": torch.int32}[data], device=DEV)
    step = 1 << 27
    if data == "zipf":
        p = 1.0 / torch.arange(1, 257, dtype=torch.float64, device=DEV)
        cdf = (torch.cumsum(p, 0) / p.sum()).float()
        perm = torch.randperm(256, device=DEV, generator=g).to(torch.uint8)
    for o in range(0, n, step):
        m = min(step, n - o)
        if data == "u12":
            out[o:o + m] = torch.randint(0, 4096, (m,), device=DEV, generator=g, dtype=torch.int32).to(torch.int16)
            continue
        x = torch.empty(m, dtype=torch.float32, device=DEV)
        if data == "exp":
            out[o:o + m] = x.exponential_(2.0 ** -14, generator=g).floor_().clamp_(max=2 ** 20 - 1).to(torch.int32)
        else:
            r = torch.searchsorted(cdf, x.uniform_(generator=g), right=True).clamp_(max=255)
            out[o:o + m] = perm[r]
    return out


def _dna(n, g):
    """Codes 0..4 (A C G N T): order-2 chains of 256 symbols each from a
    uniform start, 0.1 % N in runs of 1 to 100."""
    block = 256
    nb = (n + block - 1) // block
    trans = torch.empty((16, 4), device=DEV).exponential_(generator=g)
    cdf = torch.cumsum(trans / trans.sum(1, keepdim=True), 1)[:, :3].contiguous()
    ctx = torch.randint(0, 16, (nb,), device=DEV, generator=g)
    codes = torch.empty((block, nb), dtype=torch.uint8, device=DEV)
    for i in range(block):
        u = torch.rand((nb, 1), device=DEV, generator=g)
        c = (u > cdf[ctx]).sum(1)
        codes[i] = c
        ctx = (ctx % 4) * 4 + c
    lut = torch.tensor([0, 1, 2, 4], dtype=torch.uint8, device=DEV)
    text = torch.empty(nb * block, dtype=torch.uint8, device=DEV)
    step = 1 << 18  # blocks at a time
    for o in range(0, nb, step):
        part = codes[:, o:o + step]
        text[o * block:(o + part.shape[1]) * block] = lut[part.t().reshape(-1).long()]
    text = text[:n].contiguous()
    runs = int(n * 0.001 / 50.5)
    if runs and n > 200:
        ln = torch.randint(1, 101, (runs, 1), device=DEV, generator=g)
        st = torch.randint(0, n - 100, (runs, 1), device=DEV, generator=g)
        span = torch.arange(100, device=DEV)[None]
        text[(st + span)[span < ln]] = 3
    return text


def _host(t):
    a = t.cpu().numpy()
    return a.view({1: np.uint8, 2: np.uint16, 4: np.uint32}[a.dtype.itemsize])


def _patterns(text, nq, seed):
    """nq patterns of 8 to 32 symbols copied from the text: (symbols, offsets)."""
    g = _gen(seed + 7)
    n = text.numel()
    lens = torch.randint(8, 33, (nq,), device=DEV, generator=g)
    start = torch.randint(0, max(1, n - 32), (nq,), device=DEV, generator=g)
    off = torch.zeros(nq + 1, dtype=torch.int64, device=DEV)
    off[1:] = torch.cumsum(lens, 0)
    base = torch.repeat_interleave(start - off[:-1], lens)
    base += torch.arange(base.numel(), device=DEV)
    return text[base].contiguous(), off


def _bwt_of(text, stream):
    bw = torch.empty_like(text)
    wtg.suffix_array_device(text.data_ptr(), text.numel(), 0, bw.data_ptr(), stream)
    return bw


class State:
    tree = None
    bv = None


def prepare(case, seed):
    s = State()
    s.case, s.kind = case, case["kind"]
    s.stream = torch.cuda.current_stream().cuda_stream
    kind, n = s.kind, case.get("n")
    if kind in ("wt", "wt_int"):
        s.seq = _host(_symbols(case["data"], n, seed))
        return s
    if kind == "tree":
        s.seq = _symbols(case["data"], n, seed)
        if case["flags"] == wtg.ALL:
            nq, g = _level_queries(n), _gen(seed + 5)
            s.level = torch.randint(0, DATA[case["data"]][1], (nq,), device=DEV, generator=g)
            s.k = torch.randint(1, n + 1, (nq,), device=DEV, generator=g)
        return s
    if kind == "bv":
        size, g = case["size"], _gen(seed)
        nw = (size + 63) // 64
        words = torch.zeros(nw, dtype=torch.int64, device=DEV)
        step = 1 << 22
        weight = (torch.ones(64, dtype=torch.int64, device=DEV) << torch.arange(64, device=DEV))[None]
        for o in range(0, nw, step):
            m = min(step, nw - o)
            b = torch.rand((m, 64), device=DEV, generator=g) < case["density"]
            words[o:o + m] = (b * weight).sum(1)
        if size & 63:  # bits past the end are zero
            words[-1] &= (1 << (size & 63)) - 1
        s.words = words
        lo = int(size * min(case["density"], 1 - case["density"]) * 0.9) + 1  # fewer than either polarity has
        s.k = torch.randint(1, lo + 1, (case["nq"],), device=DEV, generator=g)
        return s
    if kind == "sa":
        s.text = _symbols(case["data"], n, seed)
        s.sa = torch.empty(n, dtype=torch.int32, device=DEV)
        s.bwt = torch.empty(n, dtype=torch.uint8, device=DEV)
        return s
    if kind in ("query", "ask"):
        eb, levels = DATA[case["data"]]
        seq = _symbols(case["data"], n, seed)
        s.tree = wtg.WaveletTree.from_device(seq.data_ptr(), n, eb, levels, wtg.ALL, s.stream)
        s.tree.sync()
        nq, g = case["nq"], _gen(seed + 3)
        idx = torch.randint(0, n, (nq,), device=DEV, generator=g)
        sym = seq[torch.randint(0, n, (nq,), device=DEV, generator=g)].long()
        if kind == "ask":
            s.idx, s.sym = (x.cpu().numpy().astype(np.uint64) for x in (idx, sym))
            occ = s.tree.rank(np.full(nq, n), s.sym)
            s.ith = (s.idx % occ) + np.uint64(1)  # an occurrence that exists
            return s
        s.idx, s.sym = idx, sym
        if case["op"] in ("lex_count", "range_count"):
            s.end = torch.clamp(idx + torch.randint(0, 1 << 20, (nq,), device=DEV, generator=g), max=n - 1)
            half = 1 << max(0, levels - 8)
            s.vlo, s.vhi = torch.clamp(sym - half, min=0), sym + half
        s.out = [torch.empty(nq, dtype=torch.int64, device=DEV) for _ in range(3 if case["op"] == "lex_count" else 1)]
        return s
    # fm_build, fm_count: a text, its BWT and patterns from it
    text = _symbols(case["data"], n, seed)
    text = text + (text < 255).to(torch.uint8)  # 0 is free for the unique last symbol
    text[-1] = 0
    s.bwt = _bwt_of(text, s.stream)
    s.sigma = 256 if case["data"] == "zipf" else 6
    s.pat, s.off = _patterns(text[:-1], case["nq"], seed)
    hist = torch.bincount(text[: 1 << 28].int(), minlength=256)
    for o in range(1 << 28, n, 1 << 28):
        hist += torch.bincount(text[o:o + (1 << 28)].int(), minlength=256)
    s.C = torch.zeros(256, dtype=torch.int64, device=DEV)
    s.C[1:] = torch.cumsum(hist, 0)[:-1]
    s.out = torch.empty(case["nq"], dtype=torch.int64, device=DEV)
    if kind == "fm_count":
        s.fm = wtg.FMIndex.from_device(s.bwt.data_ptr(), n, s.sigma, s.stream)
    return s


# -------------------------------------------------------------------- runs

class _Mem:
    def __init__(self, owner, ptr, words):
        self.owner = owner  # the words live as long as the tree that owns them
        self.__cuda_array_interface__ = {"data": (ptr, False), "shape": (words,), "typestr": "<i8", "version": 2}


def _words(tree, ptr, words):
    """The tree's own device words as a tensor (no copy)."""
    return torch.as_tensor(_Mem(tree, ptr, words), device=DEV) if words else torch.empty(0, dtype=torch.int64, device=DEV)


def _level_queries(n):
    """Per-level selects asked of a tree of n symbols."""
    return min(1 << 18, max(1 << 10, n // 64))


def _run_tree(s):
    c = s.case
    eb, levels = DATA[c["data"]]
    t = wtg.WaveletTree.from_device(s.seq.data_ptr(), c["n"], eb, levels, c["flags"], s.stream, tree=s.tree)
    t.sync()
    s.tree = t
    p = t.device_ptrs()
    out = {"bits": _words(t, p[0], t.bit_words)}
    if c["flags"] & wtg.RANK:
        out["rank"] = _words(t, p[1], t.rank_words)
    if c["flags"] == wtg.ALL:
        for t_b in (1, 0):
            got = torch.empty_like(s.k)
            t.level_select_device(t_b, s.level.data_ptr(), s.k.data_ptr(), s.k.numel(), got.data_ptr(), s.stream)
            out["select%d" % t_b] = got
    return out


def _tables(t, t_b):
    """m_superblock, the descriptors and the pool in arrays that every
    sequence of this length fits in (a caller's preallocated buffers)."""
    x = t.select_tables(t_b)
    sb = x.size // 4096 + 2
    out = []
    for a, room in ((x.sb_words, sb), (x.desc, sb), (x.pool, 32 * sb + x.size // 256 + 4096)):
        b = np.zeros(room, dtype=np.uint64)
        b[: a.size] = a
        out.append(b)
    return out


def _run_bv(s):
    c, L = s.case, wtg.lib()
    if s.bv is None:
        s.bv = _Bv()
    wtg._ck(L.wtg_bv_build_device(s.words.data_ptr(), c["size"], wtg.ALL, s.stream, ctypes.byref(s.bv.h)))
    out = [torch.empty_like(s.k) for _ in range(2)]
    for t_b in (1, 0):
        wtg._ck(L.wtg_bv_select_device(s.bv.h, t_b, s.k.data_ptr(), c["nq"], out[t_b].data_ptr(), s.stream))
    wtg._ck(L.wtg_bv_sync(s.bv.h))
    return out


class _Bv:
    """A support handle that a program keeps for rebuilds."""

    def __init__(self):
        self.h = ctypes.c_void_p()

    def __del__(self):
        if self.h:
            wtg.lib().wtg_bv_free(self.h)


def run(s):
    c, kind = s.case, s.kind
    if kind == "wt":
        nodes, bits = wtg.WT(s.seq, 1 << DATA[c["data"]][1])
        return [nodes, bits]
    if kind == "wt_int":
        t = wtg.WaveletTree(s.seq)
        out = [t.bits(), t.rank_table(), *_tables(t, 1), *_tables(t, 0)]
        t.free()
        return out
    if kind == "tree":
        return _run_tree(s)
    if kind == "bv":
        return _run_bv(s)
    if kind == "ask":
        return [s.tree.access(s.idx), s.tree.rank(s.idx, s.sym), s.tree.select(s.ith, s.sym)]
    if kind == "query":
        t, nq, st, op = s.tree, c["nq"], s.stream, c["op"]
        o = [x.data_ptr() for x in s.out]
        if op == "access":
            t.access_device(s.idx.data_ptr(), nq, o[0], st)
        elif op == "rank":
            t.rank_device(s.idx.data_ptr(), s.sym.data_ptr(), nq, o[0], st)
        elif op == "lex_count":
            t.lex_count_device(s.idx.data_ptr(), s.end.data_ptr(), s.sym.data_ptr(), nq, *o, st)
        else:
            t.range_count_device(s.idx.data_ptr(), s.end.data_ptr(), s.vlo.data_ptr(), s.vhi.data_ptr(), nq, o[0], st)
        return s.out
    if kind == "sa":
        wtg.suffix_array_device(s.text.data_ptr(), c["n"], s.sa.data_ptr(), s.bwt.data_ptr(), s.stream)
        return [s.sa, s.bwt]
    if kind == "fm_build":
        h = wtg.HuffmanTree.from_device(s.bwt.data_ptr(), c["n"], wtg.ALL, s.stream)
        h.fm_count_device(s.C.data_ptr(), s.pat.data_ptr(), s.off.data_ptr(), c["nq"], s.out.data_ptr(), s.stream)
        size = h.size
        h.free()
        return [s.out, size]
    s.fm.count_device(s.C.data_ptr(), s.pat.data_ptr(), s.off.data_ptr(), c["nq"], s.out.data_ptr(), s.stream)
    return s.out


# -------------------------------------------------------------------- work

def _table_bytes(bits, flags):
    """rank_support_v, and per polarity a mini block entry (a bit position
    within a few thousand: 13 bits) for every 64th arg of half the bits."""
    rank = 16 * (bits // 512 + 1) if flags & 1 else 0
    return rank + bin(flags >> 1).count("1") * (bits / 2 / 64 * 13 / 8)


def work(case):
    """What a pass cannot do without: inputs read once, outputs written once."""
    kind, n = case["kind"], case.get("n")
    eb, levels = DATA.get(case.get("data"), (0, 0))
    if kind == "wt":
        b = n * eb + n * levels / 8 + 2 * (1 << levels) * 20
    elif kind in ("tree", "wt_int"):
        flags = case.get("flags", 7)
        b = n * eb + n * levels / 8 + _table_bytes(n * levels, flags)
        if kind == "tree" and flags == 7:
            b += 2 * 24 * _level_queries(n)
    elif kind == "bv":
        b = case["size"] / 8 + _table_bytes(case["size"], 7) + 2 * 16 * case["nq"]
    elif kind in ("query", "ask"):
        # arguments in, answers out, and per query and level a word of bits
        # and a rank entry, or the whole tree once where that is less
        args = {"access": 2, "rank": 3, "lex_count": 6, "range_count": 5}.get(case.get("op"), 8)
        b = 8 * args * case["nq"] + min(24 * levels * case["nq"], n * levels / 8 * 1.25)
    elif kind == "sa":
        b = n * (1 + 4 + 1)
    else:
        avg = {"zipf": 6.3, "dna": 2.1}[case["data"]] if kind == "fm_build" else levels
        tree = n * avg / 8 * 1.25
        counts = case["nq"] * (16 + 20)
        b = counts + min(tree, case["nq"] * 20 * avg * 48) if kind == "fm_count" else n + 1.1 * tree + counts
    return {"bytes": float(math.ceil(b)), "flops": 0.0}
