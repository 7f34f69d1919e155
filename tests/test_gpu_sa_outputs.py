"""Suffix arrays into output arrays that the sorts cannot work in: not on a 4-byte
boundary, in managed memory, and with a BWT written over it."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def made(wtg):
    torch = pytest.importorskip("torch")
    text = np.random.default_rng(8).integers(0, 5, 70001).astype(np.uint8)
    d = torch.from_numpy(text).cuda()
    bwt, sa = wtg.bwt(text, with_sa=True)
    torch.cuda.synchronize()
    return torch, d, sa, bwt, torch.cuda.current_stream().cuda_stream


@pytest.mark.parametrize("shift", [0, 1, 2, 4])
@pytest.mark.parametrize("with_bwt", [False, True])
def test_boundaries(wtg, made, shift, with_bwt):
    torch, d, sa, bwt, st = made
    n = d.numel()
    buf = torch.full((4 * n + 16,), 99, dtype=torch.uint8, device="cuda")
    out = torch.zeros(n, dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    wtg.suffix_array_device(d.data_ptr(), n, buf.data_ptr() + shift, out.data_ptr() if with_bwt else 0, st)
    got = buf.cpu().numpy()
    assert np.array_equal(got[shift:shift + 4 * n].copy().view(np.int32), np.asarray(sa).view(np.int32))
    assert (got[:shift] == 99).all() and (got[shift + 4 * n:] == 99).all()
    if with_bwt:
        assert np.array_equal(out.cpu().numpy(), bwt)


def test_bwt_over_the_suffix_array(wtg, made):
    torch, d, sa, bwt, st = made
    n = d.numel()
    buf = torch.zeros(4 * n, dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    wtg.suffix_array_device(d.data_ptr(), n, buf.data_ptr(), buf.data_ptr(), st)
    assert np.array_equal(buf.cpu().numpy()[:n], bwt)


def test_managed_memory(wtg, made):
    torch, d, sa, bwt, st = made
    n = d.numel()
    try:
        rt = ctypes.CDLL("libcudart.so.13")
    except OSError:
        pytest.skip("no shared CUDA runtime")
    p = ctypes.c_void_p()
    if rt.cudaMallocManaged(ctypes.byref(p), ctypes.c_size_t(4 * n), ctypes.c_uint(1)) != 0:
        pytest.skip("no managed memory")
    wtg.suffix_array_device(d.data_ptr(), n, p.value, 0, st)
    got = np.ctypeslib.as_array(ctypes.cast(p, ctypes.POINTER(ctypes.c_int32)), (n,))
    assert np.array_equal(got, np.asarray(sa).view(np.int32))
    rt.cudaFree(p)
