"""The BWT gathered from packed codes (alphabets of at most 16 bytes, long
texts) against the definition, at odd lengths, text buffers that do not start
on a word, and the alphabet just past the rule."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sigma,n,shift", [(5, (1 << 25) + 3, 0), (16, 1 << 25, 3), (17, (1 << 25) + 1, 0),
                                           (1, 1 << 16, 0), (16, (1 << 25) - 1, 1)])
def test_bwt_is_the_byte_before(wtg, sigma, n, shift):
    torch = pytest.importorskip("torch")
    g = torch.Generator(device="cuda")
    g.manual_seed(sigma + n)
    buf = torch.zeros(n + 8, dtype=torch.uint8, device="cuda")
    text = buf[shift:shift + n]
    text.copy_((torch.randint(0, sigma, (n,), device="cuda", generator=g) * 7 + 3).to(torch.uint8))
    sa = torch.empty(n, dtype=torch.int32, device="cuda")
    bwt = torch.empty(n, dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    wtg.suffix_array_device(text.data_ptr(), n, sa.data_ptr(), bwt.data_ptr(), torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    at = sa.long() - 1
    at[at < 0] = n - 1
    assert torch.equal(bwt, text[at])
    assert torch.equal(torch.bincount(bwt.int(), minlength=256), torch.bincount(text.int(), minlength=256))
    first = text[sa.long()]
    assert bool((first[1:] >= first[:-1]).all())
