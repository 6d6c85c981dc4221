"""Rotary embedding of many tokens and of few: the angles beside the loads, and before the wait for the kernel before."""
import pytest

import util

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16, torch.float16])
@pytest.mark.parametrize("tokens,heads,d", [(4000, 32, 128), (1200, 5, 64), (3001, 12, 128)])
def test_slices_give_the_bits_of_the_whole(dev, pkg, dtype, tokens, heads, d):
    code = {torch.float32: pkg.capi.F32, torch.bfloat16: pkg.capi.BF16, torch.float16: pkg.capi.F16}[dtype]
    g = torch.Generator(device="cuda:0")
    g.manual_seed(1)
    whole = torch.randn(tokens, heads, d, generator=g, device="cuda:0").to(dtype)
    parts, st = whole.clone(), util.cur_stream(torch)
    dev.rope(code, 1, tokens, heads, d, 7, 1e4, whole.data_ptr(), stream=st)
    for at in range(0, tokens, 77):
        n = min(77, tokens - at)
        dev.rope(code, 1, n, heads, d, 7 + at, 1e4, parts[at].data_ptr(), stream=st)
    torch.cuda.synchronize()
    assert torch.equal(whole, parts)
