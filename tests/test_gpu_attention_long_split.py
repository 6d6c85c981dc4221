"""Few query blocks on long caches: the KV steps of a block on many CTAs, ranges of unequal length, ranges behind a row's last key."""
import pytest

import util

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("new,start,hq,hkv,d", [(1, 8191, 4, 2, 128), (30, 9000, 4, 4, 128), (200, 16000, 8, 4, 128), (300, 8300, 2, 1, 128), (17, 20011, 2, 2, 64),
                                                (257, 8000, 4, 2, 64), (129, 12345, 2, 1, 32)])
def test_prefill_against_64_bits(dev, pkg, dtype, new, start, hq, hkv, d):
    g = torch.Generator(device="cuda:0")
    g.manual_seed(new)
    total = start + new
    mk = lambda *s: torch.randn(s, generator=g, device="cuda:0").to(dtype)  # noqa: E731
    q, k, v = mk(new, hq, d), mk(hkv, total + 5, d), mk(hkv, total + 5, d)
    k[:, total:], v[:, total:] = float("nan"), float("nan")  # not filled yet
    o = torch.empty_like(q)
    code = pkg.capi.BF16 if dtype == torch.bfloat16 else pkg.capi.F16
    call = lambda out: dev.attention_prefill(code, hq, hkv, new, start, total + 5, d, q.data_ptr(), k.data_ptr(), v.data_ptr(), out.data_ptr(),  # noqa: E731
                                             stream=util.cur_stream(torch))
    call(o)
    again = torch.empty_like(q)
    call(again)
    torch.cuda.synchronize()
    assert dev.status() == 0
    kk, vv = (t[:, :total].double().repeat_interleave(hq // hkv, 0) for t in (k, v))
    s = q.double().transpose(0, 1) @ kk.transpose(1, 2) / d ** 0.5
    seen = torch.arange(total, device="cuda:0")[None, :] <= start + torch.arange(new, device="cuda:0")[:, None]
    want = (torch.softmax(s.masked_fill(~seen, float("-inf")), -1) @ vv).transpose(0, 1)
    assert float((o.double() - want).norm() / want.norm()) <= (4e-3 if dtype == torch.bfloat16 else 5e-4)  # probabilities and results rounded
    assert torch.equal(o, again)
