"""16-bit attention whose query blocks end in their first tile of 128 rows, or have no second one, against 64 bits; rows are the same bits wherever a
block starts."""
import pytest

import util

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def rnd(g, dtype, *shape):
    return torch.randn(shape, generator=g, device="cuda:0").to(dtype)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("causal", [False, True])
@pytest.mark.parametrize("batch,hq,hkv,seq,d", [(1, 2, 1, 1, 128), (2, 4, 2, 128, 128), (1, 2, 2, 129, 128), (1, 16, 4, 384, 128), (1, 3, 3, 385, 128), (1, 40, 10, 700, 128),
                                                (1, 2, 1, 128, 64), (1, 8, 2, 300, 64), (2, 30, 10, 641, 64), (1, 4, 4, 513, 32)])
def test_against_64_bits(dev, pkg, dtype, causal, batch, hq, hkv, seq, d):
    g = torch.Generator(device="cuda:0")
    g.manual_seed(seq + d)
    q, k, v = rnd(g, dtype, batch, hq, seq, d), rnd(g, dtype, batch, hkv, seq, d), rnd(g, dtype, batch, hkv, seq, d)
    o, again = torch.empty_like(q), torch.empty_like(q)
    for out in (o, again):
        dev.attention(pkg.capi.BF16 if dtype == torch.bfloat16 else pkg.capi.F16, batch, hq, hkv, seq, d, q.data_ptr(), k.data_ptr(), v.data_ptr(), out.data_ptr(),
                      causal=causal, stream=util.cur_stream(torch))
    torch.cuda.synchronize()
    assert dev.status() == 0 and torch.equal(o, again)
    kk, vv = (t.double().repeat_interleave(hq // hkv, 1) for t in (k, v))
    s = q.double() @ kk.transpose(2, 3) / d ** 0.5
    if causal:
        s = s.masked_fill(~torch.tril(torch.ones(seq, seq, dtype=torch.bool, device="cuda:0")), float("-inf"))
    want = torch.softmax(s, -1) @ vv
    # probabilities and results rounded
    assert float((o.double() - want).norm() / want.norm()) <= (4e-3 if dtype == torch.bfloat16 else 5e-4)


@pytest.mark.parametrize("hq,hkv,new,start,d", [(4, 4, 30, 3000, 128), (32, 8, 128, 900, 128), (2, 1, 100, 9000, 128), (8, 4, 129, 1000, 128), (4, 2, 128, 700, 64), (4, 2, 17, 8200, 64)])
def test_chunks_of_a_prompt(dev, pkg, hq, hkv, new, start, d):
    g = torch.Generator(device="cuda:0")
    g.manual_seed(new + start)
    total = start + new
    q, k, v = rnd(g, torch.bfloat16, new, hq, d), rnd(g, torch.bfloat16, hkv, total + 3, d), rnd(g, torch.bfloat16, hkv, total + 3, d)
    k[:, total:], v[:, total:] = float("nan"), float("nan")  # not filled yet
    o = torch.empty_like(q)

    def call(rows, first, out):
        dev.attention_prefill(pkg.capi.BF16, hq, hkv, rows.shape[0], first, total + 3, d, rows.data_ptr(), k.data_ptr(), v.data_ptr(), out.data_ptr(), stream=util.cur_stream(torch))

    call(q, start, o)
    kk, vv = (t[:, :total].double().repeat_interleave(hq // hkv, 0) for t in (k, v))
    seen = torch.arange(total, device="cuda:0")[None, :] <= start + torch.arange(new, device="cuda:0")[:, None]
    want = (torch.softmax((q.double().transpose(0, 1) @ kk.transpose(1, 2) / d ** 0.5).masked_fill(~seen, float("-inf")), -1) @ vv).transpose(0, 1)
    torch.cuda.synchronize()
    assert dev.status() == 0 and float((o.double() - want).norm() / want.norm()) <= 4e-3
    if total < 4096:  # not split: the same bits in two calls
        first, second = q[:new // 2].contiguous(), q[new // 2:].contiguous()
        o1, o2 = torch.empty_like(first), torch.empty_like(second)
        call(first, start, o1), call(second, start + new // 2, o2)
        torch.cuda.synchronize()
        assert torch.equal(o, torch.cat([o1, o2]))
