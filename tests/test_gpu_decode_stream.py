"""Decode attention on 16-bit caches as one stream of tiles: shares that begin and end inside caches, many caches to a share, many shares to a cache, whole caches,
positions that end inside a tile, what lies behind them NaN, every group up to eight heads."""
import pytest

import util

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("batch,hq,hkv,seq,spare,d", [
    (17, 32, 8, 1729, 5, 128), (5, 8, 8, 3001, 0, 128), (13, 6, 2, 4100, 1, 128), (64, 16, 8, 601, 40, 128), (1, 14, 2, 60001, 3, 64), (9, 24, 8, 2900, 100, 64), (64, 32, 8, 833, 0, 64),
    (18, 16, 8, 1, 7, 128), (37, 64, 8, 100, 0, 128), (148, 3, 1, 33, 9, 64), (74, 8, 2, 200, 0, 64), (700, 8, 8, 40, 3, 64), (3, 21, 7, 9000, 0, 128)])
def test_against_64_bits(dev, pkg, dtype, batch, hq, hkv, seq, spare, d):
    g = torch.Generator(device="cuda:0")
    g.manual_seed(seq + d)
    q = torch.randn((batch, hq, d), generator=g, device="cuda:0").to(dtype)
    k, v = (torch.randn((batch, hkv, seq + spare, d), generator=g, device="cuda:0").to(dtype) for _ in range(2))
    k[:, :, seq:], v[:, :, seq:] = float("nan"), float("nan")  # not filled yet
    o, again = torch.empty_like(q), torch.empty_like(q)
    for out in (o, again):
        dev.attention_decode(pkg.capi.BF16 if dtype == torch.bfloat16 else pkg.capi.F16, batch, hq, hkv, seq, seq + spare, d, q.data_ptr(), k.data_ptr(), v.data_ptr(), out.data_ptr(),
                             stream=util.cur_stream(torch))
    torch.cuda.synchronize()
    assert dev.status() == 0 and torch.equal(o, again)
    group = hq // hkv
    for b in range(0, batch, max(1, batch // 8)):
        kk, vv = (t[b, :, :seq].double() for t in (k, v))
        s = q[b].view(hkv, group, d).double() @ kk.transpose(1, 2) / d ** 0.5
        want = (torch.softmax(s, -1) @ vv).view(hq, d)
        # probabilities and results rounded
        assert float((o[b].double() - want).norm() / want.norm()) <= (4e-3 if dtype == torch.bfloat16 else 5e-4)


def test_far_apart_scores(dev, pkg):
    """One position outweighs all others, in one share or another; scores of -inf weigh nothing."""
    batch, hq, hkv, seq, d = 17, 32, 8, 1700, 128
    g = torch.Generator(device="cuda:0")
    g.manual_seed(1)
    q = torch.randn((batch, hq, d), generator=g, device="cuda:0").bfloat16()
    k, v = (torch.randn((batch, hkv, seq, d), generator=g, device="cuda:0").bfloat16() for _ in range(2))
    q[..., 0] = 4.0
    k[..., 0] = 0.0
    for u in range(batch * hkv):
        k[u // hkv, u % hkv, (u * 997) % seq, 0] = 300.0
        k[u // hkv, u % hkv, (u * 13 + 5) % seq, 0] = float("-inf") if (u * 13 + 5) % seq != (u * 997) % seq else 300.0
    o = torch.empty_like(q)
    dev.attention_decode(pkg.capi.BF16, batch, hq, hkv, seq, seq, d, q.data_ptr(), k.data_ptr(), v.data_ptr(), o.data_ptr(), stream=util.cur_stream(torch))
    torch.cuda.synchronize()
    assert dev.status() == 0
    for u in range(batch * hkv):
        want = v[u // hkv, u % hkv, (u * 997) % seq].float()
        assert float((o[u // hkv].view(hkv, -1, d)[u % hkv].float() - want).abs().max()) <= 2.0 ** -6
