"""Decode attention of a few long sequences (partial results in memory, merged by a second kernel) against the CPU oracle."""
import numpy as np
import pytest

import util

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


# units (batch x KV heads) from one to a dozen, groups of 1, 4, 7 and 20 heads (two passes), ranges that leave the last CTAs short or empty
@pytest.mark.parametrize("batch,hq,hkv,seq,max_seq,d", [(1, 4, 1, 5000, 5003, 128), (1, 8, 8, 16400, 16400, 128), (2, 14, 2, 9001, 9100, 64),
                                                        (1, 20, 1, 33000, 33000, 128), (1, 1, 1, 70000, 70016, 64), (3, 16, 4, 6200, 6200, 128)])
def test_few_long_caches(dev, pkg, oracle, batch, hq, hkv, seq, max_seq, d):
    capi = pkg.capi
    q = util.to_bf16(capi, util.gen_normal(capi, (batch, hq, d), 801))
    k, v = (util.to_bf16(capi, util.gen_normal(capi, (batch, hkv, max_seq, d), 802 + i)) for i in range(2))
    k[:, :, seq:], v[:, :, seq:] = 0x7fc0, 0x7fc0  # NaN beyond the filled part: must not be read
    t = [util.dev_tensor(torch, x) for x in (q, k, v)]
    o = torch.full_like(t[0], 12345)
    for _ in range(2):  # the second call takes the first one's scratch
        dev.attention_decode(capi.BF16, batch, hq, hkv, seq, max_seq, d, *(x.data_ptr() for x in t), o.data_ptr(), stream=util.cur_stream(torch))
    torch.cuda.synchronize()
    assert dev.status() == 0
    ref, _ = oracle.attention_decode_bf16(q, k, v, seq)
    util.assert_16bit_close(oracle, oracle.bf16_to_f32(o.cpu().numpy().view(np.uint16)), ref)


def test_scratch_is_safe_with_two_streams(dev, pkg, oracle):
    """Calls on two streams at once have scratch of their own."""
    capi = pkg.capi
    hq, hkv, seq, d = 8, 2, 20000, 128
    q = [util.to_bf16(capi, util.gen_normal(capi, (1, hq, d), 811 + i)) for i in range(2)]
    k, v = (util.to_bf16(capi, util.gen_normal(capi, (1, hkv, seq, d), 815 + i)) for i in range(2))
    kd, vd = util.dev_tensor(torch, k), util.dev_tensor(torch, v)
    qd = [util.dev_tensor(torch, x) for x in q]
    od = [torch.zeros_like(x) for x in qd]
    streams = [torch.cuda.Stream() for _ in range(2)]
    torch.cuda.synchronize()
    for _ in range(20):
        for i in range(2):
            dev.attention_decode(capi.BF16, 1, hq, hkv, seq, seq, d, qd[i].data_ptr(), kd.data_ptr(), vd.data_ptr(), od[i].data_ptr(),
                                 stream=streams[i].cuda_stream)
    torch.cuda.synchronize()
    for i in range(2):
        ref, _ = oracle.attention_decode_bf16(q[i], k, v, seq)
        util.assert_16bit_close(oracle, oracle.bf16_to_f32(od[i].cpu().numpy().view(np.uint16)), ref)
