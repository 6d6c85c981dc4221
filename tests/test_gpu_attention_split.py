"""16-bit attention with the KV steps of a query block dealt to several CTAs, against the CPU oracle."""
import numpy as np
import pytest

import util
from test_gpu_attention import bf16_qkv, run_attention
from test_gpu_attention_decode import run_prefill

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


# 2 to 8 CTAs per query block; lengths that leave the last CTA a short range
@pytest.mark.parametrize("s,hq,hkv,d,start", [(100, 4, 2, 128, 4001), (300, 8, 2, 128, 5000), (200, 4, 4, 128, 8200), (17, 2, 1, 128, 16500),
                                              (129, 2, 2, 64, 9000), (40, 3, 1, 64, 17000)])
def test_prefill_steps_over_several_CTAs(dev, pkg, oracle, s, hq, hkv, d, start):
    capi = pkg.capi
    max_seq = start + s + 3
    q = util.to_bf16(capi, util.gen_normal(capi, (s, hq, d), 731))
    k, v = (util.to_bf16(capi, util.gen_normal(capi, (hkv, max_seq, d), 732 + i)) for i in range(2))
    k[:, -3:], v[:, -3:] = 0x7fc0, 0x7fc0  # NaN beyond the filled part: must not be read
    o = run_prefill(dev, capi, q, k, v, start, capi.BF16).view(np.uint16)
    f = oracle.bf16_to_f32
    kz, vz = np.nan_to_num(f(k)), np.nan_to_num(f(v))
    util.assert_16bit_close(oracle, f(o), oracle.attention_prefill_f32(f(q), kz, vz, start))


# causal: the first query blocks have fewer steps than CTAs, so that some get an empty range
@pytest.mark.parametrize("hq,s,d,causal", [(1, 8300, 128, True), (1, 8300, 64, True), (2, 4200, 128, False), (1, 5000, 64, False)])
def test_attention_steps_over_several_CTAs(dev, pkg, oracle, hq, s, d, causal):
    capi = pkg.capi
    q, k, v = bf16_qkv(capi, 1, hq, 1, s, d, seed=741)
    o = oracle.bf16_to_f32(run_attention(dev, capi, q, k, v, capi.BF16, causal).view(np.uint16))
    for row0, rows in ((0, 300), (s // 2, 64), (s - 200, 200)):
        ref, _ = oracle.attention_bf16(q, k, v, causal, row0, rows)
        util.assert_16bit_close(oracle, np.ascontiguousarray(o[:, :, row0:row0 + rows]), ref)
