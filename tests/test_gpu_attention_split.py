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


# starts that are no multiple of the 128-key step, and ranges so short that the last one lies wholly behind the first rows of its
# query tile: for them it holds no visible key
@pytest.mark.parametrize("dtype", ["bf16", "f16"])
@pytest.mark.parametrize("s,hq,hkv,d,start", [(256, 8, 2, 128, 32516), (100, 8, 8, 64, 36900), (256, 4, 1, 64, 32600), (100, 4, 1, 128, 78300),
                                              (100, 1, 1, 128, 34721), (100, 1, 1, 64, 34721)])
def test_prefill_rows_without_a_key_in_the_last_range(dev, pkg, oracle, s, hq, hkv, d, start, dtype):
    capi = pkg.capi
    qf = util.gen_normal(capi, (s, hq, d), 751)
    kf, vf = (util.gen_normal(capi, (hkv, start + s, d), 752 + i) for i in range(2))
    if dtype == "bf16":
        q, k, v = (util.to_bf16(capi, t) for t in (qf, kf, vf))
        wide = oracle.bf16_to_f32
    else:
        q, k, v = (util.f32_to_f16_bits(t) for t in (qf, kf, vf))
        wide = lambda t: np.ascontiguousarray(t).view(np.float16).astype(np.float32)  # noqa: E731
    o = wide(run_prefill(dev, capi, q, k, v, start, capi.BF16 if dtype == "bf16" else capi.F16).view(np.uint16))
    util.assert_16bit_close(oracle, o, oracle.attention_prefill_f32(wide(q), wide(k), wide(v), start))


# scores of -inf in a whole 128-key step, whose maximum then stays -inf: their keys weigh nothing, the others decide
@pytest.mark.parametrize("d,first", [(128, True), (64, True), (64, False), (32, True)])
def test_a_step_of_infinite_scores(dev, pkg, oracle, d, first):
    capi = pkg.capi
    q, k, v = bf16_qkv(capi, 1, 2, 1, 400, d, seed=761)
    q[..., 0] = 0x3f80                      # 1.0
    at = slice(0, 128) if first else slice(128, 256)
    k[:, :, at, 0] = 0xff80                 # -inf
    o = oracle.bf16_to_f32(run_attention(dev, capi, q, k, v, capi.BF16, False).view(np.uint16))
    keep = np.r_[0:at.start, at.stop:400]
    f = oracle.bf16_to_f32
    qf, kf, vf = f(q)[0].astype(np.float64), f(k)[0, 0, keep].astype(np.float64), f(v)[0, 0, keep].astype(np.float64)
    x = qf @ kf.T / np.sqrt(d)
    p = np.exp(x - x.max(-1, keepdims=True))
    util.assert_16bit_close(oracle, o[0], ((p / p.sum(-1, keepdims=True)) @ vf).astype(np.float32))


# a prompt in two chunks against the whole prompt in one call: the same bits while neither is split (fewer than 4096 positions) and
# both run on one kernel; beyond, the same to the rounding of sums in another order
@pytest.mark.parametrize("dtype,d,total,first,same", [
    ("bf16", 128, 4095, 3969, True), ("bf16", 128, 4095, 130, True), ("f16", 128, 4000, 3990, True), ("bf16", 64, 4095, 65, True),
    ("bf16", 96, 5000, 4500, True), ("f32", 128, 700, 300, True), ("f32", 64, 5000, 4900, True),
    ("bf16", 128, 4096, 3900, False), ("bf16", 64, 5000, 40, False), ("f32", 128, 700, 680, False)])
def test_prompt_in_chunks(dev, pkg, dtype, d, total, first, same):
    capi = pkg.capi
    code = {"bf16": capi.BF16, "f16": capi.F16, "f32": capi.F32}[dtype]
    narrow = {"bf16": lambda t: util.to_bf16(capi, t), "f16": util.f32_to_f16_bits, "f32": lambda t: t}[dtype]
    q = narrow(util.gen_normal(capi, (total, 2, d), 771))
    k, v = (narrow(util.gen_normal(capi, (1, total, d), 772 + i)) for i in range(2))
    whole = run_prefill(dev, capi, q, k, v, 0, code)
    parts = np.concatenate([run_prefill(dev, capi, np.ascontiguousarray(q[:first]), k, v, 0, code),
                            run_prefill(dev, capi, np.ascontiguousarray(q[first:]), k, v, first, code)])
    if same:
        assert np.array_equal(whole.view(np.uint8), parts.view(np.uint8))
        return
    wide = {"bf16": lambda t: (t.view(np.uint16).astype(np.uint32) << 16).view(np.float32), "f16": lambda t: t.view(np.float16), "f32": lambda t: t}[dtype]
    a, b = wide(whole).astype(np.float64), wide(parts).astype(np.float64)
    # f32: the bound of the operator; bf16: each side rounds the probabilities and the result once, 2^-9 each
    assert np.linalg.norm(a - b) <= (1e-5 if dtype == "f32" else 2.0 ** -7) * np.linalg.norm(a)
