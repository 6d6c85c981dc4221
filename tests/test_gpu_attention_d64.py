"""16-bit attention with heads of 64 and 32 against the CPU oracle."""
import numpy as np
import pytest

import util
from test_gpu_attention import bf16_qkv, run_attention
from test_gpu_attention_decode import run_prefill

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("causal", [False, True])
@pytest.mark.parametrize("b,hq,hkv,s,d", [(1, 1, 1, 1, 64), (1, 2, 1, 127, 64), (2, 2, 2, 128, 64), (1, 4, 2, 129, 64), (1, 2, 2, 257, 64),
                                          (1, 2, 1, 1000, 64), (1, 2, 2, 384, 32), (1, 2, 1, 261, 32)])
def test_heads_up_to_64(dev, pkg, oracle, b, hq, hkv, s, d, causal):
    capi = pkg.capi
    q, k, v = bf16_qkv(capi, b, hq, hkv, s, d, seed=701)
    o = run_attention(dev, capi, q, k, v, capi.BF16, causal).view(np.uint16)
    ref, _ = oracle.attention_bf16(q, k, v, causal)
    got = oracle.bf16_to_f32(o)
    util.assert_16bit_close(oracle, got, ref)
    # the probabilities keep f32 precision (hi + lo): what is left is the rounding of the result, half a unit in its last
    # place at most, plus an f32 error far below it
    assert (np.abs(got - ref) <= 2.0 ** -8 * np.abs(ref) * (1 + 2.0 ** -5) + 2e-5).all()


@pytest.mark.parametrize("causal", [False, True])
def test_f16_heads_of_64(dev, pkg, oracle, causal):
    capi = pkg.capi
    t = [util.f32_to_f16_bits(util.gen_normal(capi, (1, 2, 333, 64), 711 + i)) for i in range(3)]
    got = run_attention(dev, capi, *t, capi.F16, causal).view(np.float16).astype(np.float32)
    ref = oracle.attention_f32(*(x.view(np.float16).astype(np.float32) for x in t), causal)
    assert (np.abs(got - ref) <= 2.0 ** -11 * np.abs(ref) * (1 + 2.0 ** -5) + 2e-5).all()


@pytest.mark.parametrize("s,hq,hkv,d,start,max_seq", [(1, 2, 2, 64, 0, 8), (130, 4, 1, 64, 77, 300), (257, 2, 2, 32, 128, 400)])
def test_prefill_heads_up_to_64(dev, pkg, oracle, s, hq, hkv, d, start, max_seq):
    capi = pkg.capi
    q = util.to_bf16(capi, util.gen_normal(capi, (s, hq, d), 721))
    k, v = (util.to_bf16(capi, util.gen_normal(capi, (hkv, max_seq, d), 722 + i)) for i in range(2))
    f = oracle.bf16_to_f32
    o = run_prefill(dev, capi, q, k, v, start, capi.BF16).view(np.uint16)
    util.assert_16bit_close(oracle, f(o), oracle.attention_prefill_f32(f(q), f(k), f(v), start))


@pytest.mark.parametrize("s", [3000, 9000])
def test_f16_a_long_tail_of_small_probabilities(dev, pkg, s):
    """One key that outweighs each of the others 2^26 times, far below f16's smallest number, but carries no value: the
    others decide.  Their probabilities are taken to 2^-32 of the largest, that is to 2^-6 of themselves."""
    capi = pkg.capi
    q, k, v = (np.zeros((1, 1, s, 64), np.float32) for _ in range(3))
    q[..., 0] = 8                       # scores: q . k / 8
    k[0, 0, 1:, 0] = -26 * np.log(2)
    v[0, 0, 1:] = 100
    got = run_attention(dev, capi, *(util.f32_to_f16_bits(t) for t in (q, k, v)), capi.F16, False).view(np.float16).astype(np.float64)
    p = np.exp(np.float64(k.astype(np.float16)[0, 0, 1, 0]))
    want = 100 * (s - 1) * p / (1 + (s - 1) * p)
    assert (np.abs(got - want) <= 2.0 ** -6 * want).all(), (got.min(), got.max(), want)
