"""f32 attention on the tcgen05 kernel against the CPU oracle."""
import numpy as np
import pytest

import util
from test_gpu_attention import run_attention
from test_gpu_attention_decode import run_prefill

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


# the tcgen05 f32 kernel: all head dims, sequences that end inside a query tile, a step, a chunk of four steps
@pytest.mark.parametrize("causal", [False, True])
@pytest.mark.parametrize("b,hq,hkv,s,d", [(1, 1, 1, 256, 128), (1, 2, 1, 257, 128), (2, 4, 2, 300, 64), (1, 3, 3, 383, 96), (1, 2, 2, 421, 32),
                                          (1, 4, 1, 1000, 128), (1, 1, 1, 2049, 64)])
def test_f32_tcgen05(dev, pkg, oracle, b, hq, hkv, s, d, causal):
    capi = pkg.capi
    q, k, v = (util.gen_normal(capi, (b, h, s, d), 751 + i) for i, h in enumerate((hq, hkv, hkv)))
    o = run_attention(dev, capi, q, k, v, capi.F32, causal)
    m = oracle.compare(o, oracle.attention_f32(q, k, v, causal))
    assert m["rel_max"] <= util.F32_REL and m["rel_fro"] <= util.F32_REL, m


def test_f32_tcgen05_growing_scores(dev, pkg, oracle):
    """Keys whose scores grow along the sequence, by more than 2^8 within a chunk of O: the chunk in tensor memory and the
    running sums are rescaled."""
    capi = pkg.capi
    s, d = 700, 64
    q = util.gen_normal(capi, (1, 2, s, d), 761)
    k = q[:, :, ::-1].copy() * np.linspace(0.1, 6.0, s, dtype=np.float32)[None, None, :, None]
    v = util.gen_normal(capi, (1, 2, s, d), 763)
    for causal in (False, True):
        o = run_attention(dev, capi, q, k, v, capi.F32, causal)
        ref = oracle.attention_f32(q, k, v, causal)
        # a score of size x carries an error of x * 2^-22 or so into its exponential: scores here reach 6 * 64 / 8 = 48
        assert oracle.compare(o, ref)["rel_fro"] <= 4 * util.F32_REL


@pytest.mark.parametrize("s,hq,hkv,d,start,max_seq", [(64, 2, 2, 128, 192, 256), (130, 6, 3, 128, 400, 700), (100, 2, 1, 64, 333, 433),
                                                      (300, 4, 4, 96, 0, 301)])
def test_f32_tcgen05_prefill(dev, pkg, oracle, s, hq, hkv, d, start, max_seq):
    capi = pkg.capi
    q = util.gen_normal(capi, (s, hq, d), 771)
    k, v = (util.gen_normal(capi, (hkv, max_seq, d), 772 + i) for i in range(2))
    k[:, start + s:], v[:, start + s:] = np.nan, np.nan  # beyond the filled part: must not be read
    o = run_prefill(dev, capi, q, k, v, start, capi.F32)
    ref = oracle.attention_prefill_f32(q, np.nan_to_num(k), np.nan_to_num(v), start, f64_acc=True)
    m = oracle.compare(o, ref)
    assert m["rel_max"] <= util.F32_REL and m["rel_fro"] <= util.F32_REL, m
