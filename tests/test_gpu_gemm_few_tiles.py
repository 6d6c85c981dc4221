"""16-bit GEMMs of few rows or few tiles on the GPU, through the C ABI, against the CPU oracle."""
import numpy as np
import pytest

import util
from test_gpu_gemm_odd import run

pytestmark = pytest.mark.gpu


# few rows of A, or too few tiles for CTA pairs: each width of the token side at its edges, split and unsplit K, ragged everything
@pytest.mark.parametrize("bt", [False, True])
@pytest.mark.parametrize("m,n,k,batch", [(1, 8, 8, 1), (1, 4096, 4096, 1), (15, 136, 200, 3), (16, 256, 1024, 1), (17, 1000, 520, 1),
                                         (32, 128, 64, 2), (33, 384, 8192, 1), (64, 200, 1544, 1), (65, 520, 456, 2),
                                         (128, 1024, 2048, 1), (129, 136, 4104, 1), (300, 2048, 512, 1), (700, 100 * 8, 264, 1),
                                         (2000, 64, 320, 1), (16, 64 * 512, 72, 1)])
def test_bf16_few_tiles(dev, pkg, oracle, m, n, k, batch, bt):
    capi = pkg.capi
    sigma = k ** -0.25
    a = util.to_bf16(capi, util.gen_normal(capi, (batch, m, k), 611, sigma))
    b = util.to_bf16(capi, util.gen_normal(capi, (batch, n, k) if bt else (batch, k, n), 612, sigma))
    c = run(dev, capi, capi.BF16, a, b, m, n, k, bt, batch=batch).view(np.uint16)
    c32 = run(dev, capi, capi.BF16, a, b, m, n, k, bt, batch=batch, out_f32=True)
    for i in range(batch):
        ref, _ = oracle.gemm_bf16(a[i], b[i], bt)
        util.assert_16bit_close(oracle, oracle.bf16_to_f32(c[i]), ref)
        mt = oracle.compare(c32[i], ref)
        assert mt["rel_max"] <= util.F32_REL and mt["rel_fro"] <= util.F32_REL, mt  # f32 sums of exact products


def test_f16_few_tiles_into_a_wider_matrix(dev, pkg, oracle):
    capi = pkg.capi
    m, n, k, ldc = 20, 264, 1032, 280
    af, bf = (util.gen_normal(capi, s, 621, k ** -0.25) for s in ((m, k), (n, k)))
    a, b = util.f32_to_f16_bits(af), util.f32_to_f16_bits(bf)
    c = run(dev, capi, capi.F16, a, b, m, n, k, True, ldc=ldc)[0]
    assert (c[:, n:] == 7).all()
    ref = oracle.gemm_f32(a.view(np.float16).astype(np.float32), b.view(np.float16).astype(np.float32), True, f64_acc=True)
    util.assert_16bit_close(oracle, np.ascontiguousarray(c[:, :n]).view(np.float16).astype(np.float32), ref)
