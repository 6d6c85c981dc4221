"""16-bit GEMMs of odd sizes with few products and a K of 128 and more: padded copies instead of the FP32 pipe."""
import numpy as np
import pytest

import util
from test_gpu_gemm_odd import run

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,n,k,bt,batch,ldc", [
    (20, 320, 693, False, 4, 0), (3, 1001, 5003, False, 1, 0), (64, 301, 129, True, 1, 0), (25, 99, 501, False, 1, 103), (3, 171, 8001, True, 1, 0),
    (5001, 65, 129, False, 1, 0), (1, 5001, 1001, True, 1, 0)])
def test_bf16(dev, pkg, oracle, m, n, k, bt, batch, ldc):
    capi = pkg.capi
    sigma = k ** -0.25
    a = util.to_bf16(capi, util.gen_normal(capi, (batch, m, k), 641, sigma))
    b = util.to_bf16(capi, util.gen_normal(capi, (batch, n, k) if bt else (batch, k, n), 642, sigma))
    c = run(dev, capi, capi.BF16, a, b, m, n, k, bt, batch=batch, ldc=ldc)
    if ldc:
        assert (c[:, :, n:] == 7).all()
    for i in range(batch):
        ref, _ = oracle.gemm_bf16(a[i], b[i], bt)
        util.assert_16bit_close(oracle, oracle.bf16_to_f32(np.ascontiguousarray(c[i, :, :n]).view(np.uint16)), ref)
