"""16-bit GEMMs of odd sizes on the GPU, through the C ABI, against the CPU oracle."""
import numpy as np
import pytest

import util
from test_gpu_gemm_odd import run

pytestmark = pytest.mark.gpu


# 16-bit rows that start anywhere: operands copied into padded scratch, in every combination of what needs it
@pytest.mark.parametrize("m,n,k,bt,batch,offset,ldc", [
    (300, 301, 1203, False, 1, 0, 0), (300, 301, 1203, True, 1, 0, 0), (257, 512, 1001, True, 2, 0, 0), (511, 257, 1024, False, 3, 0, 0),
    (400, 520, 512, False, 1, 1, 0), (400, 520, 512, True, 1, 0, 523), (28, 3134, 4883, False, 1, 0, 0),
    (30, 101, 23003, False, 1, 0, 0), (1, 1001, 67103, True, 1, 0, 0), (30, 101, 1003, False, 23, 0, 0)])
def test_bf16_rows_that_start_anywhere(dev, pkg, oracle, m, n, k, bt, batch, offset, ldc):
    capi = pkg.capi
    sigma = k ** -0.25
    a = util.to_bf16(capi, util.gen_normal(capi, (batch, m, k), 631, sigma))
    b = util.to_bf16(capi, util.gen_normal(capi, (batch, n, k) if bt else (batch, k, n), 632, sigma))
    c = run(dev, capi, capi.BF16, a, b, m, n, k, bt, batch=batch, ldc=ldc, offset=offset)
    if ldc:
        assert (c[:, :, n:] == 7).all()
    for i in range(batch):
        ref, _ = oracle.gemm_bf16(a[i], b[i], bt)
        util.assert_16bit_close(oracle, oracle.bf16_to_f32(np.ascontiguousarray(c[i, :, :n]).view(np.uint16)), ref)
