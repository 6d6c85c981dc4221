"""16-bit products of odd sizes: results written straight to rows that start anywhere by every kernel, operands that need no copy, one copy or two, pitched and
shifted ones."""
import pytest

import util

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("m,n,k,batch,bt,pads,shift", [
    (3000, 2051, 136, 1, True, (0, 0, 0), 0),        # pairs, no copy
    (513, 1999, 515, 2, False, (0, 0, 0), 0),        # both operands
    (2050, 2100, 333, 1, True, (3, 0, 0), 0),        # pitches
    (100, 30001, 200, 1, True, (0, 0, 0), 0),        # 128 x 256 tiles
    (5000, 101, 264, 4, False, (0, 3, 2), 0),
    (7, 999, 3001, 1, True, (0, 0, 1), 0),           # few rows, K over a cluster
    (90, 333, 1000, 3, False, (0, 3, 0), 0),
    (760, 144, 124, 1, True, (4, 4, 0), 0),          # K ends inside a vector, no copy
    (1, 77, 73, 1, False, (0, 0, 0), 0), (3, 123, 3313, 1, True, (0, 0, 0), 0), (1, 1, 16383, 1, False, (0, 0, 0), 0), (5, 3, 999, 64, True, (0, 0, 0), 0),  # few outputs
    (700, 901, 41, 1, True, (0, 0, 0), 0), (2500, 2501, 19, 1, False, (0, 0, 0), 0),
    (129, 257, 257, 1, False, (0, 0, 0), 1), (300, 513, 400, 1, True, (0, 0, 0), 3), (64, 1000, 81, 1, True, (0, 0, 0), 7)])
def test_against_64_bits(dev, pkg, dtype, m, n, k, batch, bt, pads, shift):
    g = torch.Generator(device="cuda:0")
    g.manual_seed(n)
    code = pkg.capi.BF16 if dtype == torch.bfloat16 else pkg.capi.F16
    rows_b, cols_b = (n, k) if bt else (k, n)
    lda, ldb, ldc = k + pads[0], cols_b + pads[1], n + pads[2]

    def matrix(rows, ld):
        flat = (torch.randn(batch * rows * ld + 16, generator=g, device="cuda:0") * k ** -0.25).to(dtype)
        return flat[shift:shift + batch * rows * ld]

    a, b = matrix(m, lda), matrix(rows_b, ldb)
    whole = torch.full((batch * m * ldc + 16,), 7.0, dtype=dtype, device="cuda:0")
    c = whole[shift:shift + batch * m * ldc]
    dev.gemm(code, m, n, k, a.data_ptr(), b.data_ptr(), c.data_ptr(), b_transposed=bt, batch=batch, lda=lda, ldb=ldb, ldc=ldc, stream=util.cur_stream(torch))
    torch.cuda.synchronize()
    assert dev.status() == 0
    av, bv = a.view(batch, m, lda)[:, :, :k].double(), b.view(batch, rows_b, ldb)[:, :, :cols_b].double()
    want = av @ (bv.transpose(1, 2) if bt else bv)
    got = c.view(batch, m, ldc)
    # half of the result's last place, as much again where the f32 sum lies beside a boundary, and 1e-5 for cancelled sums
    last = 2.0 ** (-8 if dtype == torch.bfloat16 else -11)
    assert float(((got[:, :, :n] - want).abs() / (want.abs() * last * 1.05 + 1e-5)).max()) <= 1.0
    assert bool((got[:, :, n:] == 7.0).all()) and bool((whole[:shift] == 7.0).all()) and bool((whole[shift + batch * m * ldc:] == 7.0).all())


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("m,n", [(3, 123), (1, 77), (33, 7), (501, 1)])
@pytest.mark.parametrize("k", [73, 515, 4095, 6143, 12001, 16383])
def test_few_outputs_of_positive_data(dev, pkg, dtype, m, n, k):
    """Sums that only grow are where rounding toward zero shows: no further from 64 bits, in the norm over many products, than the correctly rounded results and 2^-23."""
    code = pkg.capi.BF16 if dtype == torch.bfloat16 else pkg.capi.F16
    off = best = 0.0
    for seed in range(20000 // (m * n)):
        g = torch.Generator(device="cuda:0")
        g.manual_seed(1000003 * seed + 7 * m + k)
        a, b = torch.rand(m, k, generator=g, device="cuda:0").to(dtype), (torch.rand(k, n, generator=g, device="cuda:0") * (8.0 / k)).to(dtype)
        c = torch.empty(m, n, dtype=dtype, device="cuda:0")
        dev.gemm(code, m, n, k, a.data_ptr(), b.data_ptr(), c.data_ptr(), stream=util.cur_stream(torch))
        want = a.double() @ b.double()
        off += ((c.double() - want).square().sum() / want.square().sum()).double()
        best += ((want.to(dtype).double() - want).square().sum() / want.square().sum()).double()
    torch.cuda.synchronize()
    assert dev.status() == 0
    # of about 20000 results, whose own rounding, 2^-12.1 in the norm (bf16 2^-9.1), leaves 3e-8 of chance (bf16: 1e-7 and less of bias beside it)
    assert float((off / (20000 // (m * n))).sqrt() - (best / (20000 // (m * n))).sqrt()) <= 2.0 ** -23
