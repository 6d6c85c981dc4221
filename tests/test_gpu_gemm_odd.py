"""f32 GEMMs of odd sizes on the GPU, through the C ABI, against the CPU oracle."""
import numpy as np
import pytest

import util

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def run(dev, capi, dtype, a, b, m, n, k, bt, batch=1, out_f32=False, ldc=0, offset=0):
    """C [batch][m][ldc or n] as a host array; `offset` shifts A's start by that many elements."""
    flat = np.concatenate([np.zeros(offset, a.dtype), a.reshape(-1)])
    ad, bd = util.dev_tensor(torch, flat), util.dev_tensor(torch, b)
    f32 = dtype == capi.F32 or out_f32
    cd = torch.full((batch, m, ldc or n), 7, dtype=torch.float32 if f32 else torch.int16, device="cuda:0")
    dev.gemm(dtype, m, n, k, ad.data_ptr() + offset * ad.element_size(), bd.data_ptr(), cd.data_ptr(), b_transposed=bt,
             batch=batch, ldc=ldc, out_dtype=capi.F32 if f32 else dtype, stream=util.cur_stream(torch))
    torch.cuda.synchronize()
    assert dev.status() == 0
    return cd.cpu().numpy()


# the tcgen05 f32 kernel: rows of A, B and C that start anywhere; N even but no multiple of 4; both tile widths
@pytest.mark.parametrize("m,n,k,bt,offset,ldc", [
    (1999, 3001, 1501, False, 0, 0), (1025, 2051, 257, False, 0, 0), (1025, 2051, 259, True, 0, 0), (1030, 2050, 260, True, 0, 0),
    (1024, 2048, 512, False, 1, 0), (1024, 2048, 256, True, 0, 2050), (1024, 2048, 256, False, 0, 2051), (2300, 2300, 301, False, 3, 0),
    (100, 16386, 258, True, 0, 0)])
def test_f32_rows_that_start_anywhere(dev, pkg, oracle, m, n, k, bt, offset, ldc):
    capi = pkg.capi
    a = util.gen_uniform(capi, (m, k), 601)
    b = util.gen_uniform(capi, (n, k) if bt else (k, n), 602)
    c = run(dev, capi, capi.F32, a, b, m, n, k, bt, ldc=ldc, offset=offset)[0]
    if ldc:
        assert (c[:, n:] == 7).all()  # the pitch's gap is not written
    rows = sorted({0, 1, 31, 32, 127, 128, m // 2, m - 2, m - 1})
    rows = [r for r in rows if 0 <= r < m]
    truth = oracle.gemm_f32(np.ascontiguousarray(a[rows]), b, bt, f64_acc=True)
    mt = oracle.compare(np.ascontiguousarray(c[rows, :n]), truth)
    assert mt["rel_max"] <= util.F32_REL and mt["rel_fro"] <= util.F32_REL, mt


def test_f32_infinities_and_nans_in_odd_rows(dev, pkg, oracle):
    """An infinity times a finite number stays one (hi + lo of an infinity would be infinity + NaN), NaNs stay where they are."""
    capi = pkg.capi
    m, n, k = 2049, 2051, 301
    a, b = util.gen_uniform(capi, (m, k), 605), util.gen_uniform(capi, (k, n), 606)
    a[3, 7], a[200, 5], a[200, 6], b[11, 40] = np.inf, np.inf, -np.inf, np.nan
    a[9, 1] = np.float32(3.4028235e38)  # rounds to an infinite hi part
    c = run(dev, capi, capi.F32, a, b, m, n, k, False)[0]
    with np.errstate(all="ignore"):
        want = a.astype(np.float64) @ b.astype(np.float64)
    finite = np.isfinite(want)
    assert np.array_equal(np.isnan(c), np.isnan(want)) and np.array_equal(c[np.isinf(want)], want[np.isinf(want)])
    rows = [r for r in (0, 4, 100, 2048)]
    assert np.abs(c[rows][finite[rows]] - want[rows][finite[rows]]).max() <= util.F32_REL * np.abs(want[rows][finite[rows]]).max()
    assert np.allclose(c[9][finite[9]], want[9][finite[9]], rtol=1e-5, atol=0)
