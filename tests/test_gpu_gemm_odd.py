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


# every output infinite: all blocks are summed again, at about the FP32 pipe's rate, and nothing waits for it
@pytest.mark.parametrize("bt", [False, True])
def test_f32_odd_product_that_overflows_everywhere(dev, pkg, bt):
    capi = pkg.capi
    m, n, k = 2049, 2051, 301
    rows, cols = np.where(np.arange(m) % 3 == 1, -1, 1), np.where(np.arange(n) % 5 == 2, -1, 1)
    a = (np.abs(util.gen_uniform(capi, (m, k), 611)) + 1) * np.float32(1e20) * rows[:, None].astype(np.float32)
    b = (np.abs(util.gen_uniform(capi, (k, n), 612)) + 1) * np.float32(1e20) * cols[None, :].astype(np.float32)
    b = np.ascontiguousarray(b.T) if bt else b

    def ms(a, b):
        ad, bd = util.dev_tensor(torch, a), util.dev_tensor(torch, b)
        cd = torch.full((m, n), 7, dtype=torch.float32, device="cuda:0")
        t = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
        for _ in range(2):
            t[0].record()
            dev.gemm(capi.F32, m, n, k, ad.data_ptr(), bd.data_ptr(), cd.data_ptr(), b_transposed=bt, stream=util.cur_stream(torch))
            t[1].record()
        torch.cuda.synchronize()
        assert dev.status() == 0
        return cd.cpu().numpy(), t[0].elapsed_time(t[1])

    c, slow = ms(a, b)
    assert np.array_equal(c, np.where(rows[:, None] * cols > 0, np.float32(np.inf), np.float32(-np.inf)))
    _, fast = ms(a * np.float32(1e-20), b * np.float32(1e-20))
    # one lane after the other took 20 ms more
    assert slow <= 20 * fast + 1, (slow, fast)


@pytest.mark.parametrize("m,n,k,bt", [(2305, 4099, 5001, False), (2305, 4099, 5001, True), (66, 16387, 2051, False)])
def test_f32_an_infinite_row_of_a_long_product(dev, pkg, oracle, m, n, k, bt):
    """Several tiles per CTA, among them some with infinities: those alone are replaced, by what the FP32 pipe gives."""
    capi = pkg.capi
    a, b = util.gen_uniform(capi, (m, k), 615), util.gen_uniform(capi, (n, k) if bt else (k, n), 616)
    a[40, 3] = np.inf
    col = n - 2
    b[(col, 9) if bt else (9, col)] = -np.inf
    c = run(dev, capi, capi.F32, a, b, m, n, k, bt)[0]
    bk = lambda i: b[:, i] if bt else b[i]  # noqa: E731
    want = np.sign(bk(3)) * np.float64(np.inf)
    with np.errstate(invalid="ignore"):
        want[col] += -np.sign(a[40, 9]) * np.inf
    assert np.array_equal(c[40], want.astype(np.float32), equal_nan=True)
    want = -np.sign(a[:, 9]) * np.inf
    want[40] = c[40, col]
    assert np.array_equal(c[:, col], want.astype(np.float32), equal_nan=True)
    keep = np.delete(np.arange(n), col)
    rows = np.array([0, 39, 41, 63, 64, m - 1])
    truth = oracle.gemm_f32(np.ascontiguousarray(a[rows]), np.ascontiguousarray(b[keep] if bt else b[:, keep]), bt, f64_acc=True)
    mt = oracle.compare(np.ascontiguousarray(c[rows][:, keep]), truth)
    assert mt["rel_max"] <= util.F32_REL and mt["rel_fro"] <= util.F32_REL, mt


@pytest.mark.parametrize("m,n,k,bt,wide_a", [(1025, 2051, 301, False, True), (1025, 2051, 1503, True, False)])
def test_f32_whole_numbers_stay_exact(dev, pkg, m, n, k, bt, wide_a):
    """Entries of 21 bits on one side, of 2 on the other, sums below 2^24: hi + lo holds them, and f32 adds them exactly."""
    capi = pkg.capi
    rng = np.random.default_rng(641)
    wide = rng.integers(-(1 << 20), 1 << 20, (m, k) if wide_a else (n, k)).astype(np.float32)
    small = np.zeros((n, k) if wide_a else (m, k), np.float32)
    small[np.arange(len(small))[:, None], rng.integers(0, k, (len(small), 5))] = rng.integers(-3, 4, (len(small), 5))  # 5 * 3 * 2^20 < 2^24
    a, b = (wide, small) if wide_a else (small, wide)
    c = run(dev, capi, capi.F32, a, b if bt else np.ascontiguousarray(b.T), m, n, k, bt)[0]
    assert np.array_equal(c, a.astype(np.float64) @ b.T.astype(np.float64))
