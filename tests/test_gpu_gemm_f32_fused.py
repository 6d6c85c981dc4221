"""f32 GEMM with the operands split on the way in: tile edges, both widths, splits of K, several tiles per CTA, rows that start anywhere,
pitches, batches, and values that a split cannot represent."""

import pytest

import util

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def rnd(*shape, seed=1, sigma=1.0):
    g = torch.Generator(device="cuda:0")
    g.manual_seed(seed)
    return torch.randn(shape, generator=g, device="cuda:0") * sigma


def product(dev, capi, a, b, m, n, k, bt, batch=1, lda=0, ldb=0, ldc=0, c=None):
    c = torch.full((batch, m, ldc or n), float("nan"), device="cuda:0") if c is None else c
    dev.gemm(capi.F32, m, n, k, a.data_ptr(), b.data_ptr(), c.data_ptr(), b_transposed=bt, batch=batch, lda=lda, ldb=ldb, ldc=ldc,
             stream=util.cur_stream(torch))
    torch.cuda.synchronize()
    assert dev.status() == 0
    return c


# An accumulator takes 256 of K of aligned rows (128 of others) in 16 instructions (8) and cuts off below 2^-24 of what it holds at each,
# half of it in the mean, so 4.8e-7 (2.4e-7) of the result at its fullest, half of that while it grows.  The sums over accumulators, rounded to
# nearest, add 2^-25 times the square root of their number, and an output its own rounding, 2^-24 at the most.
def bound(k, aligned):
    if aligned and k < 160:
        return 2e-6  # the small ones of these are the warp-level kernel's, on 22 bits of each operand
    return (4.8e-7 if aligned else 2.4e-7) + 6e-8 + 3e-8 * (k / 128) ** 0.5


@pytest.mark.parametrize("bt", [False, True])
@pytest.mark.parametrize("m,n,k", [
    (1, 1, 64), (1, 1, 65), (128, 64, 64), (129, 65, 95), (127, 63, 97), (100, 70, 2501), (301, 301, 1000), (512, 512, 512), (130, 129, 1024),
    (1024, 1024, 1024), (600, 2401, 201), (600, 2400, 200), (1001, 1003, 333), (2400, 1900, 161), (2401, 1901, 65), (3000, 5000, 160), (5, 4000, 777),
    (1000, 1000, 4096), (900, 900, 20000), (64, 64, 100000), (65, 63, 100001)])
def test_against_64_bits(dev, pkg, m, n, k, bt):
    s = k ** -0.25
    a, b = rnd(m, k, sigma=s), rnd(*((n, k) if bt else (k, n)), seed=2, sigma=s)
    c = product(dev, pkg.capi, a, b, m, n, k, bt)[0]
    want = a.double() @ (b.double().T if bt else b.double())
    err = float((c - want).norm() / want.norm())
    assert err <= bound(k, k % 4 == 0 and n % 4 == 0), err


@pytest.mark.parametrize("shift", [0, 1, 2, 3])
@pytest.mark.parametrize("bt", [False, True])
def test_rows_that_start_anywhere_pitches_and_batches(dev, pkg, shift, bt):
    """Column blocks of larger matrices, `shift` elements from a 16-byte boundary; what lies around C stays."""
    m, n, k, batch = 150, 203, 300, 3
    lda, ldb, ldc = 309, 331, 223
    rows_b, cols_b = (n, k) if bt else (k, n)
    big_a, big_b = rnd(batch * m * lda + 8), rnd(batch * rows_b * ldb + 8, seed=2)
    big_c = torch.full((batch * m * ldc + 8,), 7.0, device="cuda:0")
    a, b, c = big_a[shift:], big_b[shift:], big_c[shift:]
    product(dev, pkg.capi, a, b, m, n, k, bt, batch, lda, ldb, ldc, c)
    av = a[:batch * m * lda].view(batch, m, lda)[:, :, :k].double()
    bv = b[:batch * rows_b * ldb].view(batch, rows_b, ldb)[:, :, :cols_b].double()
    want = av @ (bv.transpose(1, 2) if bt else bv)
    got = c[:batch * m * ldc].view(batch, m, ldc)
    assert float((got[:, :, :n] - want).norm() / want.norm()) <= 1e-6
    assert bool((got[:, :, n:] == 7.0).all()) and bool((big_c[:shift] == 7.0).all()) and bool((c[batch * m * ldc:] == 7.0).all())


@pytest.mark.parametrize("m,n,k,bt", [(300, 301, 2001, False), (200, 131, 333, True), (1700, 1501, 97, False), (2401, 2301, 129, True)])
def test_infinities_nans_and_the_largest_numbers_as_on_the_fp32_pipe(dev, pkg, m, n, k, bt):
    """Split K, one tile and several tiles per CTA: outputs infinite or NaN where plain f32 sums are, finite where those are finite."""
    a, b = rnd(m, k, sigma=0.1), rnd(*((n, k) if bt else (k, n)), seed=2, sigma=0.1)
    bv = b.T if bt else b
    all_ones = torch.tensor([-1], dtype=torch.int32, device="cuda:0").view(torch.float32)[0]  # a NaN whose rounding carries
    a[0, 5], a[m // 2, 0], a[m - 1, k - 1] = float("inf"), float("-inf"), all_ones
    a[1, 3], a[2, 4] = 3.4e38, -3.4028234e38   # the second rounds up to infinity as a TF32 number
    bv[3, :], bv[4, :] = 0.25, 0.5
    bv[5, n - 1] = 0.0                           # 0 * inf
    bv[k - 2, 1] = float("nan")
    c = product(dev, pkg.capi, a, b, m, n, k, bt)[0]
    want = a.double() @ bv.double()  # finite ones stay far below the largest f32 number
    want32 = want.float()
    assert torch.equal(torch.isnan(c), torch.isnan(want32))
    assert torch.equal(torch.isinf(c), torch.isinf(want32)) and torch.equal(c[torch.isinf(c)] > 0, want32[torch.isinf(c)] > 0)
    ok = torch.isfinite(want32)
    # sums of k products of 0.1 x 0.1 stand beside terms of up to 1.7e38
    scale = a.abs().nan_to_num(0, 0, 0).double() @ bv.abs().nan_to_num(0, 0, 0).double()
    assert float(((c - want).abs()[ok] / scale[ok]).max()) <= 4e-6
    whole = product(dev, pkg.capi, a, b, m, n, k, bt)[0]
    assert torch.equal(whole.view(torch.int32), c.view(torch.int32))  # the second pass has one order too


@pytest.mark.parametrize("n", [512, 511])
def test_the_largest_numbers_stay_finite(dev, pkg, n):
    """Factors up to the largest one whose hi part is finite, also where rows are aligned and no second pass looks after them."""
    m, k = 200, 512
    a, b = rnd(m, k), rnd(k, n, seed=2, sigma=1e-3)
    for i, x in enumerate((8.6e37, 1.2345678e38, 1.7014e38, 2.9876543e38, 3.4011e38, -3.4011e38, 3.3999999e38)):
        a[i * 20, :] *= 1e-3
        a[i * 20, 17 * i] = x
    c = product(dev, pkg.capi, a, b, m, n, k, False)[0]
    want = a.double() @ b.double()
    assert bool(torch.isfinite(c).all())
    scale = a.abs().double() @ b.abs().double()
    assert float(((c - want).abs() / scale).max()) <= 2e-6


def test_every_output_infinite(dev, pkg):
    m, n, k = 1500, 1301, 301
    a, b = rnd(m, k).abs() + 0.1, rnd(k, n, seed=2).abs() + 0.1
    a[:, 7] = float("inf")
    assert bool(torch.isposinf(product(dev, pkg.capi, a, b, m, n, k, False)).all())


def test_whole_numbers_stay_exact(dev, pkg):
    """Products and partial sums below 2^24 (factors of up to 13 bits: hi and lo both in use)."""
    for (m, n, k, bt) in ((200, 301, 401, False), (600, 600, 1024, True), (129, 500, 64, False)):
        g = torch.Generator(device="cuda:0")
        g.manual_seed(3)
        a = torch.randint(-8191, 8192, (m, k), generator=g, device="cuda:0").float()
        b = torch.randint(-1, 2, (n, k) if bt else (k, n), generator=g, device="cuda:0").float()
        want = a.double() @ (b.double().T if bt else b.double())
        assert float(want.abs().max()) < 2 ** 24
        assert torch.equal(product(dev, pkg.capi, a, b, m, n, k, bt)[0].double(), want)


def one_hot(rows, cols, seed):
    """Rows with a single 1, and which column has it."""
    g = torch.Generator(device="cuda:0")
    g.manual_seed(seed)
    at = torch.randint(0, cols, (rows,), generator=g, device="cuda:0")
    x = torch.zeros(rows, cols, device="cuda:0")
    x[torch.arange(rows, device="cuda:0"), at] = 1.0
    return x, at


@pytest.mark.parametrize("bt", [False, True])
@pytest.mark.parametrize("m,n,k", [(300, 301, 2001), (130, 65, 129), (2401, 1901, 65), (512, 512, 512), (1024, 1024, 1024), (600, 604, 200)])
def test_rows_picked_by_a_one_hot_matrix_keep_every_bit(dev, pkg, m, n, k, bt):
    """From either side, with values of all 24 bits between 2^-100 and 2^100."""
    def wide(*shape):
        e = torch.rand(shape, generator=torch.Generator(device="cuda:0").manual_seed(7), device="cuda:0") * 200 - 100
        return torch.ldexp(rnd(*shape, seed=5), e.floor())

    a, at = one_hot(m, k, 3)
    b = wide(k, n)
    c = product(dev, pkg.capi, a, b.T.contiguous() if bt else b, m, n, k, bt)[0]
    assert torch.equal(c, b[at])
    a = wide(m, k)
    b, at = one_hot(n, k, 4)
    c = product(dev, pkg.capi, a, b if bt else b.T.contiguous(), m, n, k, bt)[0]
    assert torch.equal(c, a[:, at])


def test_whole_numbers_of_24_bits_stay_exact(dev, pkg):
    """One factor uses all 24 bits, the other picks two of them with opposite signs; or both have 12."""
    for (m, n, k) in ((300, 301, 2001), (512, 512, 512), (129, 67, 65)):
        g = torch.Generator(device="cuda:0")
        g.manual_seed(3)
        a = torch.randint(-(2 ** 24) + 1, 2 ** 24, (m, k), generator=g, device="cuda:0").float().abs()
        plus, at = one_hot(n, k, 5)
        minus, by = one_hot(n, k, 6)
        b = (plus - minus).T.contiguous()
        assert torch.equal(product(dev, pkg.capi, a, b, m, n, k, False)[0], a[:, at] - a[:, by])
        a = torch.randint(2048, 4096, (m, k), generator=g, device="cuda:0").float()
        pick, at = one_hot(n, k, 8)
        b = (pick * 4095).T.contiguous()
        assert torch.equal(product(dev, pkg.capi, a, b, m, n, k, False)[0], a[:, at] * 4095)


@pytest.mark.parametrize("m,n,k,bt", [(300, 301, 2001, False), (200, 131, 333, True), (1700, 1501, 97, False), (512, 512, 512, False), (600, 604, 200, True)])
def test_the_smallest_numbers_count(dev, pkg, m, n, k, bt):
    """Operands down to the smallest f32 number: of one tile, of single rows, columns and elements; f32 sums of k terms are within
    k * 2^-24 of the sum of their magnitudes, and each of them is rounded to a multiple of 2^-149 where the sum is that small."""
    def check(a, b):
        c = product(dev, pkg.capi, a, b, m, n, k, bt)[0]
        bv = (b.T if bt else b).double()
        want, scale = a.double() @ bv, a.abs().double() @ bv.abs()
        assert float(((c - want).abs() / (scale * 2e-6 + k * 2.0 ** -150)).max()) <= 1.0

    a, b = rnd(m, k), rnd(*((n, k) if bt else (k, n)), seed=2)
    check(a * 2.0 ** -125, b * 2.0 ** 60)
    check(a * 2.0 ** 100, b * 2.0 ** -130)
    check(a * 2.0 ** -140, b)
    x = a.clone()
    x[m // 2], x[3, :k // 2] = a[m // 2] * 2.0 ** -120, a[3, :k // 2] * 2.0 ** -135
    check(x, b)
    w = b.clone()
    w[5] *= 2.0 ** -122
    w[:, 7] *= 2.0 ** -128
    check(a, w)
    check(x, w)


def test_captured_and_on_two_streams(dev, pkg):
    m, n, k = 300, 333, 1111
    a, b = rnd(m, k), rnd(k, n, seed=2)
    want = product(dev, pkg.capi, a, b, m, n, k, False)
    streams, outs = [torch.cuda.Stream() for _ in range(2)], [torch.zeros(m, n, device="cuda:0") for _ in range(3)]
    torch.cuda.synchronize()
    for s, o in zip(streams, outs):
        for _ in range(10):
            dev.gemm(pkg.capi.F32, m, n, k, a.data_ptr(), b.data_ptr(), o.data_ptr(), stream=s.cuda_stream)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        dev.gemm(pkg.capi.F32, m, n, k, a.data_ptr(), b.data_ptr(), outs[2].data_ptr(), stream=torch.cuda.current_stream().cuda_stream)
    graph.replay()
    torch.cuda.synchronize()
    assert all(torch.equal(o, want[0]) for o in outs)
    del graph
