"""Results of 16-bit products of odd sizes, copied out of padded scratch eight rows at a time."""
import pytest

import util

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("m,n,k,batch", [(1, 9001, 257, 1), (7, 2001, 193, 1), (8, 2001, 193, 3), (9, 1023, 301, 2), (17, 255, 1001, 1), (64, 257, 129, 5), (40000, 33, 65, 1)])
def test_every_row_arrives(dev, pkg, dtype, m, n, k, batch):
    code = pkg.capi.BF16 if dtype == torch.bfloat16 else pkg.capi.F16
    g = torch.Generator(device="cuda:0")
    g.manual_seed(1)
    pitch = n + 5
    a = (torch.randn(batch, m, k, generator=g, device="cuda:0") * k ** -0.25).to(dtype)
    b = (torch.randn(batch, k, n, generator=g, device="cuda:0") * k ** -0.25).to(dtype)
    c = torch.full((batch * m + 1, pitch), 7.0, device="cuda:0", dtype=dtype)
    dev.gemm(code, m, n, k, a.data_ptr(), b.data_ptr(), c.data_ptr(), batch=batch, ldc=pitch, stream=util.cur_stream(torch))
    torch.cuda.synchronize()
    assert dev.status() == 0
    want = a.double() @ b.double()
    got = c[:batch * m].view(batch, m, pitch)
    # half of the result's last place, as much again where the f32 sum lies beside a boundary, and 1e-5 for cancelled sums
    last = 2.0 ** (-8 if dtype == torch.bfloat16 else -11)
    assert float(((got[:, :, :n] - want).abs() / (want.abs() * last * 1.05 + 1e-5)).max()) <= 1.0
    assert bool((got[:, :, n:] == 7.0).all()) and bool((c[batch * m] == 7.0).all())


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("m,n,k", [(64, 301, 129), (20, 321, 693), (64, 65, 16001)])
@pytest.mark.parametrize("positive", [False, True])
def test_the_rounding_of_the_sums_hides_in_the_last_place(dev, pkg, dtype, m, n, k, positive):
    """The distance from the 64-bit result is that of its correctly rounded values, to 1 %: sums of 16 terms cut off below 2^-24 of what an
    accumulator holds add 2^-24 * K / 32 at most, a fiftieth of f16's rounding at the longest K here, and the two add in squares."""
    code = pkg.capi.BF16 if dtype == torch.bfloat16 else pkg.capi.F16
    g = torch.Generator(device="cuda:0")
    g.manual_seed(1)
    a, b = ((torch.randn(*s, generator=g, device="cuda:0") * k ** -0.25).to(dtype) for s in ((m, k), (k, n)))
    if positive:
        a, b = a.abs(), b.abs()
    c = torch.empty(m, n, device="cuda:0", dtype=dtype)
    dev.gemm(code, m, n, k, a.data_ptr(), b.data_ptr(), c.data_ptr(), stream=util.cur_stream(torch))
    torch.cuda.synchronize()
    want = a.double() @ b.double()
    assert float((c - want).norm()) <= 1.01 * float((want.to(dtype) - want).norm())
