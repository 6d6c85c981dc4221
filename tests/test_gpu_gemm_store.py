"""16-bit GEMM on 256 x 256 and 128 x 256 tiles: results that end inside a 32 x 64 box, pitched and batched ones, f32 results, several tiles to a CTA;
nothing past C is written, by whichever way C leaves."""
import pytest

import util

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("out", ["same", "f32"])
@pytest.mark.parametrize("dtype,m,n,k,batch,bt,pad", [
    (torch.bfloat16, 3000, 2056, 64, 1, False, 0), (torch.float16, 129, 4104, 72, 3, True, 8), (torch.bfloat16, 2561, 3848, 200, 2, True, 24), (torch.float16, 257, 136, 1032, 150, False, 0),
    (torch.bfloat16, 100, 40008, 96, 1, False, 8), (torch.float16, 5001, 120, 264, 2, True, 0), (torch.bfloat16, 3330, 3080, 2056, 1, False, 16), (torch.float16, 1025, 2000, 2048, 1, True, 0),
    (torch.bfloat16, 1500, 1608, 4104, 4, False, 0)])
def test_against_f32(dev, pkg, out, dtype, m, n, k, batch, bt, pad):
    g = torch.Generator(device="cuda:0")
    g.manual_seed(m + n)
    code = pkg.capi.BF16 if dtype == torch.bfloat16 else pkg.capi.F16
    a = (torch.randn((batch, m, k), generator=g, device="cuda:0") * k ** -0.25).to(dtype)
    b = (torch.randn((batch, n, k) if bt else (batch, k, n), generator=g, device="cuda:0") * k ** -0.25).to(dtype)
    c = torch.full((batch * m * (n + pad) + 64,), 7.0, dtype=torch.float32 if out == "f32" else dtype, device="cuda:0")
    dev.gemm(code, m, n, k, a.data_ptr(), b.data_ptr(), c.data_ptr(), b_transposed=bt, batch=batch, ldc=n + pad, out_dtype=pkg.capi.F32 if out == "f32" else None,
             stream=util.cur_stream(torch))
    torch.cuda.synchronize()
    assert dev.status() == 0
    want = a.float() @ (b.transpose(1, 2) if bt else b).float()
    got = c[:batch * m * (n + pad)].view(batch, m, n + pad)
    # f32 sums of k terms of either sign toward zero, and half a unit of the result's last place
    tol = 2e-5 if out == "f32" else 2.5e-3 if dtype == torch.bfloat16 else 3.5e-4
    assert float((got[..., :n].float() - want).norm() / want.norm()) <= tol
    assert float((got[..., :n].float() - want).abs().max()) <= 8 * tol * float(want.abs().max())
    assert bool((got[..., n:] == 7.0).all()) and bool((c[batch * m * (n + pad):] == 7.0).all())


# N mod 256 of one, two, three and four boxes of 64 columns (f32: up to eight of 32), rows of C for some or one of a tile's warps, K so short that the next tile waits
# for nothing, several tiles to a CTA.  Small whole numbers, so that every sum is exact and a result is its correctly rounded value.
@pytest.mark.parametrize("out", ["same", "f32"])
@pytest.mark.parametrize("dtype,m,n,k,batch,bt", [
    (torch.bfloat16, 2305, 3080, 16, 1, False), (torch.float16, 2337, 3136, 64, 1, True), (torch.bfloat16, 2337, 3208, 120, 1, True), (torch.float16, 2305, 3264, 200, 1, False),
    (torch.bfloat16, 129, 264, 40, 200, True), (torch.float16, 257, 320, 24, 120, False), (torch.bfloat16, 2305, 4088, 8, 1, False),
    (torch.bfloat16, 33, 40008, 16, 3, True), (torch.float16, 65, 40000, 72, 2, False), (torch.float16, 161, 72, 16, 400, False), (torch.bfloat16, 129, 64, 200, 500, True), (torch.bfloat16, 1, 8, 64, 5000, True)])
def test_tiles_that_follow_an_edge_tile(dev, pkg, out, dtype, m, n, k, batch, bt):
    g = torch.Generator(device="cuda:0")
    g.manual_seed(m + n + k)
    code = pkg.capi.BF16 if dtype == torch.bfloat16 else pkg.capi.F16
    a = torch.randint(-3, 4, (batch, m, k), generator=g, device="cuda:0").to(dtype)
    b = torch.randint(-3, 4, (batch, n, k) if bt else (batch, k, n), generator=g, device="cuda:0").to(dtype)
    want = (a.double() @ (b.transpose(1, 2) if bt else b).double()).to(torch.float32 if out == "f32" else dtype)
    c = torch.empty_like(want)
    wrong = torch.zeros((), dtype=torch.int64, device="cuda:0")
    for _ in range(150):
        c.fill_(float("nan"))
        dev.gemm(code, m, n, k, a.data_ptr(), b.data_ptr(), c.data_ptr(), b_transposed=bt, batch=batch, out_dtype=pkg.capi.F32 if out == "f32" else None, stream=util.cur_stream(torch))
        wrong += (c != want).sum()
    torch.cuda.synchronize()
    assert dev.status() == 0 and int(wrong) == 0
