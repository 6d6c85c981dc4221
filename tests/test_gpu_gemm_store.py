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
