"""Row operators, SiLU and rotation with more work than CTAs at once: two rows to a CTA and an odd number of them, one round to a CTA; and so little that
every thread has one vector at most."""
import pytest

import util

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")
CODES = {torch.float32: "F32", torch.bfloat16: "BF16", torch.float16: "F16"}


def near(got, want, dtype):
    tol = 2e-6 if dtype == torch.float32 else 5e-3 if dtype == torch.bfloat16 else 6e-4  # the result rounded once, and f32 arithmetic
    return float((got.double() - want).norm() / want.norm()) <= tol


@pytest.mark.parametrize("dtype", list(CODES))
@pytest.mark.parametrize("rows,cols", [(5001, 2056), (2369, 4096), (3333, 8192), (1, 4096), (20001, 256)])
def test_rows(dev, pkg, dtype, rows, cols):
    g = torch.Generator(device="cuda:0")
    g.manual_seed(rows)
    x = torch.randn((rows, cols), generator=g, device="cuda:0").to(dtype)
    code, st = getattr(pkg.capi, CODES[dtype]), util.cur_stream(torch)
    y = torch.full((rows + 1, cols), 7.0, dtype=dtype, device="cuda:0")
    dev.rms_norm(code, rows, cols, 1e-5, x.data_ptr(), y.data_ptr(), stream=st)
    most = torch.full((rows + 1,), 7.0, dtype=dtype, device="cuda:0")
    dev.reduce(code, pkg.capi.REDUCE_MAX, rows, cols, x.data_ptr(), most.data_ptr(), stream=st)
    torch.cuda.synchronize()
    xd = x.double()
    assert near(y[:rows], xd * torch.rsqrt(xd.square().mean(-1, keepdim=True) + 1e-5), dtype) and bool((y[rows] == 7.0).all())
    assert torch.equal(most[:rows], x.max(-1).values) and float(most[rows]) == 7.0


@pytest.mark.parametrize("dtype", list(CODES))
@pytest.mark.parametrize("rows,cols", [(1, 8), (3, 4096), (16, 16384), (147, 4104), (9001, 4096)])
def test_silu(dev, pkg, dtype, rows, cols):
    g = torch.Generator(device="cuda:0")
    g.manual_seed(cols)
    gate, up = (torch.randn((rows, cols), generator=g, device="cuda:0").to(dtype) for _ in range(2))
    y = torch.full((rows + 1, cols), 7.0, dtype=dtype, device="cuda:0")
    dev.silu_mul(getattr(pkg.capi, CODES[dtype]), rows, cols, gate.data_ptr(), up.data_ptr(), y.data_ptr(), stream=util.cur_stream(torch))
    torch.cuda.synchronize()
    assert near(y[:rows], torch.nn.functional.silu(gate.double()) * up.double(), dtype) and bool((y[rows] == 7.0).all())


@pytest.mark.parametrize("dtype", list(CODES))
@pytest.mark.parametrize("tokens,heads,d,start", [(30001, 3, 128, 5), (25000, 8, 64, 0)])
def test_rotation(dev, pkg, dtype, tokens, heads, d, start):
    g = torch.Generator(device="cuda:0")
    g.manual_seed(tokens)
    x = torch.randn((tokens + 1, heads, d), generator=g, device="cuda:0").to(dtype)
    before = x.clone()
    dev.rope(getattr(pkg.capi, CODES[dtype]), 1, tokens, heads, d, start, 10000.0, x.data_ptr(), stream=util.cur_stream(torch))
    torch.cuda.synchronize()
    i = torch.arange(0, d, 2, dtype=torch.float64, device="cuda:0")
    angle = (start + torch.arange(tokens, dtype=torch.float64, device="cuda:0"))[:, None] * 10000.0 ** (-i / d)
    co, si = angle.cos()[:, None], angle.sin()[:, None]
    a, b = before[:tokens, :, 0::2].double(), before[:tokens, :, 1::2].double()
    want = torch.stack((a * co - b * si, a * si + b * co), -1).reshape(tokens, heads, d)
    # an angle of up to 30000 in f32 is off by 2^-24 of itself, and its frequency by as much again
    tol = (tokens + start) * 2.0 ** -22 + (0 if dtype == torch.float32 else 2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -11)
    assert float((x[:tokens].double() - want).norm() / want.norm()) <= tol and torch.equal(x[tokens], before[tokens])
