"""rms_norm, reductions and SiLU * Mul one value at a time, several loads of a thread in flight: the ends of the unrolled loops."""
import pytest

import util

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")
TYPES = {"f32": torch.float32, "bf16": torch.bfloat16, "f16": torch.float16}
# f32: 512 threads add up a row in a tree, 2^-24 of the sum for each of the terms a thread adds, and expf and a division; 16 bits: half of
# the last place of the result, and as much again for the approximate exponential beside a rounding boundary
CLOSE = {"f32": 1e-5, "bf16": 2.0 ** -8, "f16": 2.0 ** -11}


def rnd(*shape, dtype, seed=1):
    g = torch.Generator(device="cuda:0")
    g.manual_seed(seed)
    return torch.randn(shape, generator=g, device="cuda:0").to(TYPES[dtype])


def code(capi, dtype):
    return {"f32": capi.F32, "bf16": capi.BF16, "f16": capi.F16}[dtype]


# a thread takes 8 values, 512 apart, at a time
@pytest.mark.parametrize("dtype", TYPES)
@pytest.mark.parametrize("cols", [1, 511, 513, 3583, 3585, 4095, 4097, 4607, 4609, 8191, 8193, 12289, 39385])
def test_rows_of_odd_widths(dev, pkg, dtype, cols):
    rows = 5
    x, y = rnd(rows, cols, dtype=dtype), torch.full((rows + 1, cols), 7.0, device="cuda:0", dtype=TYPES[dtype])
    dev.rms_norm(code(pkg.capi, dtype), rows, cols, 1e-5, x.data_ptr(), y.data_ptr(), stream=util.cur_stream(torch))
    torch.cuda.synchronize()
    want = x.double() * torch.rsqrt(x.double().square().mean(-1, keepdim=True) + 1e-5)
    assert float(((y[:rows] - want).abs() / want.abs().clamp_min(1e-3)).max()) <= CLOSE[dtype]
    assert bool((y[rows] == 7.0).all())
    top, total = torch.zeros(rows, device="cuda:0", dtype=TYPES[dtype]), torch.zeros(rows, device="cuda:0", dtype=TYPES[dtype])
    for kind, out in ((pkg.capi.REDUCE_MAX, top), (pkg.capi.REDUCE_SUM, total)):
        dev.reduce(code(pkg.capi, dtype), kind, rows, cols, x.data_ptr(), out.data_ptr(), stream=util.cur_stream(torch))
    torch.cuda.synchronize()
    assert torch.equal(top, x.max(-1).values)
    scale = x.double().abs().sum(-1)
    assert float(((total - x.double().sum(-1)).abs() / scale).max()) <= CLOSE[dtype]


# 148 SMs x 8 CTAs x 512 threads take a value each, eight times at once; fewer values, fewer CTAs
STEP = 148 * 8 * 512


@pytest.mark.parametrize("dtype", TYPES)
@pytest.mark.parametrize("gated", [True, False])
@pytest.mark.parametrize("n", [1, 511, 513, STEP - 1, STEP + 1, 7 * STEP + 3, 8 * STEP - 1, 8 * STEP + 1, 17 * STEP + 5])
def test_silu_of_odd_lengths(dev, pkg, dtype, gated, n):
    gate, up = rnd(n, dtype=dtype), rnd(n, dtype=dtype, seed=2)
    y = torch.full((n + 3,), 7.0, device="cuda:0", dtype=TYPES[dtype])
    dev.silu_mul(code(pkg.capi, dtype), 1, n, gate.data_ptr(), up.data_ptr() if gated else None, y.data_ptr(), stream=util.cur_stream(torch))
    torch.cuda.synchronize()
    want = torch.nn.functional.silu(gate.double()) * (up.double() if gated else 1.0)
    assert float(((y[:n] - want).abs() / want.abs().clamp_min(1e-3)).max()) <= CLOSE[dtype]
    assert bool((y[n:] == 7.0).all())
