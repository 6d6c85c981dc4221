"""Softmax of more rows than CTAs at once: a row to a CTA, two rows to a CTA with an odd number of rows, rows read twice by CTAs that go after one."""
import pytest

import util

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16, torch.float16])
@pytest.mark.parametrize("rows,cols", [(1, 4096), (5001, 2056), (3999, 4096), (1185, 8192), (2369, 3000), (7001, 1032), (1777, 30001), (1000, 50008), (593, 16384)])
def test_against_64_bits(dev, pkg, dtype, rows, cols):
    g = torch.Generator(device="cuda:0")
    g.manual_seed(rows)
    x = (torch.randn((rows, cols), generator=g, device="cuda:0") * 3).to(dtype)
    x[rows // 2, : cols // 2] = float("-inf")
    x[rows - 1] = 7.0
    y = torch.full((rows + 1, cols), 7.0, dtype=dtype, device="cuda:0")
    code = {torch.float32: pkg.capi.F32, torch.bfloat16: pkg.capi.BF16, torch.float16: pkg.capi.F16}[dtype]
    dev.softmax(code, rows, cols, x.data_ptr(), y.data_ptr(), stream=util.cur_stream(torch))
    torch.cuda.synchronize()
    for at in range(0, rows, 512):
        want = torch.softmax(x[at:at + 512].double(), -1)
        got = y[at:min(at + 512, rows)].double()
        if dtype == torch.float32:
            assert float(((got - want).norm(dim=-1) / want.norm(dim=-1)).max()) <= 1e-6
        else:  # half of the result's last place, and what the f32 value is off: 2^-18 of it
            last = 2.0 ** -9 if dtype == torch.bfloat16 else 2.0 ** -12
            assert float(((got - want).abs() - want * (2 * last) * 1.02).max()) <= 2.0 ** -25
    assert bool((y[rows] == 7.0).all())
