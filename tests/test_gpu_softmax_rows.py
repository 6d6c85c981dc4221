"""Row softmax over rows of any alignment and width, on the GPU through the C ABI."""
import numpy as np
import pytest

import util

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

KIND = {"f32": (torch.float32, 0), "f16": (torch.float16, 1), "bf16": (torch.bfloat16, 2)}
# against the 64-bit result: f32 as everywhere; 16 bit half a unit in the last place plus the f32 error
RTOL = {"f32": 1e-5, "f16": 2.0 ** -11 + 1e-5, "bf16": 2.0 ** -8 + 1e-5}


def check(dev, name, x, offset_y=None, offset=0):
    """x: 2-D device tensor; both buffers start `offset` elements after a 16-byte boundary (y: `offset_y`)."""
    t, code = KIND[name]
    rows, cols = x.shape
    off_y = offset if offset_y is None else offset_y
    xb = torch.zeros(rows * cols + 16, dtype=t, device="cuda:0")
    yb = torch.full((rows * cols + 32,), 5.0, dtype=t, device="cuda:0")
    xb[offset:offset + rows * cols] = x.reshape(-1)
    dev.softmax(code, rows, cols, xb.data_ptr() + offset * xb.element_size(), yb.data_ptr() + off_y * yb.element_size(),
                stream=util.cur_stream(torch))
    torch.cuda.synchronize()
    assert (yb[:off_y] == 5).all() and (yb[off_y + rows * cols:] == 5).all()  # nothing outside the rows is written
    got = yb[off_y:off_y + rows * cols].reshape(rows, cols).double()
    want = torch.softmax(x.double(), -1)
    assert torch.equal(got.isnan(), want.isnan())
    err = ((got - want).abs() - 1e-30 - (2.0 ** -25 if name == "f16" else 0.0)).nan_to_num()  # f16: half its smallest step
    assert (err <= RTOL[name] * want.nan_to_num()).all(), float((err / want.clamp_min(1e-30)).nan_to_num().max())


def rows_of(name, rows, cols, seed):
    g = torch.Generator(device="cuda:0")
    g.manual_seed(seed)
    return (torch.randn((rows, cols), generator=g, device="cuda:0") * 3).to(KIND[name][0])


@pytest.mark.parametrize("name", ["f32", "bf16", "f16"])
@pytest.mark.parametrize("rows,cols", [(9, 1), (7, 2), (5, 31), (6, 255), (5, 1023), (4, 1025), (3, 2041), (3, 2047), (3, 2050), (700, 4099),
                                       (5, 8191), (4, 16385), (3, 32771), (3, 50001), (3, 65537), (2, 131072), (2, 131069), (2, 262147)])
def test_any_width(dev, name, rows, cols):
    check(dev, name, rows_of(name, rows, cols, cols))


@pytest.mark.parametrize("name", ["f32", "bf16", "f16"])
@pytest.mark.parametrize("cols", [64, 1000, 4096, 40000])
def test_any_start(dev, name, cols):
    x = rows_of(name, 5, cols, 7)
    for offset in (1, 3):
        check(dev, name, x, offset=offset)
    check(dev, name, x, offset=1, offset_y=2)  # x and y at different offsets from a boundary


# rows for all SMs, read twice by CTAs of 1024, 512 and 256 threads, whose steps end with the row or before it
@pytest.mark.parametrize("name", ["f32", "bf16", "f16"])
@pytest.mark.parametrize("rows,cols", [(120, 8200), (148, 32771), (149, 16387), (149, 65536), (300, 16387), (300, 24576), (250, 520), (320, 1111)])
def test_many_rows(dev, name, rows, cols):
    check(dev, name, rows_of(name, rows, cols, cols))


@pytest.mark.parametrize("name", ["f32", "bf16", "f16"])
@pytest.mark.parametrize("rows,cols", [(8, 33), (8, 3001), (8, 50001), (149, 20001), (300, 1111), (300, 20001)])
def test_masks_and_specials(dev, name, rows, cols):
    x = rows_of(name, rows, cols, 9)
    low = torch.finfo(KIND[name][0]).min
    x[0, cols // 2:] = float("-inf")   # a half that is masked out: whole warps and CTAs see nothing but -inf
    x[1, :-1] = float("-inf")
    x[2, :] = float("-inf")            # nothing left: NaN
    x[3, cols // 3:] = low             # a mask of the type's lowest value
    x[4, :] = low                      # ... everywhere: uniform
    x[5, 1] = float("nan")
    x[6, cols - 1] = float("inf")
    check(dev, name, x)
