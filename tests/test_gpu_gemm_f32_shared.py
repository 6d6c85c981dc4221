"""f32 GEMM on CTA pairs whose last tiles are shared: two to four pairs to a tile, the last of them adds the partial sums."""
import pytest

import util

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def rnd(*shape, seed=1, sigma=1.0):
    g = torch.Generator(device="cuda:0")
    g.manual_seed(seed)
    return torch.randn(shape, generator=g, device="cuda:0") * sigma


def product(dev, capi, a, b, m, n, k, bt, batch=1):
    c = torch.full((batch, m, n), float("nan"), device="cuda:0")
    dev.gemm(capi.F32, m, n, k, a.data_ptr(), b.data_ptr(), c.data_ptr(), b_transposed=bt, batch=batch, stream=util.cur_stream(torch))
    torch.cuda.synchronize()
    assert dev.status() == 0
    return c


# 96 tiles of 256 x 256 on 74 pairs (22 shared by three), 85 (11 shared by four), 16 x 3 of a batch (48: none shared), 128-wide tiles,
# and K that does not divide evenly
@pytest.mark.parametrize("m,n,k,bt,batch", [
    (1999, 3001, 1501, False, 1), (2000, 3000, 1500, True, 1), (512, 10880, 999, True, 1), (512, 10881, 1300, False, 1), (1024, 1024, 1000, False, 3),
    (1300, 1300, 2049, False, 1), (600, 10500, 1025, False, 1), (520, 4096, 1024, True, 3)])
def test_against_64_bits_and_twice_the_same(dev, pkg, m, n, k, bt, batch):
    s = k ** -0.25
    a, b = rnd(batch, m, k, sigma=s), rnd(batch, *((n, k) if bt else (k, n)), seed=2, sigma=s)
    c = product(dev, pkg.capi, a, b, m, n, k, bt, batch)
    for i in range(batch):
        want = a[i].double() @ (b[i].double().T if bt else b[i].double())
        err = float((c[i] - want).norm() / want.norm())
        assert err <= (2e-6 if k % 4 == 0 and n % 4 == 0 else 1e-6), err  # as for whole tiles: chunks of 128 and of 64 of K
        assert float((c[i] - want).abs().max() / want.abs().max()) <= 1e-5
    assert torch.equal(product(dev, pkg.capi, a, b, m, n, k, bt, batch), c)  # whoever comes last, the order is one


def test_infinities_in_shared_tiles(dev, pkg):
    """Rows of odd length: outputs that come out infinite or NaN are summed again, also where several pairs made them."""
    m, n, k = 1999, 3001, 1501
    a, b = rnd(m, k, sigma=0.1), rnd(k, n, seed=2, sigma=0.1)
    a[5, 3], a[m - 1, k - 1], b[700, n - 1], b[k - 2, n - 40] = float("inf"), float("-inf"), float("nan"), float("inf")
    c = product(dev, pkg.capi, a, b, m, n, k, False)[0]
    want = (a.double() @ b.double()).float()
    assert torch.equal(c.isnan(), want.isnan()) and torch.equal(c.isinf(), want.isinf())
    assert torch.equal(c[c.isinf()] > 0, want[c.isinf()] > 0)
    ok = want.isfinite()
    assert float((c[ok] - want[ok]).abs().max()) <= 1e-5 * float(want[ok].abs().max())


def test_captured(dev, pkg):
    m, n, k = 1999, 3001, 1501
    a, b, c = rnd(m, k), rnd(k, n, seed=2), torch.zeros(m, n, device="cuda:0")
    want = product(dev, pkg.capi, a, b, m, n, k, False)[0]
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        dev.gemm(pkg.capi.F32, m, n, k, a.data_ptr(), b.data_ptr(), c.data_ptr(), stream=torch.cuda.current_stream().cuda_stream)
    for _ in range(3):
        c.zero_()
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(c, want)
    del graph
