"""f32 GEMM split on the way in: K shared by clusters of every size, shares of unequal length, rows of the sum that do not divide by the cluster."""
import pytest

import util

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


# clusters of 3, 5, 6, 7 and 8; last shares of one k-block; 1 row, a row more than a tile
@pytest.mark.parametrize("bt", [False, True])
@pytest.mark.parametrize("m,n,k,batch", [(1900, 261, 2591, 1), (549, 1064, 900, 1), (300, 260, 1024, 5), (341, 412, 796, 1), (586, 228, 1056, 1), (129, 63, 1057, 7), (2410, 108, 2256, 1),
                                         (85, 257, 387, 1), (1, 131, 1999, 1), (730, 92, 608, 1), (100, 128, 225, 13)])
def test_shares_of_k(dev, pkg, m, n, k, batch, bt):
    g = torch.Generator(device="cuda:0")
    g.manual_seed(m)
    a = torch.randn((batch, m, k), generator=g, device="cuda:0")
    b = torch.randn((batch, n, k) if bt else (batch, k, n), generator=g, device="cuda:0")
    c = torch.full((batch, m, n), 7.0, device="cuda:0")
    dev.gemm(pkg.capi.F32, m, n, k, a.data_ptr(), b.data_ptr(), c.data_ptr(), b_transposed=bt, batch=batch, stream=util.cur_stream(torch))
    torch.cuda.synchronize()
    assert dev.status() == 0
    want = a.double() @ (b.transpose(1, 2) if bt else b).double()
    # 256 of K to an accumulator: 2.4e-7 of the result off for normally distributed data; twice that
    assert float((c.double() - want).norm() / want.norm()) <= 5e-7
