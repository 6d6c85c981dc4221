"""16-bit heads of 64 and less on tcgen05: the probabilities in place of the scores, three buffers for the jobs of two tiles."""
import pytest

import util

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def reference(q, k, v, causal):
    q, k, v = (t.double() for t in (q, k, v))
    g = q.shape[1] // k.shape[1]
    k, v = k.repeat_interleave(g, 1), v.repeat_interleave(g, 1)
    s = q @ k.transpose(-1, -2) / q.shape[-1] ** 0.5
    if causal:
        s = s.masked_fill(torch.triu(torch.ones(s.shape[-2:], dtype=torch.bool, device=s.device), 1), float("-inf"))
    return torch.softmax(s, -1) @ v


# steps per tile from 1 to 12, tiles with and without a step of their own at the end, and scores that outgrow the maximum in use again
# and again; half a unit in the result's last place, and f32 errors (of probabilities up to 2^8 too large) far below it
@pytest.mark.parametrize("causal", [False, True])
@pytest.mark.parametrize("dtype,d,s,sigma", [(torch.bfloat16, 64, s, 1.0) for s in (65, 128, 129, 256, 384, 385, 512, 640, 1025, 1500)] +
                         [(torch.float16, 64, 777, 5.0), (torch.bfloat16, 64, 1300, 6.0), (torch.bfloat16, 32, 600, 3.0), (torch.float16, 32, 1100, 1.0)])
def test_against_64_bits(dev, pkg, dtype, d, s, sigma, causal):
    g = torch.Generator(device="cuda:0")
    g.manual_seed(s)
    mk = lambda h, x=1.0: (torch.randn((2, h, s, d), generator=g, device="cuda:0") * x).to(dtype)  # noqa: E731
    q, k, v = mk(4, sigma), mk(2), mk(2)
    k[:, :, ::7] *= torch.linspace(0.2, 2.0, k[:, :, ::7].shape[2], device="cuda:0").to(dtype)[:, None]  # later keys outweigh earlier ones
    o = torch.empty_like(q)
    code = pkg.capi.BF16 if dtype == torch.bfloat16 else pkg.capi.F16
    dev.attention(code, 2, 4, 2, s, d, q.data_ptr(), k.data_ptr(), v.data_ptr(), o.data_ptr(), causal=causal, stream=util.cur_stream(torch))
    torch.cuda.synchronize()
    assert dev.status() == 0
    want = reference(q, k, v, causal)
    half_ulp = 2.0 ** (-9 if dtype == torch.bfloat16 else -12)
    assert float(((o.double() - want).abs() - 2.05 * half_ulp * want.abs()).max()) <= 6e-5
    again = torch.empty_like(q)
    dev.attention(code, 2, 4, 2, s, d, q.data_ptr(), k.data_ptr(), v.data_ptr(), again.data_ptr(), causal=causal, stream=util.cur_stream(torch))
    torch.cuda.synchronize()
    assert torch.equal(o, again)
