"""f32 attention on the tcgen05 kernel against 64 bits: steps of 64 keys and tiles of 128 rows that end anywhere, few rows on many keys, rows whose
scores grow from step to step, keys behind a row's last one."""
import pytest

import util

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def rnd(g, *shape):
    return torch.randn(shape, generator=g, device="cuda:0")


def want(q, k, v, seen):
    k, v = (t.double().repeat_interleave(q.shape[0] // k.shape[0], 0) for t in (k, v))
    s = (q.double() @ k.transpose(1, 2) / q.shape[2] ** 0.5).masked_fill(~seen, float("-inf"))
    return torch.softmax(s, -1) @ v


@pytest.mark.parametrize("causal", [False, True])
@pytest.mark.parametrize("batch,hq,hkv,seq,d", [(1, 2, 1, 1, 128), (2, 2, 2, 63, 128), (1, 3, 1, 64, 128), (1, 4, 2, 65, 128), (1, 2, 2, 127, 128), (3, 2, 1, 129, 128),
                                                (1, 2, 2, 193, 96), (1, 1, 1, 65, 96), (2, 4, 2, 65, 64), (1, 2, 1, 640, 64), (1, 2, 2, 161, 32), (1, 200, 100, 257, 32)])
def test_against_64_bits(dev, pkg, batch, hq, hkv, seq, d, causal):
    g = torch.Generator(device="cuda:0")
    g.manual_seed(seq + d)
    q, k, v = rnd(g, batch, hq, seq, d), rnd(g, batch, hkv, seq, d), rnd(g, batch, hkv, seq, d)
    o, again = torch.empty_like(q), torch.empty_like(q)
    for out in (o, again):
        dev.attention(pkg.capi.F32, batch, hq, hkv, seq, d, q.data_ptr(), k.data_ptr(), v.data_ptr(), out.data_ptr(), causal=causal, stream=util.cur_stream(torch))
    torch.cuda.synchronize()
    assert dev.status() == 0 and torch.equal(o, again)
    seen = torch.ones(seq, seq, dtype=torch.bool, device="cuda:0")
    seen = torch.tril(seen) if causal else seen
    for b in range(batch):
        w = want(q[b], k[b], v[b], seen)
        # 24 bits of every operand; sums of 128 and of 64 terms: 2.6e-7 measured at most, three times that
        assert float((o[b].double() - w).norm() / w.norm()) <= 8e-7


@pytest.mark.parametrize("new,start,hq,hkv,d", [(1, 300, 4, 2, 128), (20, 1000, 8, 8, 128), (130, 62, 2, 1, 64), (63, 65, 3, 3, 96), (5, 4000, 2, 1, 32)])
def test_a_few_rows_on_many_keys(dev, pkg, new, start, hq, hkv, d):
    g = torch.Generator(device="cuda:0")
    g.manual_seed(new + start)
    total = start + new
    q, k, v = rnd(g, new, hq, d), rnd(g, hkv, total + 9, d), rnd(g, hkv, total + 9, d)
    k[:, total:], v[:, total:] = float("nan"), float("nan")  # not filled yet
    o = torch.empty_like(q)
    dev.attention_prefill(pkg.capi.F32, hq, hkv, new, start, total + 9, d, q.data_ptr(), k.data_ptr(), v.data_ptr(), o.data_ptr(), stream=util.cur_stream(torch))
    torch.cuda.synchronize()
    assert dev.status() == 0
    seen = torch.arange(total, device="cuda:0")[None, :] <= start + torch.arange(new, device="cuda:0")[:, None]
    w = want(q.transpose(0, 1), k[:, :total], v[:, :total], seen).transpose(0, 1)
    assert float((o.double() - w).norm() / w.norm()) <= 8e-7


@pytest.mark.parametrize("d", [64, 128])
def test_scores_that_grow_with_every_step(dev, pkg, d):
    """Every step raises the running maximum by more than 2^8, so that all sums before it are scaled down; then every step lowers it."""
    g = torch.Generator(device="cuda:0")
    g.manual_seed(d)
    seq = 500
    q, v = rnd(g, 2, seq, d), rnd(g, 2, seq, d)
    q[..., 0] = 8.0
    for sign in (1, -1):
        k = rnd(g, 2, seq, d) * 0.1
        k[..., 0] = sign * torch.arange(seq, device="cuda:0") // 64 * 12.0
        o = torch.empty_like(q)
        dev.attention(pkg.capi.F32, 1, 2, 2, seq, d, q.data_ptr(), k.data_ptr(), v.data_ptr(), o.data_ptr(), causal=True, stream=util.cur_stream(torch))
        torch.cuda.synchronize()
        w = want(q, k, v, torch.tril(torch.ones(seq, seq, dtype=torch.bool, device="cuda:0")))
        # scores reach 8 * 84 / sqrt(d) = 84: an error of half a unit in their last place, 4e-6, goes into the exponentials
        assert float((o.double() - w).norm() / w.norm()) <= 1e-5


def attend(dev, pkg, q, k, v):
    o = torch.empty_like(q)
    dev.attention(pkg.capi.F32, 1, q.shape[0], k.shape[0], q.shape[1], q.shape[2], q.data_ptr(), k.data_ptr(), v.data_ptr(), o.data_ptr(), causal=False, stream=util.cur_stream(torch))
    torch.cuda.synchronize()
    assert dev.status() == 0
    w = want(q, k, v, torch.ones(q.shape[1], k.shape[1], dtype=torch.bool, device="cuda:0"))
    return float((o.double() - w).norm() / w.norm())


@pytest.mark.parametrize("seq,d", [(96, 64), (300, 128), (200, 96), (400, 32)])
@pytest.mark.parametrize("v_scale,k_scale", [(1e-35, 1), (1e-37, 1), (1e36, 1), (1, 1e-36), (1, 1e-30), (1, 1e36)])
def test_tiny_and_huge_operands(dev, pkg, seq, d, v_scale, k_scale):
    """Q is as much larger as K is smaller.  Two TF32 numbers lost bits below 2^-136 (V of 1e-37 3e-5 off), three bf16 numbers as they are below 2^-133 (3e-4); the
    parts keep those from 2^-142 on."""
    g = torch.Generator(device="cuda:0")
    g.manual_seed(seq + d)
    q, k, v = ((rnd(g, 2, seq, d).double() * s).float() for s in (1 / k_scale, k_scale, v_scale))
    assert attend(dev, pkg, q, k, v) <= 8e-7 + 2.0 ** -142 / min(v_scale, k_scale, 1 / k_scale)


@pytest.mark.parametrize("seq,d", [(96, 64), (300, 128), (200, 96), (400, 32)])
def test_tiny_probabilities(dev, pkg, seq, d):
    """One key has a weight of nearly one and a V of zero; what the others, of weights about e^-85 = 1e-37, add up to is the result."""
    g = torch.Generator(device="cuda:0")
    g.manual_seed(seq + d)
    q, k, v = torch.zeros(2, seq, d, device="cuda:0"), torch.zeros(2, seq, d, device="cuda:0"), rnd(g, 2, seq, d)
    q[..., 0] = d ** 0.5
    k[..., 0] = torch.randint(-4, 5, (2, seq), generator=g, device="cuda:0") / 4
    k[:, 0, 0], v[:, 0] = 85.0, 0.0
    # scores are 123 in the exponents' units, half a unit in whose last place is 4e-6, twice
    assert attend(dev, pkg, q, k, v) <= 1e-5
