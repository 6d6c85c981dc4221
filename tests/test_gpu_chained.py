"""Calls whose kernels are placed while the one before still runs: each reads what the call before it wrote, also where it fetches
into the L2 before that call has ended.  From Python a call takes longer to issue than most of these kernels run, so the calls are also
queued behind a product that runs longer than issuing them takes, and captured and replayed."""
import pytest

import util

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")
HALF = torch.bfloat16


def rnd(*shape, dtype=HALF, seed=1, sigma=1.0):
    g = torch.Generator(device="cuda:0")
    g.manual_seed(seed)
    return (torch.randn(shape, generator=g, device="cuda:0") * sigma).to(dtype)


def buf(*shape, dtype=HALF):
    return torch.empty(shape, dtype=dtype, device="cuda:0")


# Each makes its tensors and returns the chain, as a function of what to do between two calls and of the stream, and the tensors it changes.
def weights_made_before(dev, capi):
    """B of the second product is C of the first, and the tiles it fetches early are those the first writes last."""
    a, b, x = rnd(2048, 512, sigma=0.1), rnd(512, 2048, seed=2), rnd(16, 2048, seed=3)
    w, y, z = buf(2048, 2048), buf(16, 2048), buf(16, 2048)

    def calls(sync, st):
        for k in range(4):
            b.mul_(-1.0)
            dev.gemm(capi.BF16, 2048, 2048, 512, a.data_ptr(), b.data_ptr(), w.data_ptr(), stream=st)
            sync()
            for bt in (True, False):
                dev.gemm(capi.BF16, 16, 2048, 2048, x.data_ptr(), w.data_ptr(), y.data_ptr(), b_transposed=bt, stream=st)
                sync()
                dev.silu_mul(capi.BF16, 16, 2048, y.data_ptr(), x.data_ptr(), z.data_ptr(), stream=st)
                sync()
                dev.softmax(capi.BF16, 16, 2048, z.data_ptr(), x.data_ptr(), stream=st)
                sync()
                dev.rms_norm(capi.BF16, 16, 2048, 1e-5, x.data_ptr(), x.data_ptr(), stream=st)
                sync()

    return calls, [b, w, y, z, x]


def odd_sizes(dev, capi):
    """Padded copies and products split on the way in, in turn, each on the result before it."""
    x, w = rnd(700, 701, sigma=0.04), rnd(701, 701, seed=2, sigma=0.04)
    f, g = rnd(700, 704, dtype=torch.float32, sigma=0.04), rnd(704, 704, dtype=torch.float32, seed=4, sigma=0.04)
    y, h = buf(700, 701), buf(700, 704, dtype=torch.float32)

    def calls(sync, st):
        for k in range(4):
            dev.gemm(capi.BF16, 700, 701, 701, x.data_ptr(), w.data_ptr(), y.data_ptr(), stream=st)
            sync()
            dev.softmax(capi.BF16, 700, 701, y.data_ptr(), x.data_ptr(), stream=st)
            sync()
            dev.gemm(capi.F32, 700, 704, 704, f.data_ptr(), g.data_ptr(), h.data_ptr(), stream=st)
            sync()
            dev.gemm(capi.F32, 700, 704, 704, h.data_ptr(), g.data_ptr(), f.data_ptr(), b_transposed=True, stream=st)
            sync()

    return calls, [x, y, f, h]


def one_token_at_a_time(dev, capi, dtype=HALF, batch=1, heads=8):
    code = capi.F32 if dtype == torch.float32 else capi.BF16
    new, seq, kv, d = 4, 9000, 2, 128
    q, k_new, v_new = rnd(new, batch, kv * heads, d, dtype=dtype), rnd(new, batch, kv, d, dtype=dtype, seed=2, sigma=4.0), rnd(new, batch, kv, d, dtype=dtype, seed=3)
    k, v = rnd(batch, kv, seq, d, dtype=dtype, seed=4), rnd(batch, kv, seq, d, dtype=dtype, seed=5)
    o = buf(new, batch, kv * heads, d, dtype=dtype)

    def calls(sync, st):
        for t in range(new):
            at = 3 + t  # among the rows that a CTA fetches first
            for x, n in ((q[t], kv * heads), (k_new[t], kv)):
                dev.rope(code, batch, 1, n, d, at, 1e4, x.data_ptr(), stream=st)
                sync()
            for src, dst in ((k_new[t], k), (v_new[t], v)):
                dev.kv_cache_update(code, batch, 1, kv, d, at, seq, src.data_ptr(), dst.data_ptr(), stream=st)
                sync()
            dev.attention_decode(code, batch, kv * heads, kv, seq, seq, d, q[t].data_ptr(), k.data_ptr(), v.data_ptr(), o[t].data_ptr(), stream=st)
            sync()
            if t + 1 < new:  # the next token's query takes in this one's result
                q[t + 1].add_(o[t])
                sync()

    return calls, [q, k_new, o, k, v]


def prompt_in_chunks(dev, capi, d=128):
    new, chunks, kv, hq, top = 200, 3, 2, 4, 6000
    q, k_new, v_new = rnd(chunks, new, hq, d), rnd(chunks, new, kv, d, seed=2), rnd(chunks, new, kv, d, seed=3)
    k, v, o = rnd(kv, top, d, seed=4), rnd(kv, top, d, seed=5), buf(chunks, new, hq, d)
    p = buf(chunks, hq, new, d)

    def calls(sync, st):
        for c in range(chunks):
            at = 4500 + c * new
            dev.rope(capi.BF16, 1, new, hq, d, at, 1e4, q[c].data_ptr(), stream=st)
            sync()
            dev.rope(capi.BF16, 1, new, kv, d, at, 1e4, k_new[c].data_ptr(), stream=st)
            sync()
            for src, dst in ((k_new[c], k), (v_new[c], v)):
                dev.kv_cache_update(capi.BF16, 1, new, kv, d, at, top, src.data_ptr(), dst.data_ptr(), stream=st)
                sync()
            dev.attention_prefill(capi.BF16, hq, kv, new, at, top, d, q[c].data_ptr(), k.data_ptr(), v.data_ptr(), o[c].data_ptr(), stream=st)
            sync()
            # the result, read as heads, as queries, keys and values of plain attention
            dev.attention(capi.BF16, 1, hq, hq, new, d, o[c].data_ptr(), o[c].data_ptr(), o[c].data_ptr(), p[c].data_ptr(), causal=True, stream=st)
            sync()

    return calls, [q, k_new, o, k, v, p]


CHAINS = {
    "weights made before": weights_made_before,
    "odd sizes": odd_sizes,
    "decode, one sequence": one_token_at_a_time,
    "decode, a batch": lambda *a: one_token_at_a_time(*a, batch=40),
    "decode, f32, 8 heads": lambda *a: one_token_at_a_time(*a, dtype=torch.float32, batch=4),
    "decode, f32, 1 head": lambda *a: one_token_at_a_time(*a, dtype=torch.float32, batch=4, heads=1),
    "prefill": prompt_in_chunks,
    "prefill, heads of 64": lambda *a: prompt_in_chunks(*a, d=64),
}


@pytest.mark.parametrize("name", CHAINS)
def test_a_chain_gives_the_bits_of_its_calls_one_by_one(dev, pkg, name):
    capi = pkg.capi
    # two of the same, for two streams; seeded, so alike
    chains = [CHAINS[name](dev, capi) for _ in range(2)]
    first = [t.clone() for t in chains[0][1]]
    st = util.cur_stream(torch)
    chains[0][0](torch.cuda.synchronize, st)
    torch.cuda.synchronize()
    want = [t.clone() for t in chains[0][1]]

    def reset():
        for _, tensors in chains:
            for t, f in zip(tensors, first):
                t.copy_(f)

    def check(n):
        torch.cuda.synchronize()
        assert dev.status() == 0
        for _, tensors in chains[:n]:
            assert all(torch.equal(a, b) for a, b in zip(tensors, want))

    reset()
    chains[0][0](lambda: None, st)
    check(1)
    reset()
    streams = [torch.cuda.Stream() for _ in range(2)]
    torch.cuda.synchronize()
    for s, (calls, _) in zip(streams, chains):
        with torch.cuda.stream(s):
            calls(lambda: None, s.cuda_stream)
    check(2)

    a, c = rnd(8192, 8192, sigma=0.01), buf(8192, 8192)
    for _ in range(3):
        reset()
        for _ in range(2):  # 1.7 ms
            dev.gemm(capi.BF16, 8192, 8192, 8192, a.data_ptr(), a.data_ptr(), c.data_ptr(), stream=st)
        chains[0][0](lambda: None, st)
        check(1)

    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        chains[0][0](lambda: None, torch.cuda.current_stream().cuda_stream)
    for _ in range(5):
        reset()
        graph.replay()
        check(1)
    del graph
