"""The work this library is measured on, and how its results are checked.

Each case is one call, or one short chain of calls, of ``CudaSm100Device`` on device memory: row softmax, matmul,
fused attention, and the steps of a transformer layer around them (norm, gated MLP, rotary embedding, KV-cache
append, prefill and decode attention).  ``listed()`` names the cases, ``draw()`` picks others of the same ranges.
"""
from __future__ import annotations

import importlib
import math

import torch

tsm = importlib.import_module("tile-rs_b200")
capi, hal = tsm.capi, tsm.hal

TORCH = {"f32": torch.float32, "bf16": torch.bfloat16, "f16": torch.float16}
CODE = {"f32": capi.F32, "bf16": capi.BF16, "f16": capi.F16}
SIZE = {"f32": 4, "bf16": 2, "f16": 2}
GPU = "cuda:0"
EPS, THETA = 1e-5, 10000.0

_DEVICE = None


def device():
    """One open device per process, as a program of this library keeps it."""
    global _DEVICE
    if _DEVICE is None:
        _DEVICE = hal.CudaSm100Device(0)
    return _DEVICE


def stream():
    return torch.cuda.current_stream().cuda_stream


# ---- the cases --------------------------------------------------------------------------------------------------
def listed():
    return [
        # a classifier's scores over a small batch: the whole call is launch latency
        {"name": "softmax_f32_256x1000", "op": "softmax", "dtype": "f32", "rows": 256, "cols": 1000},
        # the headline softmax configuration: a stream of 4096-wide rows through HBM
        {"name": "softmax_f32_65536x4096", "op": "softmax", "dtype": "f32", "rows": 65536, "cols": 4096},
        # next-token probabilities over a vocabulary of odd size: rows that do not start on 16-byte boundaries
        {"name": "softmax_bf16_1000x50001", "op": "softmax", "dtype": "bf16", "rows": 1000, "cols": 50001},
        # the gated MLP of one decoding step for 16 sequences: norm, three projections with [out, in] weights, SiLU * up
        {"name": "mlp_bf16_16tokens", "op": "mlp", "dtype": "bf16", "tokens": 16, "hidden": 4096, "inner": 16384},
        # the headline matmul configuration
        {"name": "gemm_bf16_8192", "op": "gemm", "dtype": "bf16", "bt": False, "batch": 1, "m": 8192, "n": 8192, "k": 8192},
        # the small f32 matmul configuration
        {"name": "gemm_f32_512", "op": "gemm", "dtype": "f32", "bt": False, "batch": 1, "m": 512, "n": 512, "k": 512},
        # numerical work on a matrix of odd sizes: no row starts on a 16-byte boundary
        {"name": "gemm_f32_1999x3001x1501", "op": "gemm", "dtype": "f32", "bt": False, "batch": 1, "m": 1999, "n": 3001, "k": 1501},
        # the headline attention configuration: causal training-size forward
        {"name": "attention_bf16_b8h32_s4096", "op": "attention", "dtype": "bf16", "causal": True, "batch": 8, "hq": 32, "hkv": 32,
         "seq": 4096, "d": 128},
        # grouped heads of 64 and a sequence that ends inside a tile
        {"name": "attention_bf16_d64_s2000", "op": "attention", "dtype": "bf16", "causal": True, "batch": 4, "hq": 32, "hkv": 8,
         "seq": 2000, "d": 64},
        # the f32 attention workload, the element type of the tile intrinsic itself
        {"name": "attention_f32_h16_s4096", "op": "attention", "dtype": "f32", "causal": True, "batch": 1, "hq": 16, "hkv": 16,
         "seq": 4096, "d": 128},
        # one chunk of a long prompt: rotate, append to the cache, attend to everything before
        {"name": "prefill_bf16_512_on_15872", "op": "prefill", "dtype": "bf16", "hq": 32, "hkv": 8, "new": 512, "start": 15872,
         "max_seq": 16384, "d": 128},
        # one generated token of one long sequence: append to the cache, attend
        {"name": "decode_bf16_b1_s32768", "op": "decode", "dtype": "bf16", "batch": 1, "hq": 32, "hkv": 8, "seq": 32768,
         "max_seq": 32768, "d": 128},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    op = rng.choice(["softmax", "softmax", "mlp", "gemm16", "gemm16", "gemm32", "gemm32", "attention", "attention", "prefill", "decode"])
    half = rng.choice(["bf16", "bf16", "f16"])
    if op == "softmax":
        dtype, cols = rng.choice(["f32", half]), _log(rng, 32, 130000)
        if rng.random() < 0.6:
            cols = max(32, cols // 8 * 8)
        rows = _log(rng, 8, max(16, min(65536, (1 << 27) // cols)))
        return {"op": "softmax", "dtype": dtype, "rows": rows, "cols": cols}
    if op == "mlp":
        hidden = 256 * _log(rng, 4, 32)
        return {"op": "mlp", "dtype": half, "tokens": _log(rng, 1, 300), "hidden": hidden, "inner": hidden * rng.choice([2, 3, 4])}
    if op == "gemm16":
        bt, batch = rng.random() < 0.5, rng.choice([1, 1, 1, 4])
        m, n, k = (_log(rng, lo, 6000) for lo in (1, 64, 64))
        if rng.random() < 0.75:  # the usual case: everything but the token count is a multiple of 8
            n, k = max(64, n // 8 * 8), max(64, k // 8 * 8)
        else:
            m = min(m, max(1, int(1.5e10 / (2.0 * n * k * batch))))
        return {"op": "gemm", "dtype": half, "bt": bt, "batch": batch, "m": m, "n": n, "k": k}
    if op == "gemm32":  # rows on 16-byte boundaries, or odd ones that never are
        m, n, k = (_log(rng, 64, 2600) for _ in range(3))
        if rng.random() < 0.5:
            n, k = n // 4 * 4, k // 4 * 4
        else:
            n, k = n | 1, k | 1
        return {"op": "gemm", "dtype": "f32", "bt": rng.random() < 0.5, "batch": 1, "m": m, "n": n, "k": k}
    d = rng.choice([64, 128, 128])
    group = rng.choice([1, 2, 4, 8])
    if op == "attention":
        dtype = rng.choice(["f32", half, half])
        hq = group * rng.choice([2, 4, 8])
        batch = rng.choice([1, 2, 4])
        top = math.sqrt((4e10 if dtype == "f32" or d != 128 else 4e11) / (4.0 * batch * hq * d))
        if dtype != "f32" and rng.random() < 0.15:
            d = rng.choice([32, 96])
        return {"op": "attention", "dtype": dtype, "causal": rng.random() < 0.6, "batch": batch, "hq": hq, "hkv": hq // group,
                "seq": min(8192, _log(rng, 64, max(128, top))), "d": d}
    if op == "prefill":
        new, start = _log(rng, 17, 2048), _log(rng, 1, 16384)
        return {"op": "prefill", "dtype": half, "hq": 4 * group, "hkv": 4, "new": new, "start": start,
                "max_seq": new + start + rng.randrange(0, 200), "d": 128}
    seq, batch = _log(rng, 100, 40000), _log(rng, 1, 64)
    if seq * batch > 400000:
        batch = max(1, 400000 // seq)
    return {"op": "decode", "dtype": rng.choice(["f32", half, half]), "batch": batch, "hq": group * 8, "hkv": 8, "seq": seq,
            "max_seq": seq + rng.randrange(0, 100), "d": d}


# ---- inputs -----------------------------------------------------------------------------------------------------
def _normal(gen, shape, dtype, sigma=1.0):
    out = torch.empty(shape, dtype=TORCH[dtype], device=GPU)
    flat, step = out.view(-1), 1 << 26
    for at in range(0, flat.numel(), step):
        n = min(step, flat.numel() - at)
        flat[at:at + n] = torch.randn(n, generator=gen, device=GPU) * sigma
    return out


def _softmax_input(gen, shape, dtype):
    """3 * N(0, 1) with about one position in a hundred at +20: rows of scores with a few that stand out."""
    x = _normal(gen, shape, dtype, 3.0)
    flat, step = x.view(-1), 1 << 26
    for at in range(0, flat.numel(), step):
        n = min(step, flat.numel() - at)
        flat[at:at + n].masked_fill_(torch.rand(n, generator=gen, device=GPU) < 0.01, 20.0)
    return x


def prepare(case, seed):
    gen = torch.Generator(device=GPU)
    gen.manual_seed(int(seed))
    c, t = dict(case), case["dtype"]
    s = {"case": c, "dev": device()}
    if c["op"] == "softmax":
        s["x"] = _softmax_input(gen, (c["rows"], c["cols"]), t)
        s["y"] = torch.empty_like(s["x"])
    elif c["op"] == "mlp":
        n, h, f = c["tokens"], c["hidden"], c["inner"]
        s["x"] = _normal(gen, (n, h), t)
        s["gate_w"], s["up_w"] = (_normal(gen, (f, h), t, h ** -0.5) for _ in range(2))
        s["down_w"] = _normal(gen, (h, f), t, f ** -0.5)
        s["norm"], s["y"] = torch.empty_like(s["x"]), torch.empty_like(s["x"])
        s["gate"], s["up"], s["act"] = (torch.empty((n, f), dtype=TORCH[t], device=GPU) for _ in range(3))
    elif c["op"] == "gemm":
        b, m, n, k = c["batch"], c["m"], c["n"], c["k"]
        sigma = k ** -0.25
        s["a"] = _normal(gen, (b, m, k), t, sigma)
        s["b"] = _normal(gen, (b, n, k) if c["bt"] else (b, k, n), t, sigma)
        s["c"] = torch.empty((b, m, n), dtype=TORCH[t], device=GPU)
    elif c["op"] == "attention":
        b, q, kv, n, d = c["batch"], c["hq"], c["hkv"], c["seq"], c["d"]
        s["q"] = _normal(gen, (b, q, n, d), t)
        s["k"], s["v"] = (_normal(gen, (b, kv, n, d), t) for _ in range(2))
        s["o"] = torch.empty_like(s["q"])
    elif c["op"] == "prefill":
        s["q"] = _normal(gen, (c["new"], c["hq"], c["d"]), t)
        s["k_new"], s["v_new"] = (_normal(gen, (c["new"], c["hkv"], c["d"]), t) for _ in range(2))
        s["k"], s["v"] = (_normal(gen, (c["hkv"], c["max_seq"], c["d"]), t) for _ in range(2))
        s["q_rot"], s["k_rot"], s["o"] = torch.empty_like(s["q"]), torch.empty_like(s["k_new"]), torch.empty_like(s["q"])
    else:
        s["q"] = _normal(gen, (c["batch"], c["hq"], c["d"]), t)
        s["k_new"], s["v_new"] = (_normal(gen, (c["batch"], c["hkv"], c["d"]), t) for _ in range(2))
        s["k"], s["v"] = (_normal(gen, (c["batch"], c["hkv"], c["max_seq"], c["d"]), t) for _ in range(2))
        s["o"] = torch.empty_like(s["q"])
    return s


# ---- one pass ---------------------------------------------------------------------------------------------------
def run(s):
    c, dev, st = s["case"], s["dev"], stream()
    t = CODE[c["dtype"]]
    if c["op"] == "softmax":
        dev.softmax(t, c["rows"], c["cols"], s["x"].data_ptr(), s["y"].data_ptr(), stream=st)
        return s["y"]
    if c["op"] == "mlp":
        n, h, f = c["tokens"], c["hidden"], c["inner"]
        norm, gate, up, act = (s[k].data_ptr() for k in ("norm", "gate", "up", "act"))
        dev.rms_norm(t, n, h, EPS, s["x"].data_ptr(), norm, stream=st)
        dev.gemm(t, n, f, h, norm, s["gate_w"].data_ptr(), gate, b_transposed=True, stream=st)
        dev.gemm(t, n, f, h, norm, s["up_w"].data_ptr(), up, b_transposed=True, stream=st)
        dev.silu_mul(t, n, f, gate, up, act, stream=st)
        dev.gemm(t, n, h, f, act, s["down_w"].data_ptr(), s["y"].data_ptr(), b_transposed=True, stream=st)
        return s["y"]
    if c["op"] == "gemm":
        dev.gemm(t, c["m"], c["n"], c["k"], s["a"].data_ptr(), s["b"].data_ptr(), s["c"].data_ptr(), b_transposed=c["bt"],
                 batch=c["batch"], stream=st)
        return s["c"]
    if c["op"] == "attention":
        dev.attention(t, c["batch"], c["hq"], c["hkv"], c["seq"], c["d"], s["q"].data_ptr(), s["k"].data_ptr(),
                      s["v"].data_ptr(), s["o"].data_ptr(), causal=c["causal"], stream=st)
        return s["o"]
    kv, d, top = c["hkv"], c["d"], c["max_seq"]
    if c["op"] == "prefill":
        # rope works in place; the projections' outputs are kept, so that the pass can be repeated
        s["q_rot"].copy_(s["q"])
        s["k_rot"].copy_(s["k_new"])
        dev.rope(t, 1, c["new"], c["hq"], d, c["start"], THETA, s["q_rot"].data_ptr(), stream=st)
        dev.rope(t, 1, c["new"], kv, d, c["start"], THETA, s["k_rot"].data_ptr(), stream=st)
        dev.kv_cache_update(t, 1, c["new"], kv, d, c["start"], top, s["k_rot"].data_ptr(), s["k"].data_ptr(), stream=st)
        dev.kv_cache_update(t, 1, c["new"], kv, d, c["start"], top, s["v_new"].data_ptr(), s["v"].data_ptr(), stream=st)
        dev.attention_prefill(t, c["hq"], kv, c["new"], c["start"], top, d, s["q_rot"].data_ptr(), s["k"].data_ptr(),
                              s["v"].data_ptr(), s["o"].data_ptr(), stream=st)
        return s["o"]
    dev.kv_cache_update(t, c["batch"], 1, kv, d, c["seq"] - 1, top, s["k_new"].data_ptr(), s["k"].data_ptr(), stream=st)
    dev.kv_cache_update(t, c["batch"], 1, kv, d, c["seq"] - 1, top, s["v_new"].data_ptr(), s["v"].data_ptr(), stream=st)
    dev.attention_decode(t, c["batch"], c["hq"], kv, c["seq"], top, d, s["q"].data_ptr(), s["k"].data_ptr(),
                         s["v"].data_ptr(), s["o"].data_ptr(), stream=st)
    return s["o"]


# ---- what a pass cannot do without ------------------------------------------------------------------------------
def work(case):
    c, e = case, SIZE[case["dtype"]]
    if c["op"] == "softmax":
        n = c["rows"] * c["cols"]
        return {"bytes": 2 * n * e, "flops": 0}
    if c["op"] == "mlp":
        n, h, f = c["tokens"], c["hidden"], c["inner"]
        return {"bytes": e * (3 * h * f + 2 * n * h), "flops": 6 * n * h * f}
    if c["op"] == "gemm":
        b, m, n, k = c["batch"], c["m"], c["n"], c["k"]
        return {"bytes": e * b * (m * k + k * n + m * n), "flops": 2 * b * m * n * k}
    d = c["d"]
    if c["op"] == "attention":
        n = c["seq"]
        pairs = n * (n + 1) // 2 if c["causal"] else n * n
        return {"bytes": 2 * e * c["batch"] * (c["hq"] + c["hkv"]) * n * d, "flops": 4 * c["batch"] * c["hq"] * pairs * d}
    if c["op"] == "prefill":
        n, past = c["new"], c["start"]
        pairs = n * past + n * (n + 1) // 2
        return {"bytes": e * d * (2 * n * c["hq"] + 2 * c["hkv"] * (past + 2 * n)), "flops": 4 * c["hq"] * pairs * d}
    return {"bytes": e * d * c["batch"] * (2 * c["hq"] + 2 * c["hkv"] * (c["seq"] + 1)),
            "flops": 4 * c["batch"] * c["hq"] * c["seq"] * d}


# ---- how close a correct result is ------------------------------------------------------------------------------
def tolerance(case):
    """About four times the distance from the 64-bit result that was measured over listed and drawn cases; a 16-bit result
    is at least half a unit in its last place away (bf16 1.7e-3 of the value, root mean square, f16 2e-4).  f32 attention
    was 8e-6 away at 4096 keys and 1.4e-5 at its worst: the tensor core's accumulators round toward zero."""
    op, t = case["op"], case["dtype"]
    if t == "f32":
        return {"rel": {"softmax": 1.5e-6, "gemm": 4e-6, "attention": 4e-5, "decode": 4e-6}[op]}
    if op == "mlp":  # the norm, both projections and the activation are rounded too
        return {"rel": 2e-2 if t == "bf16" else 2.5e-3}
    if op == "prefill":  # the rotated q and k and the probabilities are rounded too
        return {"rel": 2e-2 if t == "bf16" else 2.5e-3}
    if op in ("attention", "decode"):  # the probabilities may be rounded to the storage type
        return {"rel": 1e-2 if t == "bf16" else 1.5e-3}
    return {"rel": 7e-3 if t == "bf16" else 1e-3}


# ---- the same in 64 bits ----------------------------------------------------------------------------------------
def _attend(q, k, v, limit):
    """softmax(q k^T / sqrt(d)) v for one head, in 64 bits, 1024 rows at a time; row r sees limit(r) keys."""
    out = torch.empty_like(q)
    place = torch.arange(k.shape[0], device=GPU)
    for at in range(0, q.shape[0], 1024):
        rows = torch.arange(at, min(at + 1024, q.shape[0]), device=GPU)
        sees = limit(rows)
        most = int(sees.max())
        p = q[rows] @ k[:most].T / math.sqrt(q.shape[1])
        p = p.masked_fill(place[None, :most] >= sees[:, None], -math.inf)
        out[rows] = torch.softmax(p, -1) @ v[:most]
    return out


def _rotate(x, start):
    """Pairs (x[2i], x[2i+1]) of token s rotated by (start + s) * theta^(-2i/d); x is [tokens, heads, d]."""
    n, _, d = x.shape
    freq = THETA ** (-torch.arange(0, d, 2, dtype=torch.float64, device=GPU) / d)
    angle = (start + torch.arange(n, dtype=torch.float64, device=GPU))[:, None] * freq
    co, si = angle.cos()[:, None], angle.sin()[:, None]
    a, b = x[..., 0::2], x[..., 1::2]
    return torch.stack((a * co - b * si, a * si + b * co), -1).reshape(x.shape)


def exact(case, seed):
    c = dict(case)
    flops = work(c)["flops"]
    if flops > 3e12:
        return None
    s = prepare(c, seed)
    if c["op"] == "softmax":
        out = torch.empty((c["rows"], c["cols"]), dtype=torch.float64, device=GPU)
        step = max(1, (1 << 26) // c["cols"])
        for at in range(0, c["rows"], step):
            out[at:at + step] = torch.softmax(s["x"][at:at + step].double(), -1)
        return out
    if c["op"] == "mlp":
        x = s["x"].double()
        x = x * torch.rsqrt(x.square().mean(-1, keepdim=True) + EPS)
        gate, up = x @ s["gate_w"].double().T, x @ s["up_w"].double().T
        return (torch.nn.functional.silu(gate) * up) @ s["down_w"].double().T
    if c["op"] == "gemm":
        b = s["b"].double()
        return s["a"].double() @ (b.transpose(1, 2) if c["bt"] else b)
    if c["op"] == "attention":
        n, group = c["seq"], c["hq"] // c["hkv"]
        out = torch.empty(s["q"].shape, dtype=torch.float64, device=GPU)
        sees = (lambda r: r + 1) if c["causal"] else (lambda r: torch.full_like(r, n))
        for b in range(c["batch"]):
            for h in range(c["hq"]):
                out[b, h] = _attend(s["q"][b, h].double(), s["k"][b, h // group].double(), s["v"][b, h // group].double(), sees)
        return out
    group = c["hq"] // c["hkv"]
    if c["op"] == "prefill":
        start, new = c["start"], c["new"]
        q, kn = _rotate(s["q"].double(), start), _rotate(s["k_new"].double(), start)
        k, v = s["k"].double(), s["v"].double()
        k[:, start:start + new], v[:, start:start + new] = kn.transpose(0, 1), s["v_new"].double().transpose(0, 1)
        out = torch.empty_like(q)
        for h in range(c["hq"]):
            out[:, h] = _attend(q[:, h].contiguous(), k[h // group], v[h // group], lambda r: start + r + 1)
        return out
    out = torch.empty(s["q"].shape, dtype=torch.float64, device=GPU)
    for b in range(c["batch"]):
        for g in range(c["hkv"]):
            k, v = s["k"][b, g, :c["seq"]].double(), s["v"][b, g, :c["seq"]].double()
            k[-1], v[-1] = s["k_new"][b, g].double(), s["v_new"][b, g].double()
            p = s["q"][b, g * group:(g + 1) * group].double() @ k.T / math.sqrt(c["d"])
            out[b, g * group:(g + 1) * group] = torch.softmax(p, -1) @ v
    return out
