"""Device scratch of the operators: a pool of the library's own, given back, captured into graphs, and done without."""
import ctypes as C
import subprocess
import sys
from pathlib import Path

import pytest

import util

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")
ROOT = Path(__file__).resolve().parent.parent


def bits(t):
    return t.view(torch.int16) if t.element_size() == 2 else t.view(torch.int32)


def rnd(*shape, dtype=torch.bfloat16, seed=1, sigma=1.0):
    g = torch.Generator(device="cuda:0")
    g.manual_seed(seed)
    return (torch.randn(shape, generator=g, device="cuda:0") * sigma).to(dtype)


def calls(capi):
    """The calls that take scratch, by what they take it for: name -> (function name, descriptor, inputs, output)."""
    f32, half = torch.float32, torch.bfloat16
    gemm = lambda t, o, bt, b, m, n, k: capi.GemmDesc(t, o, bt, b, m, n, k)  # noqa: E731
    return {
        "f32 GEMM": ("gemm", gemm(capi.F32, capi.F32, 0, 1, 1024, 2048, 512), [rnd(1024, 512, dtype=f32), rnd(512, 2048, dtype=f32, seed=2)],
                     torch.zeros(1024, 2048, device="cuda:0")),
        "f32 GEMM of odd sizes": ("gemm", gemm(capi.F32, capi.F32, 0, 1, 1025, 2051, 301), [rnd(1025, 301, dtype=f32), rnd(301, 2051, dtype=f32, seed=2)],
                                  torch.zeros(1025, 2051, device="cuda:0")),
        "16-bit GEMM of odd sizes": ("gemm", gemm(capi.BF16, capi.BF16, 0, 1, 300, 301, 1203), [rnd(300, 1203, sigma=0.2), rnd(1203, 301, seed=2, sigma=0.2)],
                                     torch.zeros(300, 301, dtype=half, device="cuda:0")),
        "f32 attention": ("attention", capi.AttentionDesc(capi.F32, 1, 1, 4, 2, 520, 64), [rnd(4, 520, 64, dtype=f32), rnd(2, 520, 64, dtype=f32, seed=2),
                                                                                            rnd(2, 520, 64, dtype=f32, seed=3)], torch.zeros(4, 520, 64, device="cuda:0")),
        "split prefill": ("attention_prefill", capi.AttentionPrefillDesc(capi.BF16, 4, 2, 100, 5000, 5100, 128),
                          [rnd(100, 4, 128), rnd(2, 5100, 128, seed=2), rnd(2, 5100, 128, seed=3)], torch.zeros(100, 4, 128, dtype=half, device="cuda:0")),
        "decode of few caches": ("attention_decode", capi.AttentionDecodeDesc(capi.BF16, 1, 16, 8, 9000, 9000, 128),
                                 [rnd(16, 128), rnd(8, 9000, 128, seed=2), rnd(8, 9000, 128, seed=3)], torch.zeros(16, 128, dtype=half, device="cuda:0")),
        "decode as one stream": ("attention_decode", capi.AttentionDecodeDesc(capi.BF16, 17, 32, 8, 801, 805, 128),
                                 [rnd(17, 32, 128), rnd(17, 8, 805, 128, seed=2), rnd(17, 8, 805, 128, seed=3)], torch.zeros(17, 32, 128, dtype=half, device="cuda:0")),
        "f32 attention of few keys": ("attention", capi.AttentionDesc(capi.F32, 1, 1, 4, 2, 40, 128), [rnd(4, 40, 128, dtype=f32), rnd(2, 40, 128, dtype=f32, seed=2),
                                                                                                       rnd(2, 40, 128, dtype=f32, seed=3)], torch.zeros(4, 40, 128, device="cuda:0")),
        "16-bit GEMM of a short odd K": ("gemm", gemm(capi.F16, capi.F16, 0, 1, 760, 145, 127), [rnd(760, 127, dtype=torch.float16), rnd(127, 145, dtype=torch.float16, seed=2)],
                                         torch.zeros(760, 145, dtype=torch.float16, device="cuda:0")),
    }


NAMES = ["f32 GEMM", "f32 GEMM of odd sizes", "16-bit GEMM of odd sizes", "f32 attention", "split prefill", "decode of few caches", "decode as one stream", "f32 attention of few keys",
         "16-bit GEMM of a short odd K"]


def run(capi, dev, call):
    op, desc, inputs, out = call
    fn = getattr(capi.lib(), f"tsm100_{op}")
    assert fn(dev._h, C.byref(desc), *(x.data_ptr() for x in inputs), out.data_ptr(), util.cur_stream(torch) or None) == capi.OK, capi.last_error()


@pytest.mark.parametrize("name", NAMES)
def test_captured_calls_replay(dev, pkg, name):
    """A graph with such a call can be replayed on new inputs; every replay gives the bits of the call itself."""
    capi = pkg.capi
    call = calls(capi)[name]
    graph = torch.cuda.CUDAGraph()
    run(capi, dev, call)
    torch.cuda.synchronize()
    with torch.cuda.graph(graph):
        run(capi, dev, call)
        run(capi, dev, call)
    for step in range(3):
        for x in call[2]:
            x.copy_((x.float() * 0.5 + 0.25 * step).to(x.dtype))
        call[3].zero_()
        graph.replay()
        torch.cuda.synchronize()
        replayed = call[3].clone()
        call[3].zero_()
        run(capi, dev, call)
        torch.cuda.synchronize()
        assert torch.equal(bits(replayed), bits(call[3])) and bool(call[3].float().abs().sum() > 0)
    assert dev.status() == 0
    del graph


POOL = """
import ctypes as C, sys
sys.path.insert(0, {root!r})
import torch
import __graft_entry__ as entry
pkg = entry.load_package()
torch.zeros(1, device="cuda:0")
cu, pool, keep = C.CDLL("libcuda.so.1"), C.c_void_p(), C.c_uint64(12345678)
assert cu.cuDeviceGetDefaultMemPool(C.byref(pool), 0) == 0
assert cu.cuMemPoolSetAttribute(pool, 4, C.byref(keep)) == 0  # CU_MEMPOOL_ATTR_RELEASE_THRESHOLD
dev, other = pkg.hal.CudaSm100Device(0), pkg.hal.CudaSm100Device(0)
a, b, c = (torch.randn(4096, 4096, device="cuda:0") for _ in range(3))
stream = torch.cuda.current_stream().cuda_stream
free = lambda: (torch.cuda.synchronize(), torch.cuda.mem_get_info()[0])[1]
before = free()
dev.gemm(pkg.capi.F32, 4096, 4096, 4096, a.data_ptr(), b.data_ptr(), c.data_ptr(), stream=stream)
assert dev.status() == 0
held = before - free()
assert cu.cuMemPoolGetAttribute(pool, 4, C.byref(keep)) == 0 and keep.value == 12345678, keep.value
assert held >= 4 * 4096 * 4096 * 4, held  # four planes: kept for the next call
other.close()
assert before - free() == held  # one handle is still open
dev.close()
assert before - free() < held // 4, (held, before - free())
"""


def test_the_default_pool_is_left_alone_and_scratch_is_given_back():
    r = subprocess.run([sys.executable, "-c", POOL.format(root=str(ROOT))], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr


NO_SCRATCH = """
#define TSM100_SCRATCH_LIMIT 0
#include "ops.cuh"
using namespace tsm100;
#define CALL(NAME, DESC, ...) \\
  extern "C" int32_t no_scratch_##NAME(const DESC* d, const void* a, const void* b, const void* v, void* o, uint32_t* status, void* s) { \\
    std::string err; return ops::NAME(&err, d, a, b, __VA_ARGS__); }
CALL(gemm, tsm100_gemm_desc, o, status, s)
CALL(attention, tsm100_attention_desc, v, o, status, s)
CALL(attention_prefill, tsm100_attention_prefill_desc, v, o, status, s)
CALL(attention_decode, tsm100_attention_decode_desc, v, o, s, status)
"""


@pytest.fixture(scope="module")
def without(tmp_path_factory, pkg):
    """The operators, built so that none of them gets scratch."""
    src = tmp_path_factory.mktemp("no_scratch") / "no_scratch.cu"
    src.write_text(NO_SCRATCH)
    out = src.with_suffix(".so")
    b = pkg.build
    subprocess.run([b.nvcc(), "-gencode", "arch=compute_100a,code=sm_100a", "-std=c++17", "-O3", "-split-compile=0", "--expt-relaxed-constexpr", "-w",
                    "-shared", "-Xcompiler", "-fPIC", f"-I{b.CSRC}", f"-I{b.INCLUDE}", "-cudart", "static", "-o", str(out), str(src)], check=True)
    return C.CDLL(str(out))


@pytest.mark.parametrize("name", NAMES)
def test_without_scratch(dev, pkg, without, name):
    """The form that needs none gives the same result up to the order of its sums (and, in 16 bits, one rounding)."""
    capi = pkg.capi
    op, desc, inputs, out = call = calls(capi)[name]
    run(capi, dev, call)
    torch.cuda.synchronize()
    want = out.clone()
    out.zero_()
    status = torch.zeros(1, dtype=torch.int32, device="cuda:0")
    p = [C.c_void_p(x.data_ptr()) for x in inputs] + [C.c_void_p(0)] * (3 - len(inputs))
    st = getattr(without, f"no_scratch_{op}")(C.byref(desc), *p, C.c_void_p(out.data_ptr()), C.c_void_p(status.data_ptr()), C.c_void_p(util.cur_stream(torch)))
    torch.cuda.synchronize()
    assert st == capi.OK and int(status[0]) == 0
    diff = float((out.double() - want.double()).norm() / want.double().norm())
    # f32: sums in another order (1e-5, the bound of the f32 operators); bf16: both round once to 8 bits, 2^-9 each
    assert 0 < diff <= (1e-5 if out.dtype == torch.float32 else 2.0 ** -8), diff
