"""bench.py on a machine without GPUs: the reference arm prints one well-formed line for any configuration, both
arms describe a configuration with the same dictionary, and the GPU arm refuses to run without a device."""
import json
import os
import subprocess
import sys
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parent.parent


def _run(*args, env=None):
    e = dict(os.environ)
    e.update(env or {})
    return subprocess.run([sys.executable, str(ROOT / "bench.py"), *args], capture_output=True, text=True, env=e, timeout=600)


@pytest.mark.parametrize("workload", ["softmax_f32", "gemm_f32_512", "attention_causal"])
def test_reference_arm_line(workload):
    r = _run("--impl", "reference", "--workload", workload, "--steps", "1", "--warmup", "3", "--no-extras",
             env={"OMP_NUM_THREADS": "1"})  # what a launcher exports; the arm must undo it
    assert r.returncode == 0, r.stderr
    line = json.loads(r.stdout.strip().splitlines()[-1])
    for key in ("impl", "metric", "value", "unit", "n_gpus", "steps", "warmup", "ms_per_step", "higher_is_better", "scaling",
                "dtype", "data", "config", "cpu_baseline", "e2e"):
        assert key in line, key
    assert line["impl"] == "reference" and line["value"] > 0 and line["config"]["workload"] == workload
    assert line["cpu_baseline"]["kind"] == "port" and line["cpu_baseline"]["cores"] == len(os.sched_getaffinity(0))
    assert line["e2e"] == {"value": line["value"], "unit": line["unit"], "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0}


def test_other_ranks_of_the_reference_arm_do_nothing():
    r = _run("--impl", "reference", "--steps", "1", "--no-extras", env={"RANK": "1", "WORLD_SIZE": "2"})
    assert r.returncode == 0 and r.stdout.strip() == ""


def test_both_arms_describe_a_configuration_identically():
    sys.path.insert(0, str(ROOT))
    import bench
    for name in bench.ORDER:
        assert bench.config_for(name) == bench.config_for(name)
        assert set(bench.SUMMARY) <= set(bench.ORDER)
    assert bench.config_for("gemm_bf16_8192")["m"] == 8192 and "l2" in bench.config_for("softmax_f32")


def test_gpu_arm_needs_a_gpu():
    import torch
    if torch.cuda.is_available():
        pytest.skip("this check is for machines without a GPU")
    r = _run("--steps", "1", "--no-extras")
    assert r.returncode != 0 and "no CPU fallback" in (r.stderr + r.stdout)


class _Gemm:
    """Stands in for the device: products by numpy on host memory, f32 sums in one order for every size but `whole` rows."""
    def __init__(self, np, whole):
        self.np, self.whole = np, whole

    def gemm(self, code, m, n, k, a, b, c, stream=None):
        import ctypes
        view = lambda at, *shape: self.np.ctypeslib.as_array(ctypes.cast(at, ctypes.POINTER(ctypes.c_float)), shape)
        x, y = view(a, m, k), view(b, k, n)
        view(c, m, n)[:] = x @ y if m != self.whole else x[:, :k // 2] @ y[:k // 2] + x[:, k // 2:] @ y[k // 2:]


@pytest.mark.parametrize("m,spoil,ok", [(700, None, True), (700, (399, 2, 1e-6), False), (700, (1, 0, 1e-6), False), (700, (699, 7, 0.5), False), (128, None, False)])
def test_end_to_end_check_of_f32_products(m, spoil, ok):
    """Row blocks of 128, each compared bit for bit with a call of its size; a sum in another order over the whole only where there are several blocks."""
    sys.path.insert(0, str(ROOT))
    import types

    import bench
    import numpy as np
    import torch
    n, k = 8, 40960  # 100 rows of A are 16 MiB
    rng = np.random.default_rng(m)
    wl = object.__new__(bench.GemmWL)
    wl.units, wl.m, wl.n, wl.k, wl.es, wl.dtype, wl.code = 1, m, n, k, 4, "f32", 0
    a, b = (rng.uniform(-1, 1, shape).astype(np.float32) for shape in ((1, m, k), (1, k, n)))
    wl.a, wl.b, wl.c = torch.from_numpy(a), torch.from_numpy(b), torch.zeros(1, m, n)
    dev = _Gemm(np, whole=m)
    wl.ctx = types.SimpleNamespace(dev=dev, tdev="cpu", stream=0)
    dev.gemm(0, m, n, k, wl.a.data_ptr(), wl.b.data_ptr(), wl.c.data_ptr())
    host = np.empty((1, m, n), np.float32)
    assert [r for r, _ in wl._host_blocks()] == list(range(0, m, 128))
    for row in range(0, m, 128):
        rows = np.ascontiguousarray(a[0, row:row + 128])
        host[0, row:row + 128] = rows @ b[0]
    assert not np.array_equal(host, wl.c.numpy())
    if spoil:
        host[0, spoil[0], spoil[1]] += np.float32(spoil[2]) * max(1.0, abs(host[0, spoil[0], spoil[1]]))
    wl.c_host = types.SimpleNamespace(array=host)
    assert wl.e2e_check() == ok


def test_the_result_line_stays_short():
    """A line of 20 KB, with every workload's record in full, was not read whole; the records go to stderr."""
    sys.path.insert(0, str(ROOT))
    import types

    import bench
    roofline = {"bound": "tensor", "achieved": 1234.56, "peak": 1655.1, "unit": "TFLOP/s", "frac": 0.7459, "peak_source": "measured", "traffic": 1071900000.0}
    clocks = {"sm_mhz": 1965.0, "sm_max_mhz": 1965.0, "reasons": ["sw_power_cap"], "samples": 16, "source": "nvml"}
    rec = {"value": 1234.56, "unit": "TFLOP/s", "ms_per_step": 12.3456, "dtype": "bf16", "config": bench.config_for("attention_gqa_causal"), "roofline": roofline, "launches": 20,
           "clocks": clocks, "sustained": {"value": 1234.56, "roofline_frac": 0.9999, "tflops_per_ghz": 1044.4}, "verify": {"ok": True, "tolerance": "x" * 120},
           "cpu_baseline": {"value": 0.1234, "unit": "TFLOP/s", "cores": 16, "kind": "port", "sample": "x" * 120}, "context": {"torch_sdpa_tflops": 1231.2},
           "e2e": {"value": 185.08, "unit": "TFLOP/s", "h2d_bytes_per_step": 4294967296, "d2h_bytes_per_step": 2147483648, "api": "x" * 120},
           "strong": {"speedup_vs_one_gpu": 7.45}, "latency": {"host_us_per_call": 3.81, "device_us_per_call_back_to_back": 9.33}}
    args = types.SimpleNamespace(workload="softmax_f32", steps=20, warmup=5)
    extras = {n: rec for n in bench.ORDER if n != "softmax_f32"}
    extras["reduce_sum_f32"] = {"error": "x" * 600}
    line, detail = bench.result_line(args, 8, 16, rec, extras, ["reduce_sum_f32"])
    assert len(json.dumps(line)) <= 8192 and set(line["workloads"]) | set(line["summary"]) == set(extras)
    for key in ("metric", "value", "unit", "n_gpus", "steps", "warmup", "ms_per_step", "higher_is_better", "scaling", "vs_baseline", "dtype", "data", "config", "e2e", "gpu_launches", "clocks"):
        assert key in line, key
    assert detail["workloads"] == extras
