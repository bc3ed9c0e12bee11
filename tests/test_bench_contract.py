"""The reference arm of bench.py runs on host cores only, so its JSON line can be checked here."""
import json
import os
import subprocess
import sys

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

BASE_KEYS = {"metric", "value", "unit", "n_gpus", "steps", "warmup", "ms_per_step", "higher_is_better", "scaling",
             "vs_baseline", "dtype", "data", "config", "e2e", "impl", "cpu_baseline"}


def _run(extra, env=None):
    cmd = [sys.executable, os.path.join(ROOT, "bench.py"), "--impl", "reference", "--steps", "2", "--warmup", "1",
           "--cpu-budget", "0.2"] + extra
    e = dict(os.environ)
    e.update(env or {})
    r = subprocess.run(cmd, cwd=ROOT, env=e, capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stderr[-2000:]
    return [l for l in r.stdout.splitlines() if l.startswith("{")]


def test_reference_arm_line():
    lines = _run([])
    assert len(lines) == 1
    d = json.loads(lines[0])
    assert BASE_KEYS <= set(d)
    assert d["impl"] == "reference" and d["unit"] == "TFLOP/s" and d["higher_is_better"] is True
    assert d["value"] > 0 and d["steps"] == 2 and d["n_gpus"] == 1
    assert d["e2e"] == {"value": d["value"], "unit": d["unit"], "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0}
    cb = d["cpu_baseline"]
    assert cb["kind"] in ("port", "reference") and cb["cores"] >= 1 and cb["value"] == d["value"] and cb["sample"]
    assert "workload" in d["config"] and "model" not in d["config"]


def test_reference_arm_other_ranks_stay_silent():
    assert _run([], env={"RANK": "1", "WORLD_SIZE": "2"}) == []


def test_reference_arm_names_the_same_workload_as_the_gpu_arm():
    sys.path.insert(0, ROOT)
    import bench
    d = json.loads(_run([])[0])
    assert d["config"]["workload"] == bench.LINEAR_NAME
    assert d["metric"] == "conv/linear fwd+bwd TFLOP/s"


def test_line_stays_short():
    """The line is read from the last 3000 characters of a log: with every block filled in, and numbers of full length, it has
    the contract's keys and fits; the per-layer table does not go into it."""
    sys.path.insert(0, ROOT)
    import bench
    v = 1234.567890123456
    clocks = {"sm_mhz": 1905.0, "sm_max_mhz": 1965.0, "reasons": ["hw_slowdown", "sw_power_cap"], "samples": 173, "source": "nvml"}
    roof = {"bound": "tensor", "achieved": v, "peak": v, "unit": "TFLOP/s", "frac": v, "peak_source": "measured burst bf16 (MEASURED_PEAKS.json)",
            "kernel": "umma_conv_kernel", "traffic": v, "algorithmic_bytes_per_launch": v, "clocks": clocks, "nominal_source": "x" * 80}
    work = {"value": v, "unit": "TFLOP/s", "ms_per_step": v, "contraction_tflops": v, "roofline": roof, "per_layer": [dict(roof)] * 48,
            "workload": bench.PIX2PIX_NAME, "clocks": clocks, "cpu_baseline": {"value": v}}
    e2e = {"value": v, "unit": "TFLOP/s", "h2d_bytes_per_step": 10 ** 9, "d2h_bytes_per_step": 10 ** 9,
           "returns": "dw, db of every layer (y and dx stay on the device, where the reference's host ops leave every result)"}
    record = {"metric": "conv/linear fwd+bwd TFLOP/s", "value": v, "unit": "TFLOP/s", "n_gpus": 8, "steps": 20, "warmup": 5, "ms_per_step": v,
              "higher_is_better": True, "scaling": "weak", "vs_baseline": None, "dtype": "f16 (fp32 accumulate)", "data": "synthetic",
              "impl": "nectarml_b200", "e2e": e2e, "e2e_all_results": e2e, "gpu_launches": 123456, "clocks": clocks, "roofline": roof,
              "per_layer": [dict(roof)] * 18, "comm_ms_exposed": v, "sustained": dict(work, frac_of_sustained_peak=v, seconds=v),
              "config": {"workload": bench.LINEAR_NAME, "layers": 6, "parallelism": "dp8 (rows / batch sharded, NCCL all-reduce of 3 flat dW/db "
                         "buckets, NCCL_MAX_CTAS=16, 16 SMs left to it while in flight)", "host_cpus_bound": 56,
                         "launch": "CUDA graph replay of the step's kernels, all-reduces issued between the graphs of the buckets",
                         "l2": "inputs and outputs of one step exceed the 126 MB L2 several times over",
                         "timing": "burst of `steps` steps from an idle GPU (0.5 s pause); `sustained`: the same step for >= 3.0 s"},
              "workloads": {k: work for k in ("resnet_conv", "pix2pix_conv", "config1_fp32_3xtf32", "resnet50_step", "pix2pix_step")},
              "cpu_baseline": {"value": v, "unit": "TFLOP/s", "cores": 16, "kind": "port", "sample": "x" * 100, "seconds": v}}
    line = bench.summary(record)
    assert len(json.dumps(line)) <= bench.LINE_LIMIT, len(json.dumps(line))
    assert (BASE_KEYS | {"gpu_launches", "clocks", "roofline"}) <= set(line) and "per_layer" not in line
    assert line["e2e"].keys() >= {"value", "unit", "h2d_bytes_per_step", "d2h_bytes_per_step"} and set(line["workloads"]) == set(record["workloads"])
