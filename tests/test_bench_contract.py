"""The JSON line of bench.py (reference arm: it needs no GPU) carries the keys its consumers read."""
import json
import os
import subprocess
import sys

from conftest import ROOT


def test_reference_arm_prints_one_json_line_with_the_contract_keys():
    out = subprocess.run([sys.executable, os.path.join(ROOT, "bench.py"), "--impl", "reference", "--workload", "cfg2-small",
                          "--steps", "2", "--warmup", "1"], capture_output=True, text=True, timeout=600,
                         env={**os.environ, "CUDA_VISIBLE_DEVICES": ""})
    assert out.returncode == 0, out.stderr[-2000:]
    lines = [l for l in out.stdout.splitlines() if l.startswith("{")]
    assert len(lines) == 1
    j = json.loads(lines[0])
    for key in ("impl", "metric", "value", "unit", "n_gpus", "steps", "warmup", "ms_per_step", "higher_is_better",
                "scaling", "vs_baseline", "dtype", "data", "config", "cpu_baseline", "e2e"):
        assert key in j, key
    assert j["impl"] == "reference" and j["metric"] == "spmm_gflops" and j["unit"] == "GFLOP/s" and j["value"] > 0
    assert j["cpu_baseline"]["kind"] == "port" and j["cpu_baseline"]["cores"] >= 1 and j["cpu_baseline"]["sample"]
    assert j["e2e"]["h2d_bytes_per_step"] == 0 and j["e2e"]["d2h_bytes_per_step"] == 0
    assert "workload" in j["config"] and j["steps"] == 2 and j["warmup"] == 1


def test_other_ranks_of_the_reference_arm_exit_quietly():
    out = subprocess.run([sys.executable, os.path.join(ROOT, "bench.py"), "--impl", "reference", "--workload", "cfg2-small",
                          "--gpus", "2"], capture_output=True, text=True, timeout=120,
                         env={**os.environ, "RANK": "1", "WORLD_SIZE": "2", "LOCAL_RANK": "1", "CUDA_VISIBLE_DEVICES": ""})
    assert out.returncode == 0 and out.stdout.strip() == ""


def test_roofline_of_the_transforms():
    sys.path.insert(0, ROOT)
    import bench
    rows = 1_000_000
    apart, paired = (bench.transform_roofline(p, 0.25, rows, 6000.0) for p in (False, True))
    assert apart["kernel"] == "gemm_tf32_128_kernel" and paired["kernel"] == "gemm_tf32_pair_kernel"
    assert apart["algorithmic_bytes_per_launch"] == 1024 * rows + 65536 and paired["algorithmic_bytes_per_launch"] == 1024 * rows + 131072
    assert abs(apart["achieved"] - (1024 * rows + 65536) / 0.25e6) < 1e-6 and abs(paired["achieved"] - (1024 * rows + 131072) / 0.5e6) < 1e-6
