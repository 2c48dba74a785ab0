"""The reference arm of bench.py runs without a GPU (it times the CPU oracle port), so its JSON line is checked
here: one line, the keys the benchmark contract names, the reference-arm conventions."""
import json
import os
import subprocess
import sys

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_scan_kernel_is_named_by_the_library():
    """The stand-alone scan of 16 x 4096 x 1536 has 5 warps of chains per SM: one pass, one launch, also in segments; a shard of
    an eighth of it looks back."""
    import torch
    sys.path.insert(0, ROOT)
    import bench
    from helixml_b200 import ops
    cfg = {"batch": 16, "seq_len": 4096, "d_inner": 1536}
    splits = ops.suggest_splits(16, 4096, 1536, torch.bfloat16)
    assert splits > 1 and bench.scan_kernel_name("auto", cfg, splits) == "scan_direct_kernel"
    assert bench.scan_kernel_name("auto", cfg, 1) == "scan_direct_kernel"
    assert "look-back" in bench.scan_kernel_name("auto", dict(cfg, batch=2), ops.suggest_splits(2, 4096, 1536, torch.bfloat16))
    assert bench.scan_kernel_name("tiled", cfg) == "scan_tiled_kernel" and "look-back" in bench.scan_kernel_name("lookback", cfg, 8)


def test_reference_arm_prints_one_contract_line():
    out = subprocess.run([sys.executable, os.path.join(ROOT, "bench.py"), "--impl", "reference", "--steps", "1", "--warmup", "0"],
                         cwd=ROOT, capture_output=True, text=True, timeout=600)
    assert out.returncode == 0, out.stderr[-2000:]
    lines = [l for l in out.stdout.strip().splitlines() if l.startswith("{")]
    assert len(lines) == 1
    j = json.loads(lines[0])
    for key in ("metric", "value", "unit", "n_gpus", "steps", "warmup", "higher_is_better", "scaling", "vs_baseline", "dtype",
                "data", "config", "cpu_baseline", "e2e", "impl"):
        assert key in j, key
    assert j["impl"] == "reference" and j["unit"] == "tokens/s" and j["higher_is_better"] is True
    assert j["value"] > 0 and j["vs_baseline"] is None and j["data"] == "synthetic"
    assert j["config"]["workload"] == "lm_cfg3" and "model" not in j["config"]
    assert j["cpu_baseline"]["kind"] == "port" and j["cpu_baseline"]["cores"] >= 1 and j["cpu_baseline"]["value"] == j["value"]
    assert j["e2e"] == {"value": j["value"], "unit": "tokens/s", "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0}
