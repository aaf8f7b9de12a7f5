"""The benchmark's reference arm on the host cores, launched the way the N>1 runs are: rank 0
alone measures and prints one JSON line, the other ranks leave without work."""
import json
import re
import subprocess
import sys
from pathlib import Path

ROOT = Path(__file__).resolve().parents[1]


def test_reference_arm_under_two_ranks_prints_one_line():
    cmd = [sys.executable, "-m", "torch.distributed.run", "--nnodes=1", "--nproc-per-node", "2", "--master-addr", "127.0.0.1",
           "--master-port", "29573", str(ROOT / "bench.py"), "--impl", "reference", "--gpus", "2", "--steps", "1", "--warmup", "1"]
    out = subprocess.run(cmd, cwd=ROOT, capture_output=True, text=True, timeout=600)
    assert out.returncode == 0, out.stderr[-2000:]
    lines = [l for l in out.stdout.splitlines() if l.startswith("{")]
    assert len(lines) == 1, out.stdout
    d = json.loads(lines[0])
    assert d["impl"] == "reference" and d["n_gpus"] == 2 and d["steps"] == 1
    assert d["metric"] == "MoE-layer prefill tokens/sec at T=4096" and d["unit"] == "tokens/s" and d["higher_is_better"] is True
    assert d["value"] > 0 and d["ms_per_step"] > 0
    assert d["e2e"] == {"value": d["value"], "unit": "tokens/s", "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0}
    cb = d["cpu_baseline"]
    assert cb["kind"] in ("reference", "port") and cb["cores"] >= 1 and cb["value"] == d["value"] and cb["sample"]
    assert "workload" in d["config"] and "model" not in d["config"]


def test_launches_are_counted_by_the_kernels_of_each_size():
    """Routing takes two launches up to OMNI_ROUTE_MAX_ROWS tokens on one GPU and three above; longer batches run in arena pieces."""
    sys.path.insert(0, str(ROOT))
    import bench
    source = (ROOT / "cleffa_b200" / "csrc" / "omni_internal.h").read_text()
    assert bench.SHORT_TOKENS == int(re.search(r"OMNI_ROUTE_MAX_ROWS = (\d+)", source)[1])
    assert bench.ARENA_TOKENS == int(re.search(r"OMNI_CHUNK = (\d+)", source)[1])
    assert [bench.kernel_launches(T, 1, 1, False) for T in (1, 384, 385, 4096, 16384, 16385, 32768)] == [6, 6, 7, 7, 7, 12, 13]
    assert bench.kernel_launches(4096, 8, 1, False) == 10 and bench.kernel_launches(100, 8, 1, False) == 10
    assert bench.kernel_launches(4096, 1, 48, True) == 1 + 48 * 7
