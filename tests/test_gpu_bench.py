"""bench.py runs through, its end-to-end check included, and prints its one line."""
import json
import subprocess
import sys
from pathlib import Path

import pytest

pytestmark = pytest.mark.gpu
ROOT = Path(__file__).resolve().parent.parent


def test_bench_line_has_an_end_to_end_value():
    run = subprocess.run([sys.executable, "bench.py", "--gpus", "1", "--steps", "3", "--warmup", "3", "--no-extra"], cwd=ROOT,
                         capture_output=True, text=True, timeout=300)
    assert run.returncode == 0, run.stderr[-2000:]
    line = json.loads(run.stdout.strip().splitlines()[-1])
    assert line["metric"] == "causal_rope_fwd_tflops" and line["n_gpus"] == 1 and line["gpu_launches"] > 0
    assert 0 < line["e2e"]["value"] < line["value"]
