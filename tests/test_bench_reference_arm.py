"""bench.py --impl reference where the reference is not built: one JSON line
that says so, exit status 0."""
import json
import os
import subprocess
import sys
from pathlib import Path

import pytest

from oracle.oracle import reference_binary

ROOT = Path(__file__).resolve().parents[1]


def test_reference_arm_without_the_reference():
    if reference_binary("cpu", "symmetric").exists():
        pytest.skip("the reference is built here")
    env = {k: v for k, v in os.environ.items() if k not in ("RANK", "WORLD_SIZE", "LOCAL_RANK")}
    r = subprocess.run([sys.executable, "bench.py", "--impl", "reference", "--steps", "2", "--warmup", "1"], cwd=ROOT,
                       env=env, capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stderr[-2000:]
    line = json.loads(r.stdout.strip())
    assert line["impl"] == "reference" and "ref_cpu_symmetric" in line["unavailable"]
