"""Without the reference in baseline/_ref, bench.py's reference arm says so in
one line and exits 0: no number of another implementation stands in its place."""
import json
import os
import subprocess
import sys
from pathlib import Path

import pytest

REPO = Path(__file__).resolve().parents[1]


def test_reference_arm_without_the_reference():
    if (REPO / "baseline" / "_ref").exists():
        pytest.skip("the reference is installed")
    env = {k: v for k, v in os.environ.items() if k not in ("WORLD_SIZE", "RANK", "LOCAL_RANK")}
    r = subprocess.run([sys.executable, str(REPO / "bench.py"), "--impl", "reference", "--steps", "1", "--warmup", "1"],
                       cwd=REPO, env=env, capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stderr[-2000:]
    line = json.loads(r.stdout)
    assert line["impl"] == "reference" and "value" not in line and "\n" not in line["unavailable"]
