"""A status of the library in a native node becomes an exception with its text
(in a child process: with a second libstdc++ in the binding, writing the
status's number ended the process)."""
import subprocess
import sys
from pathlib import Path

import pytest

pytestmark = pytest.mark.gpu

CHILD = """
import sys; sys.path.insert(0, {pkg!r})
import torch
import fvr._lib as L
from fvr.registration import biplanar_loss_per_candidate
x = torch.rand((1, 1, 20, 400), device="cuda")  # the crop leaves no row
try:
    biplanar_loss_per_candidate(x, x, x, x)
except L.FvrError as e:
    print(e)
"""


def test_status_in_a_native_forward_is_an_error_not_a_crash():
    pkg = str(Path(__file__).resolve().parents[1] / "diff-fvr_b200")
    r = subprocess.run([sys.executable, "-c", CHILD.format(pkg=pkg)], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
    assert "failed with status 1" in r.stdout
