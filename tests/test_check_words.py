"""The bounds-checked debug build reads the check word of every unit that has
checked accesses, the whole-image kernels' among them, and those kernels stay
in bounds at minimum, odd and largest sizes."""
import json
import os
import re
import subprocess
import sys
from pathlib import Path

import numpy as np
import pytest

REPO = Path(__file__).resolve().parents[1]
CSRC = REPO / "diff-fvr_b200" / "csrc"
LIBDIR = REPO / "diff-fvr_b200" / "fvr"
# guards and the samplers of the headers that hold them
CHECKED = re.compile(r"\b(fvr_checked|ldg_in|atomic_add_in|slice_sample|stencil_sample\w*|pair_load|tab_load\w*)\b")


def test_every_unit_with_checked_accesses_has_its_word_read():
    api = (CSRC / "fvr_api.cu").read_text()
    units = [f for f in CSRC.glob("*.cu") if CHECKED.search(re.sub(r"//.*", "", f.read_text()))]
    assert {"fvr_tc.cu", "fvr_image.cu", "fvr_pou.cu", "fvr_pou_sep.cu"} <= {f.name for f in units}
    for f in units:
        names = re.findall(r"^FVR_CHECK_ACCESSOR\((\w+)\)", f.read_text(), re.M)
        assert len(names) == 1, f.name
        assert len(re.findall(rf"\b{names[0]}\b", api)) >= 2, f.name  # declared and read


CHILD = """
import ctypes, json, sys
sys.path.insert(0, {pkg!r})
import torch, fvr
from fvr import _lib as L
from fvr.synthetic import make_ellipsoid_volume, make_poses
out = {{}}
poses = torch.from_numpy(make_poses(3, 2)).cuda()
for dt in (torch.float32, torch.bfloat16, torch.float16):
    eng = fvr.TorchDiffFVREngine(torch.from_numpy(make_ellipsoid_volume(24, 1)))
    if dt != torch.float32:
        eng.to_precision(dt)
    for R in (2, 3, 20, 23, 97, 144):
        for view in ("ap", "lateral"):
            p = poses.clone().requires_grad_(True)
            img = eng(p, view=view, out_res=R)
            loss = eng.spectral_ncc_loss(img, img.detach()[:1] + torch.linspace(0, 1, R, device="cuda"))
            loss.backward()
            out[f"{{dt}}_{{R}}_{{view}}"] = [float(loss.detach())] + p.grad.flatten().tolist() + img.flatten().tolist()[::37]
g = torch.Generator(device="cuda").manual_seed(1)
for H, W in ((2, 2), (5, 60), (61, 4), (100, 99)):
    x = torch.rand((2, 1, H, W), generator=g, device="cuda").requires_grad_(True)
    loss = eng.spectral_ncc_loss(x, torch.rand((2, 1, H, W), generator=g, device="cuda"))
    loss.backward()
    out[f"ncc_{{H}}_{{W}}"] = [float(loss.detach())] + x.grad.flatten().tolist()[::11]
torch.cuda.synchronize()
words = (ctypes.c_ulonglong * 4)()
out["check"] = [L.load().fvr_check_words(words, 4, 1)] + [int(w) for w in words]
print(json.dumps(out))
"""


def _run(lib):
    r = subprocess.run([sys.executable, "-c", CHILD.format(pkg=str(REPO / "diff-fvr_b200"))], capture_output=True,
                       text=True, timeout=600, env=dict(os.environ, FVR_B200_LIB=str(lib)))
    assert r.returncode == 0, r.stderr[-2000:]
    return json.loads(r.stdout.strip().splitlines()[-1])


@pytest.mark.gpu
def test_image_kernels_stay_in_bounds():
    chk = LIBDIR / "libfvr_b200_check.so"
    if not chk.exists():
        subprocess.run(["make", "-C", str(CSRC), "-j8", "check"], check=True)
    normal, checked = _run(LIBDIR / "libfvr_b200.so"), _run(chk)
    assert checked.pop("check") == [0, 0, 0, 0, 0]
    normal.pop("check")
    assert len(normal) == 40
    for k, v in normal.items():
        a, b = np.asarray(v, np.float64), np.asarray(checked[k], np.float64)
        assert np.linalg.norm(a - b) <= 5e-6 * max(np.linalg.norm(a), 1e-30), k
