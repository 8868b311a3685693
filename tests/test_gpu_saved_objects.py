"""Engines and models saved by an earlier version of the package, which lack the
records that the native binding's calls keep, still render."""
import copy

import pytest
import torch

pytestmark = pytest.mark.gpu


def test_engine_without_image_records():
    import fvr
    from fvr import synthetic

    eng = fvr.TorchDiffFVREngine(torch.from_numpy(synthetic.make_ellipsoid_volume(24, 2)))
    poses = torch.from_numpy(synthetic.make_poses(3, 4)).cuda()
    want = eng(poses, out_res=28)
    old = copy.deepcopy(eng)
    del old.__dict__["_image_plans"]
    assert torch.equal(copy.deepcopy(old)(poses, out_res=28), want)
    assert torch.equal(old(poses, out_res=28), want)
