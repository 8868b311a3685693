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


def test_records_follow_a_changed_geometry(monkeypatch):
    """Block spacing of a renderer, voxel spacing of an engine: the prepared
    records give what the Python nodes, which keep none, give."""
    import fvr
    import fvr._native as NA
    import fvr.torch_engine as te
    from fvr import synthetic
    from fvr.cone_beam_fvr import PerspectiveSlabFVR

    m = PerspectiveSlabFVR.from_volume(synthetic.make_ellipsoid_volume(40, 2), vox_mm=2.0, grid_blocks=(2, 2, 2),
                                       block_res=32, overlap=0.5)
    k_inv = torch.tensor([[1 / 500.0, 0, -0.05], [0, 1 / 500.0, -0.04], [0, 0, 1.0]], device="cuda")
    lat = m.make_pinhole_lattice(k_inv, 1020.0, 41, 50)
    mats = synthetic.make_pinhole_mats(3, 5, device="cuda")
    eng = fvr.TorchDiffFVREngine(torch.from_numpy(synthetic.make_ellipsoid_volume(24, 2)))
    poses = torch.from_numpy(synthetic.make_poses(3, 4)).cuda().requires_grad_(True)
    f = eng.prepare_spectral_target(eng(poses.detach()[:1], out_res=28))
    m.forward_pinhole(mats, lat)
    first = float(eng.forward_spectral_ncc(poses, f))
    m.ds_block *= 1.1
    eng.spacing = tuple(1.5 * s for s in eng.spacing)
    got = m.forward_pinhole(mats, lat), eng.forward_spectral_ncc(poses, f)
    monkeypatch.setattr(NA, "_MOD", None)
    monkeypatch.setattr(te, "_NATIVE", None)
    eng._fused_calls.clear()
    assert torch.equal(got[0], m.forward_pinhole(mats, lat))
    want = float(eng.forward_spectral_ncc(poses, f))
    assert float(got[1]) == want and want != first
