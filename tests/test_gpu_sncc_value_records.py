"""The value-only spectral NCC where its finalize takes an item's records by ten
lanes a moment (24 records and more) and where one lane takes them: the float64
oracle's loss, 1e-5 as at ordinary sizes."""
import pytest
import torch

from oracle import torch_convention as tc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("C,R", [(1, 8), (1, 97), (2, 200), (9, 96), (40, 33)])
def test_value(C, R):
    import fvr

    vol = tc.make_ellipsoid_volume(24, 11)
    eng = fvr.TorchDiffFVREngine(torch.from_numpy(vol), spacing=(1.0, 1.0, 1.0))
    spec, poses = tc.spectrum(vol, 2.0), tc.make_poses(C, 12)
    ft = tc.prepare_spectral_target(tc.forward_image(spec, tc.make_poses(1, 13), "lateral", R))
    with torch.no_grad():
        loss = eng.forward_spectral_ncc(torch.from_numpy(poses).cuda(), torch.from_numpy(ft).to(torch.complex64).cuda(),
                                        view="lateral")
    assert abs(float(loss) - tc.spectral_ncc(spec, poses, ft, "lateral")[0]) < 1e-5
