"""The spectral-NCC epilogue where several threads share an item's records (up
to 15 items of many row tiles) and at the counts around it, one and two views:
loss and pose gradient against the float64 oracle.  Tolerances of the same call
at ordinary sizes: 1e-5 of the loss, 1e-4 of the gradient."""
import numpy as np
import pytest
import torch

from conftest import rel_l2
from oracle import torch_convention as tc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("C,R,views", [(1, 5, 1), (1, 97, 2), (3, 200, 1), (7, 64, 2), (8, 64, 2), (15, 33, 1),
                                       (16, 33, 1), (31, 40, 1)])
def test_loss_and_gradient(C, R, views):
    import fvr

    vol = tc.make_ellipsoid_volume(24, 11)
    eng = fvr.TorchDiffFVREngine(torch.from_numpy(vol), spacing=(1.0, 1.0, 1.0))
    spec, poses = tc.spectrum(vol, 2.0), tc.make_poses(C, 12)
    names = ("ap", "lateral")[:views]
    fts = [tc.prepare_spectral_target(tc.forward_image(spec, tc.make_poses(1, 13), v, R)) for v in names]
    dev = [torch.from_numpy(f).to(torch.complex64).cuda() for f in fts]
    loss, grad = eng.spectral_ncc_value_and_grad(torch.from_numpy(poses).cuda(), dev, views=names)
    want = sum(tc.spectral_ncc(spec, poses, f, v)[0] for f, v in zip(fts, names))
    gwant = sum(tc.spectral_ncc_grad(spec, poses, f, v) for f, v in zip(fts, names))
    assert abs(float(loss) - want) < 1e-5
    assert rel_l2(grad.cpu().numpy(), np.asarray(gwant)) < 1e-4
