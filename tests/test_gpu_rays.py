"""project_rays_batched with the detector axes taken from the lattice (one
library call per direction) against the same renderer given axes formed by
tensor operations (_extract_detector_basis, differentiated by autograd): images
and gradients to sources and detector points.  Lattices of 2 x 2 points, odd
sizes, one above the 2048-point tiles of the centroid sum, and a mirrored one
(v x u points back to the source, so n is turned).

Both sides form the axes of the same float32 points, one in float64 and one in
float32: a relative 2e-7 of the axes moves a sampling position (at most 100
image pixels from the centre) by 2e-5 pixels, hence 1e-4 for images of white
edges and their gradients, 1e-3 for the gradient's corner points, which add the
axes' share of every pixel."""
import pytest
import torch

from conftest import rel_l2

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,H,W,mirror,block_res", [(1, 2, 2, False, 32), (3, 33, 17, False, 32), (2, 40, 60, True, 48),
                                                    (2, 70, 65, False, 32), (2, 24, 20, False, 25)])
def test_lattice_axes_match_given_axes(N, H, W, mirror, block_res):
    from fvr import synthetic
    from fvr.cone_beam_fvr import PerspectiveSlabFVR

    m = PerspectiveSlabFVR.from_volume(synthetic.make_ellipsoid_volume(48, 2), vox_mm=2.0, grid_blocks=(2, 2, 2),
                                       block_res=block_res, overlap=0.5)
    mats = synthetic.make_pinhole_mats(N, 5, sad_mm=400.0, device="cuda")
    pix = 160.0 / max(H, W)
    x = (torch.arange(W, device="cuda") - 0.5 * (W - 1)) * pix
    y = (torch.arange(H, device="cuda") - 0.5 * (H - 1)) * pix
    if mirror:
        x = -x
    cam = torch.stack([x[None, :].expand(H, W), y[:, None].expand(H, W), torch.full((H, W), 600.0, device="cuda")], -1)
    trg = torch.einsum("nij,hwj->nhwi", mats[:, :3, :3], cam) + mats[:, None, None, :3, 3]
    g = torch.randn((N, H, W), generator=torch.Generator(device="cuda").manual_seed(1), device="cuda")
    res = []
    for given in (False, True):
        s, t = mats[:, :3, 3].clone().requires_grad_(True), trg.clone().requires_grad_(True)
        axes = m._extract_detector_basis(s, t) if given else (None, None, None)
        out = m.project_rays_batched(s, t, *axes)
        res.append((out.detach(), *torch.autograd.grad(out, (s, t), g)))
    for a, b, tol in zip(res[0], res[1], (1e-4, 1e-3, 1e-3)):
        assert a.shape == b.shape and a.dtype == b.dtype
        assert float(b.abs().sum()) > 0
        assert rel_l2(a.cpu().numpy(), b.cpu().numpy()) < tol
