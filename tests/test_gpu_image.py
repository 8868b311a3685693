"""The whole-image kernels (image forward and adjoint, image spectral
NCC) against the float64 oracle at the sizes where they can go wrong: odd and
even lengths (self-conjugate rows and columns), lengths below a warp, with
prime factors above the register butterflies (7, 29, 47) and a single prime,
the largest length that fits, non-square image pairs, one and several targets,
no high-pass, and the first size that takes the separate passes.

Tolerances: line transforms of at most 8 passes in float32 on values of one
magnitude, 1e-6 relative L2 of an image; a pose gradient sums products with
spatial derivatives, 2e-5; the NCC gradient cancels against its own
projection, 2e-5; the loss is reduced in float64, 1e-6."""
import numpy as np
import pytest
import torch

from conftest import rel_l2
from oracle import torch_convention as tc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("R,whole", [(5, 1), (14, 1), (29, 1), (47, 1), (58, 1), (96, 1), (99, 1), (128, 1), (144, 1),
                                     (160, 0)])
def test_image_and_pose_gradient_vs_oracle(R, whole):
    import fvr
    import fvr._lib as L

    vol = tc.make_ellipsoid_volume(40, 3)
    eng = fvr.TorchDiffFVREngine(torch.from_numpy(vol), spacing=(0.8, 0.8, 1.2))
    assert L.query("fvr_image_supported", R, R) == whole
    poses = tc.make_poses(3, 4)
    spec = tc.spectrum(vol)
    w = np.random.default_rng(R).standard_normal((3, 1, R, R))
    for view in ("ap", "lateral"):
        p = torch.from_numpy(poses).cuda().requires_grad_(True)
        img = eng(p, view=view, out_res=R)
        (g,) = torch.autograd.grad(img, p, torch.from_numpy(w.astype(np.float32)).cuda())
        ref = tc.forward_image(spec, poses, view, R, 0.8)
        assert rel_l2(img.detach().cpu().numpy(), ref) < 1e-5  # the float32 spectrum's own rounding included
        gref = tc.forward_image_grad(spec, poses, w.astype(np.float32), view, R, 0.8)
        assert rel_l2(g.cpu().numpy(), gref) < 1e-4


@pytest.mark.parametrize("B,Bt,H,W,hp", [(1, 1, 2, 3, False), (3, 1, 9, 14, True), (2, 2, 29, 16, True),
                                         (2, 1, 58, 47, True), (3, 3, 96, 96, True), (2, 1, 120, 130, False),
                                         (2, 1, 144, 144, True), (2, 2, 200, 150, True)])
def test_image_spectral_ncc_vs_oracle(B, Bt, H, W, hp):
    import fvr

    rng = np.random.default_rng(H * 100 + W)
    y, x = np.linspace(0, 3, H)[:, None], np.linspace(0, 4, W)[None]

    def image(n):
        ph = rng.random((n, 1, 1, 1))
        return (2.0 + np.sin(2 * y + 6 * ph) * np.cos(3 * x - 4 * ph) + 0.2 * rng.standard_normal((n, 1, H, W))).astype(
            np.float32)

    pred, targ = image(B), image(Bt)
    eng = fvr.TorchDiffFVREngine(torch.zeros((8, 8, 8)) + 1.0)
    t = torch.from_numpy(pred).cuda().requires_grad_(True)
    loss = eng.spectral_ncc_loss(t, torch.from_numpy(targ).cuda(), high_pass=hp)
    (g,) = torch.autograd.grad(2.5 * loss, t)
    with torch.no_grad():
        again = eng.spectral_ncc_loss(t, torch.from_numpy(targ).cuda(), high_pass=hp)
    p64, t64 = pred.astype(np.float64), targ.astype(np.float64)
    assert abs(float(loss) - tc.spectral_ncc_loss_images(p64, t64, hp)) < 1e-6
    assert abs(float(again) - float(loss)) < 1e-7
    ref = tc.spectral_ncc_loss_images_grad(p64, t64, hp, g=2.5)
    assert g.shape == t.shape
    assert rel_l2(g.cpu().numpy(), ref) < 2e-5


def test_image_spectral_ncc_of_unlike_magnitudes():
    """The pair shares one complex transform: an image of zeros (ncc 0, loss 1),
    and images 1e-6 and 1e5 times the target keep their own accuracy (loss and
    relative gradient as at equal magnitude)."""
    import fvr

    rng = np.random.default_rng(0)
    base = (1.0 + rng.random((1, 1, 48, 40))).astype(np.float32)
    targ = (base + 0.3 * rng.random(base.shape)).astype(np.float32)
    pred = np.concatenate([0.0 * base, np.float32(1e-6) * base, np.float32(1e5) * base])
    eng = fvr.TorchDiffFVREngine(torch.zeros((8, 8, 8)) + 1.0)
    for i in range(3):
        t = torch.from_numpy(pred[i:i + 1]).cuda().requires_grad_(True)
        loss = eng.spectral_ncc_loss(t, torch.from_numpy(targ).cuda())
        (g,) = torch.autograd.grad(loss, t)
        p64, t64 = pred[i:i + 1].astype(np.float64), targ.astype(np.float64)
        assert abs(float(loss) - tc.spectral_ncc_loss_images(p64, t64)) < 1e-6
        if i:
            assert rel_l2(g.cpu().numpy(), tc.spectral_ncc_loss_images_grad(p64, t64)) < 2e-5


@pytest.mark.parametrize("R", [6, 29, 64, 99, 128])
def test_two_ctas_an_image_equal_one(R):
    """Few images take two CTAs each, more than half the SMs' number one: the
    line transforms are the same arithmetic either way, so images agree bit for
    bit; the sums of the NCC and of the pose gradient are float64 sums of the
    same float32 products in another order, 1e-6."""
    import fvr

    n = torch.cuda.get_device_properties(0).multi_processor_count // 2 + 3
    eng = fvr.TorchDiffFVREngine(torch.from_numpy(tc.make_ellipsoid_volume(24, 3)), spacing=(0.8, 0.8, 1.2))
    poses = torch.from_numpy(tc.make_poses(n, 4)).cuda()
    targ = eng(poses[:1] + 0.01, view="ap", out_res=R).detach()

    def run(p):
        p = p.clone().requires_grad_(True)
        img = eng(p, view="ap", out_res=R)
        loss = eng.spectral_ncc_loss(img, targ)
        (g,) = torch.autograd.grad(loss * p.shape[0], p)
        return img.detach(), g

    img, g = run(poses)
    for lo, hi in ((0, 1), (n // 2, n // 2 + 3)):
        few, gf = run(poses[lo:hi])
        assert torch.equal(few, img[lo:hi])
        assert rel_l2(g[lo:hi].cpu().numpy(), gf.cpu().numpy()) < 1e-5
