"""The separable pinhole warp and its adjoint (fvr_pou_warp_sep,
fvr_pou_warp_sep_adjoint) against the float64 oracle, at the sizes where the
marching kernels can go wrong: one detector pixel, detectors around multiples
of the 32 columns of a warp and the 4 / 16 rows of a band, image sizes that are
no multiple of the 8-row bands or 32-column groups, less than one and more than
128 detector columns per group of image columns, tables that run backwards,
images that the detector only grazes, and enough poses for the wide forms.

Tolerances: sums of f32 products over at most a few hundred detector pixels
per image pixel, so 2e-6 relative L2 forward and 1e-5 for the gradients."""
import numpy as np
import pytest
import torch

from conftest import rel_l2
from oracle import pou as opou

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,N,P,H,W,pitch,flip,shift", [
    (1, 1, 16, 1, 1, 1.0, 0, 0.0), (2, 2, 30, 31, 33, 0.7, 0, 0.3), (3, 1, 64, 16, 32, 2.3, 0, 0.0),
    (2, 3, 64, 65, 64, 0.9, 1, 0.0), (17, 1, 40, 40, 300, 0.2, 0, 0.0), (2, 1, 64, 300, 47, 0.25, 2, 5.0),
    (2, 2, 96, 37, 129, 0.8, 3, -70.0), (1, 2, 33, 20, 270, 0.02, 0, 0.0), (2, 2, 160, 211, 247, 0.6, 0, 0.0),
    (2, 300, 32, 33, 65, 0.6, 1, 0.0), (34, 100, 20, 18, 70, 0.5, 0, 0.0), (2, 130, 32, 121, 130, 0.3, 2, 0.0),
    (1, 60, 48, 130, 40, 0.28, 0, 0.0),
])
def test_separable_warp_and_adjoint_vs_oracle(B, N, P, H, W, pitch, flip, shift):
    import fvr._lib as L

    rng = np.random.default_rng(P * 1000 + H + W)
    ds, c = 1.5, float(P // 2)
    db = 700.0 + rng.uniform(-60, 60, (B, N))
    cu, cv = rng.uniform(-4, 4, (B, N)) - shift * ds, rng.uniform(-4, 4, (B, N)) + 0.5 * shift * ds
    rxc = ((np.arange(W) - 0.5 * W + 0.37) * pitch * ds / 700.0).astype(np.float32)
    ryr = ((np.arange(H) - 0.5 * H + 0.41) * pitch * ds / 700.0).astype(np.float32)
    if flip & 1:
        rxc = rxc[::-1].copy()
    if flip & 2:
        ryr = ryr[::-1].copy()
    imgs = rng.standard_normal((B, N, P, P)).astype(np.float32)
    ic = (1.0 + 0.1 * rng.random((H, W))).astype(np.float32)
    g = rng.standard_normal((N, H, W)).astype(np.float32)
    rx, ry = np.broadcast_to(rxc[None, :], (H, W)), np.broadcast_to(ryr[:, None], (H, W))
    ref = opou.warp_sum(imgs.astype(np.float64), db, cu, cv, rx.astype(np.float64), ry.astype(np.float64),
                        ic.astype(np.float64), 1.0 / ds, c)
    gi, gd, gu, gv = opou.warp_sum_adjoint(imgs.astype(np.float64), db, cu, cv, rx.astype(np.float64),
                                           ry.astype(np.float64), ic.astype(np.float64), 1.0 / ds, c,
                                           g.astype(np.float64))
    dev = torch.device("cuda", 0)
    t = {k: torch.from_numpy(np.ascontiguousarray(v)).to(dev) for k, v in
         dict(imgs=imgs, offs=np.stack([db, cu, cv], -1), rxc=rxc, ryr=ryr, ic=ic, g=g).items()}
    out = torch.full((N, H, W), float("nan"), device=dev)
    gim = torch.full((B, N, P, P), float("nan"), device=dev)
    goffs = torch.full((3, B, N), float("nan"), dtype=torch.float64, device=dev)
    head = (L.ptr(t["imgs"]), B, N, P, L.ptr(t["offs"]), L.ptr(t["rxc"]), L.ptr(t["ryr"]), L.ptr(t["ic"]), H, W,
            1.0 / ds, c)
    L.call("fvr_pou_warp_sep", *head, L.ptr(out), L.stream_ptr(dev))
    assert L.query("fvr_pou_warp_sep_adjoint_supported", P, H, W) == 1
    ws = torch.empty(L.query("fvr_pou_warp_sep_adjoint_workspace", N, H, W), dtype=torch.uint8, device=dev)
    L.call("fvr_pou_warp_sep_adjoint", *head, L.ptr(t["g"]), L.ptr(ws), ws.numel(), L.ptr(gim), L.ptr(goffs),
           L.stream_ptr(dev))
    assert np.linalg.norm(ref) > 0
    assert rel_l2(out.cpu().numpy(), ref) < 2e-6
    assert rel_l2(gim.cpu().numpy(), gi) < 1e-5
    for got, want in zip(goffs.cpu().numpy(), (gd, gu, gv)):
        assert rel_l2(got, want) < 1e-5


@pytest.mark.parametrize("B,N,P,H,W", [(3, 40, 40, 45, 140), (1, 75, 33, 37, 60), (9, 21, 64, 67, 300),
                                       (2, 186, 32, 13, 33)])
def test_separable_warp_of_four_rows_vs_oracle(B, N, P, H, W):
    """Detectors and pose counts that leave 5 to 8 warps an SM: four rows per
    CTA, row counts that are no multiple of four.  Tolerance as above."""
    import fvr._lib as L

    rng = np.random.default_rng(P + H + W)
    ds, c = 1.5, float(P // 2)
    db, cu, cv = (m + rng.uniform(-s, s, (B, N)) for m, s in ((700.0, 60), (0.0, 4), (0.0, 4)))
    rxc = ((np.arange(W) - 0.5 * W + 0.37) * 0.6 * ds / 700.0).astype(np.float32)
    ryr = ((np.arange(H) - 0.5 * H + 0.41) * 0.6 * ds / 700.0).astype(np.float32)
    imgs = rng.standard_normal((B, N, P, P)).astype(np.float32)
    ic = (1.0 + 0.1 * rng.random((H, W))).astype(np.float32)
    rx, ry = np.broadcast_to(rxc[None, :], (H, W)), np.broadcast_to(ryr[:, None], (H, W))
    ref = opou.warp_sum(imgs.astype(np.float64), db, cu, cv, rx.astype(np.float64), ry.astype(np.float64),
                        ic.astype(np.float64), 1.0 / ds, c)
    dev = torch.device("cuda", 0)
    t = {k: torch.from_numpy(np.ascontiguousarray(v)).to(dev) for k, v in
         dict(imgs=imgs, offs=np.stack([db, cu, cv], -1), rxc=rxc, ryr=ryr, ic=ic).items()}
    out = torch.full((N, H, W), float("nan"), device=dev)
    L.call("fvr_pou_warp_sep", L.ptr(t["imgs"]), B, N, P, L.ptr(t["offs"]), L.ptr(t["rxc"]), L.ptr(t["ryr"]),
           L.ptr(t["ic"]), H, W, 1.0 / ds, c, L.ptr(out), L.stream_ptr(dev))
    assert rel_l2(out.cpu().numpy(), ref) < 2e-6


@pytest.mark.parametrize("db0,H,W,P,pitch", [
    (0.0, 33, 70, 40, 1.0), (0.9, 40, 65, 64, 1.0), (2.5, 31, 130, 64, 1.0), (-650.0, 70, 300, 96, 0.5),
    (-2.0, 20, 33, 33, 1.0), (650.0, 9, 140, 129, 0.7), (700.0, 140, 600, 64, 0.25),
])
def test_separable_adjoint_moments_vs_oracle(db0, H, W, P, pitch):
    """The adjoint's cell moments where their reference points matter: blocks in
    and next to the source plane (every pixel in one cell; rx and ry taken from
    the lattice), behind it (reversed columns and rows), images whose last
    column group is one column wide, units of several column groups, and more
    than 128 detector columns in one.  Same tolerances as above; the offset
    gradients of the blocks at depth 2 to 2.5 multiply a ray coordinate of at
    most 0.1 that is recovered from a position next to an integer, hence 1e-4
    there."""
    import fvr._lib as L

    rng = np.random.default_rng(P + H + W)
    B, N, ds, c = 2, 2, 1.5, float(P // 2)
    db = db0 + rng.uniform(-0.05, 0.05, (B, N))
    cu, cv = rng.uniform(-4, 4, (B, N)), rng.uniform(-4, 4, (B, N))
    rxc = ((np.arange(W) - 0.5 * W + 0.37) * pitch * ds / 700.0).astype(np.float32)
    ryr = ((np.arange(H) - 0.5 * H + 0.41) * pitch * ds / 700.0).astype(np.float32)
    imgs = rng.standard_normal((B, N, P, P)).astype(np.float32)
    ic = (1.0 + 0.1 * rng.random((H, W))).astype(np.float32)
    g = rng.standard_normal((N, H, W)).astype(np.float32)
    rx, ry = np.broadcast_to(rxc[None, :], (H, W)), np.broadcast_to(ryr[:, None], (H, W))
    gi, gd, gu, gv = opou.warp_sum_adjoint(imgs.astype(np.float64), db, cu, cv, rx.astype(np.float64),
                                           ry.astype(np.float64), ic.astype(np.float64), 1.0 / ds, c,
                                           g.astype(np.float64))
    dev = torch.device("cuda", 0)
    t = {k: torch.from_numpy(np.ascontiguousarray(v)).to(dev) for k, v in
         dict(imgs=imgs, offs=np.stack([db, cu, cv], -1), rxc=rxc, ryr=ryr, ic=ic, g=g).items()}
    gim = torch.full((B, N, P, P), float("nan"), device=dev)
    goffs = torch.full((3, B, N), float("nan"), dtype=torch.float64, device=dev)
    ws = torch.empty(L.query("fvr_pou_warp_sep_adjoint_workspace", N, H, W), dtype=torch.uint8, device=dev)
    L.call("fvr_pou_warp_sep_adjoint", L.ptr(t["imgs"]), B, N, P, L.ptr(t["offs"]), L.ptr(t["rxc"]), L.ptr(t["ryr"]),
           L.ptr(t["ic"]), H, W, 1.0 / ds, c, L.ptr(t["g"]), L.ptr(ws), ws.numel(), L.ptr(gim), L.ptr(goffs),
           L.stream_ptr(dev))
    assert rel_l2(gim.cpu().numpy(), gi) < 1e-5
    for got, want, tol in zip(goffs.cpu().numpy(), (gd, gu, gv), (1e-4 if abs(db0) < 3 else 1e-5, 1e-5, 1e-5)):
        assert rel_l2(got, want) < tol


def test_large_gradient_buffers_take_the_one_launch_adjoint(monkeypatch):
    """Above _GRAD_IMAGE_BYTES the adjoint that keeps dL/dimgs in shared memory
    runs (fvr_pou_warp_image_adjoint); same pose gradient."""
    import fvr.cone_beam_fvr as cb
    from fvr import synthetic

    m = cb.PerspectiveSlabFVR.from_volume(synthetic.make_ellipsoid_volume(48, 0), vox_mm=2.0, grid_blocks=(2, 2, 2),
                                          block_res=32, overlap=0.5)
    f = 1020.0 / 2.0
    k_inv = torch.tensor([[1 / f, 0, -32 / f], [0, 1 / f, -24 / f], [0, 0, 1.0]], device="cuda")
    lat = m.make_pinhole_lattice(k_inv, 1020.0, 48, 64)
    mats = synthetic.make_pinhole_mats(3, 3, device="cuda")
    grads = []
    for limit in (4 << 30, 0):
        monkeypatch.setattr(cb, "_GRAD_IMAGE_BYTES", limit)
        mm = mats.clone().requires_grad_(True)
        out = m.forward_pinhole(mm, lat)
        (out * out).sum().backward()
        grads.append(mm.grad.cpu().numpy())
    assert rel_l2(grads[0], grads[1]) < 1e-5
