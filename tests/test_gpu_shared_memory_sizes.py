"""Sizes whose dynamic shared memory lies just below 48 KB, where the static
arrays of the kernel take it past what a launch has without the opt-in, and
the largest sizes beside them: the separable warp at P = 320 with each of its
row counts, at P = 340 and 512, the general warp adjoint of many blocks, and the
spectral NCC at R of about 1000.  Oracle and tolerances as in the tests of the
same kernels at ordinary sizes."""
import ctypes

import numpy as np
import pytest
import torch

from conftest import rel_l2
from oracle import pou as opou
from oracle import torch_convention as tc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("P,N,rows", [(320, 75, 16), (340, 75, 16), (512, 75, 16), (322, 38, 8), (336, 12, 4),
                                      (320, 2, 0)])
def test_separable_warp_of_large_images(P, N, rows):
    import fvr._lib as L

    B, H, W, ds, c = 1, 256, 20, 1.5, float(P // 2)
    if rows:  # the row count that the launch rule gives
        assert (N * 16 >= 1184, N * 32 >= 1184, N * 64 >= 740) == (rows == 16, rows >= 8, rows >= 4)
    rng = np.random.default_rng(P)
    db, cu, cv = (m + rng.uniform(-s, s, (B, N)) for m, s in ((700.0, 60), (0.0, 4), (0.0, 4)))
    rxc = ((np.arange(W) - 0.5 * W + 0.37) * 5.0 * ds / 700.0).astype(np.float32)
    ryr = ((np.arange(H) - 0.5 * H + 0.41) * 1.1 * ds / 700.0).astype(np.float32)
    imgs = rng.standard_normal((B, N, P, P), dtype=np.float32)
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


@pytest.mark.parametrize("P,B", [(128, 272), (64, 1030)])
def test_general_warp_adjoint_of_many_blocks(P, B):
    """Tolerances of the per-pixel path: f32 atomics, 1e-5."""
    import fvr._lib as L

    N, H, W, ds, c = 1, 9, 31, 1.5, float(P // 2)
    rng = np.random.default_rng(P)
    db, cu, cv = (m + rng.uniform(-s, s, (B, N)) for m, s in ((700.0, 60), (0.0, 30), (0.0, 30)))
    rx, ry = (rng.uniform(-0.05, 0.05, (H, W)).astype(np.float32) for _ in range(2))
    imgs = rng.standard_normal((B, N, P, P), dtype=np.float32)
    ic = (1.0 + 0.1 * rng.random((H, W))).astype(np.float32)
    g = rng.standard_normal((N, H, W)).astype(np.float32)
    ref = opou.warp_sum_adjoint(imgs.astype(np.float64), db, cu, cv, rx.astype(np.float64), ry.astype(np.float64),
                                ic.astype(np.float64), 1.0 / ds, c, g.astype(np.float64))
    dev = torch.device("cuda", 0)
    t = {k: torch.from_numpy(np.ascontiguousarray(v)).to(dev) for k, v in
         dict(imgs=imgs, offs=np.stack([db, cu, cv], -1), rx=rx, ry=ry, ic=ic, g=g).items()}
    offs = [ctypes.c_void_p(t["offs"].data_ptr() + 8 * k) for k in range(3)]
    gim = torch.zeros((B, N, P, P), device=dev)
    goffs = torch.empty((3, B, N), dtype=torch.float64, device=dev)
    ws = torch.empty(L.query("fvr_pou_warp_bwd_workspace", B, N, H * W), dtype=torch.uint8, device=dev)
    L.call("fvr_pou_warp_bwd", L.ptr(t["imgs"]), B, N, P, *offs, 1, 3, L.ptr(t["rx"]), L.ptr(t["ry"]), L.ptr(t["ic"]),
           H * W, 0, 1.0 / ds, c, L.ptr(t["g"]), L.ptr(gim), L.ptr(goffs), None, L.ptr(ws), ws.numel(),
           L.stream_ptr(dev))
    for got, want in zip((gim, *goffs), ref):
        assert rel_l2(got.cpu().numpy(), want) < 1e-5


@pytest.mark.parametrize("R", [1000, 1016])
def test_spectral_ncc_at_a_thousand_columns(R):
    import fvr

    vol = tc.make_ellipsoid_volume(16, 11)
    eng = fvr.TorchDiffFVREngine(torch.from_numpy(vol), spacing=(1.0, 1.0, 1.0))
    poses = tc.make_poses(1, 12)
    spec = tc.spectrum(vol, 2.0)
    ft = tc.prepare_spectral_target(tc.forward_image(spec, tc.make_poses(1, 13), "ap", R))
    p = torch.from_numpy(poses).cuda().requires_grad_(True)
    loss = eng.forward_spectral_ncc(p, torch.from_numpy(ft).to(torch.complex64).cuda(), view="ap")
    loss.backward()
    want, _ = tc.spectral_ncc(spec, poses, ft, "ap")
    assert abs(float(loss) - want) < 1e-5
    assert rel_l2(p.grad.cpu().numpy(), tc.spectral_ncc_grad(spec, poses, ft, "ap")) < 1e-4
