"""The pinhole backward in chunks of poses: image gradients within the budget,
whatever the detector and the block size, and the same pose gradient (the poses
are independent; a chunk may run with another block size, so up to the order of
float32 sums)."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("route", ["native", "python", "sections"])
@pytest.mark.parametrize("block_res,H,W,N,chunk", [(32, 33, 64, 70, 7), (32, 20, 301, 300, 299), (48, 40, 50, 150, 1),
                                                   (80, 30, 47, 40, 9), (40, 24, 40, 10, 3)])
def test_chunked_backward(block_res, H, W, N, chunk, route, monkeypatch):
    import fvr._native as NA
    import fvr.cone_beam_fvr as cb
    from fvr import profiling, synthetic

    if route != "native":
        monkeypatch.setattr(NA, "_MOD", None)
    m = cb.PerspectiveSlabFVR.from_volume(synthetic.make_ellipsoid_volume(48, 0), vox_mm=2.0, grid_blocks=(2, 2, 2),
                                          block_res=block_res, overlap=0.5)
    f = 1020.0 * W / 160.0
    k_inv = torch.tensor([[1 / f, 0, -0.5 * W / f], [0, 1 / f, -0.5 * H / f], [0, 0, 1.0]], device="cuda")
    lat = m.make_pinhole_lattice(k_inv, 1020.0, H, W)
    mats = synthetic.make_pinhole_mats(N, 3, device="cuda")
    image = 4 * m.B * m.P * m.P
    up = torch.randn((N, 1, H, W), generator=torch.Generator(device="cuda").manual_seed(1), device="cuda")
    grads, extra = [], []
    for budget in (4 << 30, chunk * image):
        monkeypatch.setattr(cb, "_GRAD_IMAGE_BYTES", budget)
        x = mats.clone().requires_grad_(True)
        if route == "sections":
            with profiling.LaunchTimer(["pou_warp_bwd"], capacity=N):
                out = m.forward_pinhole(x, lat)
                base = torch.cuda.memory_allocated()
                torch.cuda.reset_peak_memory_stats()
                out.backward(up)
        else:
            out = m.forward_pinhole(x, lat)
            base = torch.cuda.memory_allocated()
            torch.cuda.reset_peak_memory_stats()
            out.backward(up)
        extra.append(torch.cuda.max_memory_allocated() - base)
        grads.append(x.grad)
        del out
    assert torch.allclose(grads[1], grads[0], rtol=1e-4, atol=1e-5 * float(grads[0].abs().max()))
    # beside the image gradients (and, where P has no fused transform, their complex copies): the weighed detector
    # gradient of a chunk, offset gradients and records of all poses
    copies = 1 if m.P in (64, 96, 128, 160) else 6
    small = 8 * chunk * H * W + 200 * m.B * N * (1 if copies == 1 else 2 + m.P * m.P // 256) + (1 << 20)
    assert extra[1] <= copies * chunk * image + small


def test_backward_holds_a_bounded_buffer():
    """2200 poses of eight 128 x 128 block images (1.15 GB): the gradients of no more
    than 1 GB at a time, beside a chunk's weighed detector gradient."""
    import fvr.cone_beam_fvr as cb
    from fvr import synthetic

    m = cb.PerspectiveSlabFVR.from_volume(synthetic.make_ellipsoid_volume(48, 0), vox_mm=2.0, grid_blocks=(2, 2, 2),
                                          block_res=64, overlap=0.5)
    N, H, W = 2200, 24, 32
    f = 1020.0 * W / 160.0
    k_inv = torch.tensor([[1 / f, 0, -0.5 * W / f], [0, 1 / f, -0.5 * H / f], [0, 0, 1.0]], device="cuda")
    lat = m.make_pinhole_lattice(k_inv, 1020.0, H, W)
    x = synthetic.make_pinhole_mats(N, 3, device="cuda").requires_grad_(True)
    out = m.forward_pinhole(x, lat).sum()
    base = torch.cuda.memory_allocated()
    torch.cuda.reset_peak_memory_stats()
    out.backward()
    assert 4 * m.B * N * m.P ** 2 > 1 << 30
    assert torch.cuda.max_memory_allocated() - base < (1 << 30) + 4 * N * H * W * 2 + 200 * m.B * N + (4 << 20)
