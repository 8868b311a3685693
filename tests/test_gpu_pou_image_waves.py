"""Block images with 256 threads, two to an SM (many images a call), against the
512-thread form (few images a call) that the unfused slice + FFT path pins: the
forward does the same arithmetic per element and agrees bit for bit, the
adjoint adds the same f32 products over other lanes (at most 64 a lane before
they are summed in f64), so 2e-5 relative L2, the bound of the unfused
comparison.  P = 160 keeps 512 threads at any count."""
import ctypes

import numpy as np
import pytest
import torch

from conftest import rel_l2

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("block_res,dtype", [(32, torch.float32), (48, torch.float32), (64, torch.float16),
                                             (32, torch.bfloat16), (64, torch.float32), (80, torch.bfloat16)])
def test_many_block_images_equal_few(block_res, dtype):
    import fvr._lib as L
    from fvr.cone_beam_fvr import PerspectiveSlabFVR
    from fvr.synthetic import make_ellipsoid_volume, make_pinhole_mats

    m = PerspectiveSlabFVR.from_volume(make_ellipsoid_volume(48, 3), vox_mm=1.5, grid_blocks=(1, 2, 1),
                                       block_res=block_res, overlap=0.5, dtype=dtype)
    B, P, dev, st = m.B, m.P, m._dev, m._stencil
    sms = torch.cuda.get_device_properties(dev).multi_processor_count
    N = (4 * sms + B - 1) // B  # four waves of one image an SM
    mats = make_pinhole_mats(N, 4, sad_mm=400.0, device=dev).to(torch.float32).contiguous()
    geo = torch.empty((N, int(L.query("fvr_pou_geo_stride"))), dtype=torch.float64, device=dev)
    offs = torch.empty((B, N, 3), dtype=torch.float64, device=dev)
    base = (ctypes.c_double * 12)(*([0.0] * 3 + [1.0, 0, 0] + [0, 1.0, 0] + [0, 0, 1.0]))
    s = L.stream_ptr(dev)
    L.call("fvr_pou_pose", L.ptr(mats), None, N, base, float(P) * m.ds_block, L.ptr(m.centers), B, L.ptr(geo),
           L.ptr(offs), s)
    g = torch.from_numpy(np.random.default_rng(1).standard_normal((B, N, P, P)).astype(np.float32)).to(dev)

    def run(lo, hi):
        n = hi - lo
        imgs = torch.full((B, n, P, P), float("nan"), device=dev)
        gg, geo_n = g[:, lo:hi].contiguous(), geo[lo:hi].contiguous()
        head = (st.code, L.ptr(st.data), L.ptr(st.scales), B, P, L.ptr(geo_n), n, L.ptr(m._freqs))
        L.call("fvr_pou_slice_image", *head, L.ptr(imgs), s)
        wsb = L.query("fvr_pou_slice_image_adjoint_workspace", B, n)
        ws = torch.empty(wsb, dtype=torch.uint8, device=dev)
        L.call("fvr_pou_slice_image_adjoint", *head, L.ptr(gg), L.ptr(ws), wsb, s)
        return imgs, ws[: n * B * 48].view(torch.float64).view(n, B, 6).cpu().numpy()

    many, adj = run(0, N)
    for lo, hi in ((0, 1), (N // 2, N // 2 + 3), (N - 1, N)):
        few, part = run(lo, hi)
        assert torch.equal(few, many[:, lo:hi])
        assert rel_l2(adj[lo:hi], part) < 2e-5
