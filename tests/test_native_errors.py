"""Errors of the native nodes: a library status is an FvrError in the forward
and in the backward, torch's own errors (out of memory) keep their type, and
the process survives both."""
import ctypes

import pytest
import torch


def test_call_leaves_the_types_of_errors_alone():
    import fvr._native as NA

    def full(*_):
        raise torch.OutOfMemoryError("no memory")

    with pytest.raises(torch.OutOfMemoryError):
        NA.call(full, 0)


@pytest.fixture
def failing_entry():
    """Bind the native nodes to an entry that answers status 5 (on the host, nothing is launched)."""
    import fvr._lib as L
    import fvr._native as NA

    fake = ctypes.CFUNCTYPE(ctypes.c_int)(lambda: 5)
    lib = L.load()

    def bind(name):
        addr = {n: ctypes.cast(getattr(lib, n), ctypes.c_void_p).value for n in NA._ENTRIES}
        addr[name] = ctypes.cast(fake, ctypes.c_void_p).value
        NA._MOD.bind(addr, int(lib.fvr_pou_geo_stride()), int(lib.fvr_reg_loss_stats_count()))

    assert NA.module() is not None
    yield bind
    NA._bound = None
    NA.module()


@pytest.mark.gpu
def test_library_status_in_the_backward(failing_entry):
    import fvr._lib as L
    from fvr.registration import biplanar_loss_per_candidate

    x = torch.rand((2, 1, 40, 40), device="cuda", requires_grad=True)
    y = torch.rand((1, 1, 40, 40), device="cuda")
    failing_entry("fvr_reg_loss_backward")
    loss = biplanar_loss_per_candidate(x, x, y, y).sum()
    with pytest.raises(L.FvrError, match="fvr_reg_loss_backward failed with status 5"):
        loss.backward()


@pytest.mark.gpu
def test_library_status_of_a_prepared_launch():
    import fvr
    import fvr._lib as L
    import fvr._native as NA
    import fvr.torch_engine as te
    from fvr import synthetic

    eng = fvr.TorchDiffFVREngine(torch.from_numpy(synthetic.make_ellipsoid_volume(24, 2)))
    p = torch.from_numpy(synthetic.make_poses(2, 4)).cuda().requires_grad_(True)
    f = eng.prepare_spectral_target(eng(p.detach()[:1], out_res=20))
    good = te._fused_call(eng, 2, 20, (0,), (f,), None, p)
    fake = ctypes.CFUNCTYPE(ctypes.c_int)(lambda: 4)
    st = eng._sncc_storage()
    bad = NA._MOD.SnccCall(
        fn=ctypes.cast(fake, ctypes.c_void_p).value,
        status=ctypes.cast(L.load().fvr_status_string, ctypes.c_void_p).value, dtype=st.code,
        stencil=int(st.data.data_ptr()), scales=0, D=st.dims[0], H=st.dims[1], W=st.dims[2], C=2, views=[0],
        ftargs=[int(f.data_ptr())], hp=0, lin=int(f.data_ptr()), R=20, kappa=1.0, variant=0, ws=int(f.data_ptr()),
        ws_bytes=0, device=0, keep=[])
    with pytest.raises(L.FvrError, match="status 4"):
        NA.call(NA._MOD.sncc_loss, 2, p, bad)
    with pytest.raises(L.FvrError, match="shape"):
        NA.call(NA._MOD.sncc_loss, 2, p[:1], good.native)


@pytest.mark.gpu
@pytest.mark.parametrize("name", ["pinhole", "rays", "image", "image_ncc", "reg_loss"])
def test_out_of_memory_keeps_its_type(name):
    import fvr
    from fvr import synthetic
    from fvr.cone_beam_fvr import PerspectiveSlabFVR
    from fvr.registration import biplanar_loss_per_candidate

    n = 4096  # outputs of 67 MB and more
    if name in ("pinhole", "rays"):
        m = PerspectiveSlabFVR.from_volume(synthetic.make_ellipsoid_volume(40, 2), vox_mm=2.0, grid_blocks=(2, 2, 2),
                                           block_res=32, overlap=0.5)
        k_inv = torch.tensor([[1 / 500.0, 0, -0.05], [0, 1 / 500.0, -0.04], [0, 0, 1.0]], device="cuda")
        lat = m.make_pinhole_lattice(k_inv, 1020.0, 64, 64)
        mats = synthetic.make_pinhole_mats(1, 5, device="cuda").expand(n, 4, 4).contiguous()
        xs = torch.arange(64, device="cuda") * 2.0 - 64
        trg = torch.stack([xs[None].expand(64, 64), xs[:, None].expand(64, 64), torch.full((64, 64), 60.0, device="cuda")],
                          -1)[None].repeat(n, 1, 1, 1)
        src = torch.tensor([[0.0, 0.0, -300.0]], device="cuda").repeat(n, 1)
        call = (lambda: m.forward_pinhole(mats, lat)) if name == "pinhole" else (lambda: m.project_rays_batched(src, trg))
    elif name == "reg_loss":
        a = torch.rand((n, 1, 64, 64), device="cuda", requires_grad=True)
        call = lambda: biplanar_loss_per_candidate(a, a, a.detach(), a.detach())  # noqa: E731
    else:
        eng = fvr.TorchDiffFVREngine(torch.from_numpy(synthetic.make_ellipsoid_volume(24, 2)))
        poses = torch.from_numpy(synthetic.make_poses(1, 4)).cuda().expand(n, 6).contiguous()
        pred = torch.rand((n, 1, 64, 64), device="cuda", requires_grad=True)
        call = (lambda: eng(poses, out_res=64)) if name == "image" else (
            lambda: eng.spectral_ncc_loss(pred, pred.detach()[:1]))
    torch.cuda.empty_cache()
    total = torch.cuda.get_device_properties(0).total_memory
    try:  # the allocator refuses further segments on the host
        torch.cuda.set_per_process_memory_fraction(torch.cuda.memory_reserved() / total, 0)
        hold = []
        try:
            while True:
                hold.append(torch.empty(1 << 21, dtype=torch.uint8, device="cuda"))
        except torch.OutOfMemoryError:
            pass
        try:
            while True:
                hold.append(torch.empty(512, dtype=torch.uint8, device="cuda"))
        except torch.OutOfMemoryError:
            pass
        with pytest.raises(torch.OutOfMemoryError):
            call()
    finally:
        torch.cuda.set_per_process_memory_fraction(1.0, 0)
    del hold
    assert torch.isfinite(call()).all()
