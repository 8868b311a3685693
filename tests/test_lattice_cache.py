"""Preparing a pinhole lattice: tensors that start at the same address but are
another view, or that were written to, are another lattice."""
import pytest
import torch


def _lattice(H, W, device="cpu"):
    rx = torch.linspace(-0.1, 0.1, W, device=device).expand(H, W).contiguous()
    ry = torch.linspace(-0.08, 0.08, H, device=device)[:, None].expand(H, W).contiguous()
    ic = torch.sqrt(1.0 + rx * rx + ry * ry)
    eye = torch.eye(3, device=device)
    trg = torch.stack([1000.0 * rx, 1000.0 * ry, torch.full_like(rx, 1000.0)], -1)
    return (torch.zeros(3, device=device), trg, eye[0], eye[1], eye[2], rx, ry, ic, rx.reshape(-1), ry.reshape(-1),
            ic.reshape(-1))


def _view(lattice, f):
    v = [f(t) if t.dim() >= 2 else t for t in lattice[:8]]
    return (*v, *(t.reshape(-1) for t in v[5:8]))


VIEWS = {"coarse": lambda t: t[::2, ::2], "crop": lambda t: t[:5, :7], "rows": lambda t: t[:6]}


@pytest.mark.parametrize("native", [True, False])
@pytest.mark.parametrize("name", VIEWS)
def test_views_of_a_lattice_are_their_own(name, native, monkeypatch):
    import fvr._native as NA
    from fvr.cone_beam_fvr import _prepared_lattice

    if not native:
        monkeypatch.setattr(NA, "_MOD", None)
    lat = _lattice(12, 16)
    dev = torch.device("cpu")
    full = _prepared_lattice(lat, dev)
    sub = _view(lat, VIEWS[name])
    assert all(a.data_ptr() == b.data_ptr() for a, b in zip(lat[:8], sub[:8]))
    got = _prepared_lattice(sub, dev)
    for k in range(3):
        assert torch.equal(got[2][k], sub[5 + k])
    assert torch.equal(got[4][0], sub[5][0]) and torch.equal(got[4][1], sub[6][:, 0])
    assert _prepared_lattice(lat, dev) is full and _prepared_lattice(sub, dev) is got


@pytest.mark.parametrize("native", [True, False])
def test_a_written_lattice_is_prepared_again(native, monkeypatch):
    import fvr._native as NA
    from fvr.cone_beam_fvr import _prepared_lattice

    if not native:
        monkeypatch.setattr(NA, "_MOD", None)
    lat = _lattice(12, 16)
    dev = torch.device("cpu")
    first = _prepared_lattice(lat, dev)
    lat[8].mul_(0.5)  # the flat view of rx
    lat[2].neg_()
    again = _prepared_lattice(lat, dev)
    assert again is not first and list(again[1])[3:6] == lat[2].double().tolist()
    assert torch.equal(again[4][0], lat[5][0])
    with torch.inference_mode():  # no versions to compare
        assert _prepared_lattice(_lattice(3, 4), dev)[4] is not None


@pytest.mark.gpu
def test_a_lattice_first_used_under_a_launch_timer_takes_the_native_node():
    from fvr import profiling, synthetic
    from fvr.cone_beam_fvr import PerspectiveSlabFVR

    m = PerspectiveSlabFVR.from_volume(synthetic.make_ellipsoid_volume(40, 2), vox_mm=2.0, grid_blocks=(2, 2, 2),
                                       block_res=32, overlap=0.5)
    mats = synthetic.make_pinhole_mats(2, 5, device="cuda").requires_grad_(True)
    lat = _lattice(24, 40, "cuda")
    with profiling.LaunchTimer(["pou_warp"]):
        assert "_PinholeFn" in m.forward_pinhole(mats, lat).grad_fn.name()
    assert "_PinholeFn" not in m.forward_pinhole(mats, lat).grad_fn.name()


@pytest.mark.gpu
def test_rendering_on_views_and_after_a_write():
    from fvr import synthetic
    from fvr.cone_beam_fvr import PerspectiveSlabFVR

    m = PerspectiveSlabFVR.from_volume(synthetic.make_ellipsoid_volume(40, 2), vox_mm=2.0, grid_blocks=(2, 2, 2),
                                       block_res=32, overlap=0.5)
    mats = synthetic.make_pinhole_mats(2, 5, device="cuda")
    lat = _lattice(24, 40, "cuda")
    full = m.forward_pinhole(mats, lat)
    coarse = m.forward_pinhole(mats, _view(lat, VIEWS["coarse"]))
    assert coarse.shape == (2, 1, 12, 20)
    assert torch.allclose(coarse, full[:, :, ::2, ::2], rtol=1e-5, atol=1e-5 * float(full.max()))
    lat[7].mul_(2.0)
    assert torch.allclose(m.forward_pinhole(mats, lat), 2.0 * full, rtol=1e-6)


@pytest.mark.gpu
@pytest.mark.parametrize("native", [True, False])
def test_a_write_between_forward_and_backward_is_an_error(native, monkeypatch):
    """autograd's rule for what a node keeps, on the native node as on the Python node."""
    import fvr._native as NA
    from fvr import synthetic
    from fvr.cone_beam_fvr import PerspectiveSlabFVR

    if not native:
        monkeypatch.setattr(NA, "_MOD", None)
    m = PerspectiveSlabFVR.from_volume(synthetic.make_ellipsoid_volume(40, 2), vox_mm=2.0, grid_blocks=(2, 2, 2),
                                       block_res=32, overlap=0.5)
    mats = synthetic.make_pinhole_mats(2, 5, device="cuda").requires_grad_(True)
    lat = _lattice(24, 40, "cuda")
    out = m.forward_pinhole(mats, lat).sum()
    lat[7].mul_(2.0)
    with pytest.raises(RuntimeError, match="modified by an inplace operation"):
        out.backward()


@pytest.mark.gpu
def test_a_lattice_of_inference_tensors_still_gives_gradients():
    from fvr import synthetic
    from fvr.cone_beam_fvr import PerspectiveSlabFVR

    m = PerspectiveSlabFVR.from_volume(synthetic.make_ellipsoid_volume(40, 2), vox_mm=2.0, grid_blocks=(2, 2, 2),
                                       block_res=32, overlap=0.5)
    with torch.inference_mode():
        inf = _lattice(24, 40, "cuda")
    grads = []
    for lat in (inf, _lattice(24, 40, "cuda")):
        mats = synthetic.make_pinhole_mats(2, 5, device="cuda").requires_grad_(True)
        m.forward_pinhole(mats, lat).sum().backward()
        grads.append(mats.grad)
    assert torch.equal(*grads)
