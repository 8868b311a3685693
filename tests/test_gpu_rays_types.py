"""project_rays_batched without given axes: float64 points keep detector axes
formed in float64 (the general path, to the last bit), in value and gradient."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _model():
    from fvr import synthetic
    from fvr.cone_beam_fvr import PerspectiveSlabFVR

    return PerspectiveSlabFVR.from_volume(synthetic.make_ellipsoid_volume(48, 2), vox_mm=2.0, grid_blocks=(2, 2, 2),
                                          block_res=32, overlap=0.5)


def _points(H, W, dtype):
    g = torch.Generator(device="cuda").manual_seed(3)
    x = (torch.arange(W, device="cuda", dtype=dtype) - 0.5 * (W - 1)) * (160.0 / max(H, W))
    y = (torch.arange(H, device="cuda", dtype=dtype) - 0.5 * (H - 1)) * (160.0 / max(H, W))
    trg = torch.stack([x[None].expand(H, W), y[:, None].expand(H, W), torch.full_like(x[None].expand(H, W), 200.0)], -1)
    trg = trg[None].repeat(2, 1, 1, 1)
    if dtype == torch.float64:
        trg = trg + 1e-6 * torch.rand(trg.shape, generator=g, device="cuda", dtype=dtype)
    return torch.tensor([[3.0, -2.0, -400.0], [0.0, 5.0, -410.0]], device="cuda", dtype=dtype), trg


def test_float64_points_keep_float64_axes():
    from fvr.cone_beam_rays import project_rays_batched

    m = _model()
    src, trg = _points(31, 40, torch.float64)
    res = []
    for given in (False, True):
        s, t = src.clone().requires_grad_(True), trg.clone().requires_grad_(True)
        out = project_rays_batched(m, s, t, *m._extract_detector_basis(s, t)) if given else m.project_rays_batched(s, t)
        up = torch.linspace(0.5, 1.5, out.numel(), device="cuda").view(out.shape)
        res.append((out.detach(), *torch.autograd.grad(out, (s, t), up)))
    assert torch.equal(res[0][0], res[1][0])
    for a, b in zip(res[0][1:], res[1][1:]):  # the warp adjoint adds with atomics: equal up to their order
        assert a.dtype == torch.float64 and torch.allclose(a, b, rtol=1e-3, atol=1e-5 * float(b.abs().max()))


def test_whole_number_points_stay_refused():
    m = _model()
    src, trg = _points(3, 4, torch.float32)
    with pytest.raises(RuntimeError):
        m.project_rays_batched(src, trg.round().to(torch.int64))


@pytest.mark.parametrize("H,W", [(1, 1), (1, 6), (5, 1)])
def test_lattices_of_one_row_or_column(H, W):
    """An axis without extent is a zero vector and gets no gradient; the other
    axis and the rays keep theirs."""
    from fvr.cone_beam_rays import project_rays_batched

    m = _model()
    src, trg = _points(H, W, torch.float32)
    res = []
    for given in (False, True):
        s, t = src.clone().requires_grad_(True), trg.clone().requires_grad_(True)
        if given:
            u, v, n = (torch.zeros_like(s) for _ in range(3))
            if W > 1:
                u = t[:, 0, -1] - t[:, 0, 0]
                u = u / (u.norm(dim=-1, keepdim=True) + 1e-12)
            if H > 1:
                v = t[:, -1, 0] - t[:, 0, 0]
                v = v / (v.norm(dim=-1, keepdim=True) + 1e-12)
            out = project_rays_batched(m, s, t, u, v, n.detach())
        else:
            out = m.project_rays_batched(s, t)
        up = torch.linspace(0.5, 1.5, out.numel(), device="cuda").view(out.shape)
        res.append((out.detach(), *torch.autograd.grad(out, (s, t), up)))
    for a, b in zip(*res):
        assert torch.allclose(a, b, rtol=1e-3, atol=1e-4 * float(b.abs().max()) + 1e-6)
