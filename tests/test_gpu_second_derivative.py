"""Second derivatives of the spectral-NCC losses: the nodes keep the gradient
of the forward, so its own derivative is refused, natively and in Python,
instead of being left out of the result; the derivative of that gradient by
the upstream factor of the pose loss is there."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _engine(native, monkeypatch):
    import fvr
    import fvr._native as NA
    import fvr.torch_engine as te
    from fvr import synthetic

    assert NA._MOD is not None
    if not native:
        monkeypatch.setattr(NA, "_MOD", None)
        monkeypatch.setattr(te, "_NATIVE", None)
    eng = fvr.TorchDiffFVREngine(torch.from_numpy(synthetic.make_ellipsoid_volume(24, 2)))
    return eng, torch.from_numpy(synthetic.make_poses(3, 4)).cuda()


@pytest.mark.parametrize("native", [True, False])
def test_image_loss_refuses_a_second_derivative(native, monkeypatch):
    eng, _ = _engine(native, monkeypatch)
    g = torch.Generator(device="cuda").manual_seed(0)
    pred = torch.rand((2, 1, 20, 24), generator=g, device="cuda").requires_grad_(True)
    target = torch.rand((1, 1, 20, 24), generator=g, device="cuda")
    loss = eng.spectral_ncc_loss(pred, target)
    (first,) = torch.autograd.grad(loss ** 2, pred, create_graph=True)
    assert first.abs().max() > 0
    with pytest.raises(RuntimeError):
        torch.autograd.grad(first.square().sum(), pred)


@pytest.mark.parametrize("native", [True, False])
def test_pose_loss_refuses_a_second_derivative_in_the_poses(native, monkeypatch):
    eng, poses = _engine(native, monkeypatch)
    f = eng.prepare_spectral_target(eng(poses[:1] + 1.0, out_res=20))
    p = poses.clone().requires_grad_(True)
    w = torch.tensor(0.7, device="cuda", requires_grad=True)
    loss = eng.forward_spectral_ncc(p, f)
    (first,) = torch.autograd.grad(w * loss, p, create_graph=True)
    (by_w,) = torch.autograd.grad(first.sum(), w, retain_graph=True)
    assert torch.allclose(by_w * w, first.sum(), rtol=1e-5)
    with pytest.raises(RuntimeError):
        torch.autograd.grad(first.sum(), p, retain_graph=True)
    (nonlinear,) = torch.autograd.grad(loss ** 2, p, create_graph=True)
    with pytest.raises(RuntimeError):
        torch.autograd.grad(nonlinear.sum(), p)
    # poses written to before the backward, as an optimiser's loop may do, stay allowed
    q = poses.clone().requires_grad_(True)
    loss = eng.forward_spectral_ncc(q, f)
    with torch.no_grad():
        q.add_(1.0)
    loss.backward()
    assert torch.allclose(q.grad * 1.0, first.detach() / 0.7, rtol=1e-5)
