"""The native autograd nodes against the Python nodes (the same library calls):
equal values and gradients to the last bit for the pinhole and explicit-ray
renderers, the image step and the registration loss; saved-tensor hooks see
what the nodes keep; half-precision inputs get gradients of their type; a
replaced storage is picked up; models that rendered can be copied and pickled."""
import copy
import io

import pytest
import torch

pytestmark = pytest.mark.gpu


def _model():
    from fvr import synthetic
    from fvr.cone_beam_fvr import PerspectiveSlabFVR

    m = PerspectiveSlabFVR.from_volume(synthetic.make_ellipsoid_volume(40, 2), vox_mm=2.0, grid_blocks=(2, 2, 2),
                                       block_res=32, overlap=0.5)
    k_inv = torch.tensor([[1 / 500.0, 0, -0.05], [0, 1 / 500.0, -0.04], [0, 0, 1.0]], device="cuda")
    return m, m.make_pinhole_lattice(k_inv, 1020.0, 41, 50), synthetic.make_pinhole_mats(3, 5, device="cuda")


def _engine():
    import fvr
    from fvr import synthetic

    eng = fvr.TorchDiffFVREngine(torch.from_numpy(synthetic.make_ellipsoid_volume(24, 2)))
    return eng, torch.from_numpy(synthetic.make_poses(3, 4)).cuda()


def _calls():
    from fvr.registration import biplanar_loss_per_candidate

    g = torch.Generator(device="cuda").manual_seed(0)
    m, lat, mats = _model()
    eng, poses = _engine()
    trg = torch.rand((2, 9, 11, 3), generator=g, device="cuda") * 4 + torch.tensor([0.0, 0.0, 60.0], device="cuda")
    xs = torch.arange(11, device="cuda") * 9.0 - 45
    ys = torch.arange(9, device="cuda") * 9.0 - 36
    trg = trg + torch.stack([xs[None].expand(9, 11), ys[:, None].expand(9, 11), torch.zeros((9, 11), device="cuda")], -1)
    src = torch.tensor([[0.0, 0.0, -300.0], [5.0, 2.0, -310.0]], device="cuda")
    imgs = [torch.rand((3, 1, 40, 98), generator=g, device="cuda") for _ in range(2)]
    refs = [torch.rand((1, 1, 40, 98), generator=g, device="cuda") for _ in range(2)]
    targ = torch.rand((1, 1, 28, 28), generator=g, device="cuda")
    return {
        "pinhole": (lambda a: m.forward_pinhole(a, lat), [mats]),
        "rays": (lambda s, t: m.project_rays_batched(s, t), [src, trg]),
        "image": (lambda p: eng(p, view="lateral", out_res=28), [poses]),
        "image_ncc": (lambda p: eng.spectral_ncc_loss(eng(p, out_res=28), targ), [poses]),
        "reg_loss": (lambda a, b: biplanar_loss_per_candidate(a, b, *refs), imgs),
    }


@pytest.mark.parametrize("name", ["pinhole", "rays", "image", "image_ncc", "reg_loss"])
def test_native_nodes_equal_python_nodes(name, monkeypatch):
    import fvr._native as NA

    assert NA.module() is not None
    fn, inputs = _calls()[name]
    res = []
    for native in (True, False):
        if not native:
            monkeypatch.setattr(NA, "_MOD", None)
        x = [t.clone().requires_grad_(True) for t in inputs]
        out = fn(*x)
        up = torch.linspace(0.5, 1.5, out.numel(), device="cuda").view(out.shape)
        res.append([out.detach(), *torch.autograd.grad(out, x, up)])
        with torch.no_grad():
            assert torch.equal(fn(*inputs), res[-1][0])
    # the explicit rays' warp adjoint adds with atomics: equal up to the order of its float additions
    for a, b in zip(*res):
        if name == "rays":
            assert torch.allclose(a, b, rtol=1e-4, atol=1e-5 * float(b.abs().max()))
        else:
            assert torch.equal(a, b)
    monkeypatch.undo()
    packed = []
    with torch.autograd.graph.saved_tensors_hooks(lambda t: packed.append(t.shape) or t.cpu(), lambda t: t.cuda()):
        x = [t.clone().requires_grad_(True) for t in inputs]
        out = fn(*x)
    up = torch.linspace(0.5, 1.5, out.numel(), device="cuda").view(out.shape)
    again = torch.autograd.grad(out, x, up)
    assert packed
    for a, b in zip(again, res[0][1:]):
        assert torch.allclose(a, b, rtol=1e-4, atol=1e-5 * float(b.abs().max()))


def test_native_nodes_types_and_replaced_storage():
    m, lat, mats = _model()
    a = mats.double().requires_grad_(True)
    out = m.forward_pinhole(a, lat)
    (g,) = torch.autograd.grad(out.sum(), a)
    assert out.dtype == torch.float32 and g.dtype == torch.float64
    f32 = out.detach().clone()
    m.to_precision(torch.bfloat16)
    bf16 = m.forward_pinhole(mats, lat)
    assert not torch.equal(bf16, f32) and torch.allclose(bf16, f32, atol=0.02 * float(f32.max()))
    eng, poses = _engine()
    before = eng(poses, out_res=28)
    eng.to_precision(torch.float16)
    after = eng(poses, out_res=28)
    assert not torch.equal(before, after) and torch.allclose(before, after, atol=0.01 * float(before.max()))
    for obj, call in ((m, lambda o: o.forward_pinhole(mats, lat)), (eng, lambda o: o(poses, out_res=28))):
        want = call(obj)
        assert torch.equal(call(copy.deepcopy(obj)), want)
        buf = io.BytesIO()
        torch.save(obj, buf)
        buf.seek(0)
        assert torch.equal(call(torch.load(buf, weights_only=False)), want)
