"""The fused per-candidate registration loss and its image gradients against a
float64 torch composition of the same loss, at the sizes where the marching
kernels' strips can go wrong: widths around multiples of the 60 (moments) and
56 (adjoint) columns a warp produces, odd widths (scalar loads), heights
around multiples of the 32 rows, three rows and columns of interior, widths on both
sides of the second scale's limit of 96, one and several references, and
images that are not 8-byte aligned.

Tolerance: every f32 value of the pipeline is rounded about 20 times, so 2e-6
of the loss (|loss| <= 2) and 1e-5 relative L2 of a gradient whose fields
cancel by up to a factor ten."""
import pytest
import torch

from conftest import rel_l2

pytestmark = pytest.mark.gpu


def _loss64(ims, refs):
    import torch.nn.functional as F

    k = torch.tensor([[-1.0, 0, 1], [-2, 0, 2], [-1, 0, 1]], dtype=torch.float64, device=ims[0].device)
    W = ims[0].shape[-1]
    crop = max(4, W // 8)

    def conv(x, f):
        return F.conv2d(x, f[None, None], padding=1)

    def ncc(a, b):
        a, b = a - a.mean((-2, -1), keepdim=True), b - b.mean((-2, -1), keepdim=True)
        den = (a.square().sum((-2, -1)) * b.square().sum((-2, -1))).clamp(min=1e-12).sqrt()
        return ((a * b).sum((-2, -1)) / den)[:, 0]

    def edge(a, b):
        s = slice(crop, -crop)
        return 0.5 * (ncc(conv(a, k)[..., s, s], conv(b, k)[..., s, s]) +
                      ncc(conv(a, k.T)[..., s, s], conv(b, k.T)[..., s, s]))

    def sim(a, b):
        e = edge(a, b)
        if W >= 96:
            box = torch.full((3, 3), 1.0 / 9.0, dtype=torch.float64, device=a.device)
            e = 0.75 * e + 0.25 * edge(conv(a, box), conv(b, box))
        return 0.75 * e + 0.25 * ncc(a, b)

    return 1.0 - 0.5 * sum(sim(a, b) for a, b in zip(ims, refs))


@pytest.mark.parametrize("B,Bt,H,W,offset", [
    (1, 1, 11, 11, 0), (2, 1, 33, 59, 0), (3, 3, 32, 60, 0), (2, 2, 31, 61, 0), (2, 1, 40, 95, 0), (3, 1, 64, 96, 0),
    (2, 2, 65, 112, 0), (1, 1, 97, 113, 0), (5, 5, 63, 120, 0), (2, 1, 27, 100, 0), (2, 1, 70, 128, 1),
    (3, 1, 256, 256, 0),
])
def test_fused_loss_vs_float64(B, Bt, H, W, offset):
    from fvr.registration import biplanar_loss_per_candidate

    g = torch.Generator(device="cuda").manual_seed(H * 1000 + W)

    def image(n, level):  # smooth structure on a level, plus noise
        y = torch.linspace(0, 3, H, device="cuda")[:, None]
        x = torch.linspace(0, 4, W, device="cuda")
        ph = torch.rand((n, 1, 1, 1), generator=g, device="cuda")
        v = level + torch.sin(2 * y + 6 * ph) * torch.cos(3 * x - 4 * ph) + 0.1 * torch.randn(
            (n, 1, H, W), generator=g, device="cuda")
        flat = torch.empty(v.numel() + offset, device="cuda")
        flat[offset:] = v.reshape(-1)
        return flat[offset:].view(n, 1, H, W)

    ims = [image(B, 2.0).requires_grad_(True) for _ in range(2)]
    refs = [image(Bt, 1.0) for _ in range(2)]
    up = torch.rand(B, generator=g, device="cuda") + 0.5
    loss = biplanar_loss_per_candidate(ims[0], ims[1], refs[0], refs[1])
    grads = torch.autograd.grad(loss, ims, up)
    i64 = [x.detach().double().requires_grad_(True) for x in ims]
    ref = _loss64(i64, [x.double() for x in refs])
    gref = torch.autograd.grad(ref, i64, up.double())
    assert loss.shape == (B,)
    assert (loss.double() - ref).abs().max() < 2e-6
    for a, b in zip(grads, gref):
        assert rel_l2(a.cpu().numpy(), b.cpu().numpy()) < 1e-5


def test_loss_composed_when_the_references_need_a_gradient():
    """References that need a gradient (and mismatched views) keep the composed
    loss, with the same value as the fused one."""
    from fvr.registration import biplanar_loss_per_candidate

    g = torch.Generator(device="cuda").manual_seed(3)
    ims = [torch.rand((2, 1, 48, 100), generator=g, device="cuda") for _ in range(2)]
    refs = [torch.rand((2, 1, 48, 100), generator=g, device="cuda") for _ in range(2)]
    fused = biplanar_loss_per_candidate(*ims, *refs)
    rg = refs[0].clone().requires_grad_(True)
    composed = biplanar_loss_per_candidate(ims[0], ims[1], rg, refs[1])
    assert torch.allclose(fused, composed, atol=2e-6)
    (gr,) = torch.autograd.grad(composed.sum(), rg)
    assert gr.shape == rg.shape and bool(gr.abs().sum() > 0)
