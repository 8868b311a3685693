"""The image-NCC share of the registration loss on images whose mean is large
against their spread, odd widths among them: sums about a value of the image
itself, so 1e-6 relative against float64 whatever the mean; the gradient is two
products of centred values per pixel, a few roundings, the same 1e-6."""
import pytest
import torch

from conftest import rel_l2

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("H,W", [(40, 41), (70, 128)])
@pytest.mark.parametrize("mean", [0.0, 10.0, 100.0, 1000.0])
def test_image_ncc_of_images_with_a_mean(mean, H, W, monkeypatch):
    import fvr.registration as reg

    monkeypatch.setattr(reg, "_EDGE_WEIGHT", 0.0)
    g = torch.Generator(device="cuda").manual_seed(int(mean) + H)
    a, b, ra, rb = (mean * s + torch.randn((n, 1, H, W), generator=g, device="cuda")
                    for s, n in ((1.0, 3), (0.5, 3), (1.0, 3), (2.0, 1)))
    ra = (ra + a) / 2  # correlated with a
    x, y = a.clone().requires_grad_(True), b.clone().requires_grad_(True)
    loss = reg.biplanar_loss_per_candidate(x, y, ra, rb)
    up = torch.tensor([1.0, -0.5, 2.0], device="cuda")
    got = torch.autograd.grad(loss, (x, y), up)

    def ncc(p, r):
        p, r = (t - t.mean(dim=(-2, -1), keepdim=True) for t in (p, r))
        return ((p * r).sum(dim=(-2, -1)) / (p.square().sum(dim=(-2, -1)) * r.square().sum(dim=(-2, -1))).sqrt())[:, 0]

    x64, y64 = a.double().requires_grad_(True), b.double().requires_grad_(True)
    want = 1.0 - 0.5 * (ncc(x64, ra.double()) + ncc(y64, rb.double()))
    want_g = torch.autograd.grad(want, (x64, y64), up.double())
    assert rel_l2(loss.detach().cpu().numpy(), want.detach().cpu().numpy()) < 1e-6
    for p, q in zip(got, want_g):
        assert rel_l2(p.cpu().numpy(), q.cpu().numpy()) < 1e-6


def test_moments_add_few_products_in_float32():
    """A triangle wave whose Sobel response is +-a with a long mantissa: every sum
    of squares rounds the same way in every lane.  Four products in float32
    before float64: partial sums of 1/4 .. 1, so at most 2.5 x 2^-24 relative (64
    in a row would give 9.5e-7)."""
    import fvr._lib as L

    H, W, crop = 128, 250, 8
    s = 1.0 + 4031 / 4096
    dev = torch.device("cuda", 0)
    x = torch.arange(W, device=dev) % 16
    img = (s * torch.where(x < 8, x, 16 - x).float())[None, None, None].expand(1, 1, H, W).contiguous()
    wsb = L.query("fvr_edge_ncc_workspace", 1, 1, H, W, crop)
    ws = torch.empty(wsb, dtype=torch.uint8, device=dev)
    stats, out = torch.zeros(40, dtype=torch.float64, device=dev), torch.empty(1, device=dev)
    L.call("fvr_edge_ncc_forward", L.ptr(img), L.ptr(img), 1, 1, 1, H, W, crop, 0.0, 0, L.ptr(ws), wsb, L.ptr(stats),
           L.ptr(out), L.stream_ptr(dev))
    row = img[0, 0, 0].double()
    g = 4.0 * (row[2:] - row[:-2])[crop - 1:W - crop - 1]  # Sobel x of columns crop .. W - crop - 1
    want = float((g * g).sum()) * (H - 2 * crop)
    got = stats.cpu().numpy()
    for k in (2, 3, 4):  # S_uu, S_vv, S_uv
        assert abs(got[k] / want - 1.0) < 2.5 * 2.0 ** -24, got[k] / want - 1.0
