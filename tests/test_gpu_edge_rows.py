"""The marching edge kernels at every number of rows a warp may take: batches at
which the launch rules give 8, 12, 16, 24 and 32 (moments and adjoint each), a
height that leaves a remainder of five rows for all of them.  Registration loss
against float64 torch, tolerances of test_gpu_reg_loss; edge NCC means of one
and of several items against the items themselves."""
import pytest
import torch

from conftest import rel_l2
from test_gpu_reg_loss import _loss64

pytestmark = pytest.mark.gpu
H, W = 197, 100  # two strips of 60 columns (moments) and of 56 (adjoint)


def _rows(pairs):
    jobs = {r: pairs * 2 * -(-H // r) for r in (8, 12, 16, 24, 32)}
    best, cost = 32, None
    for r in (32, 24, 16, 12, 8):
        c = -(-jobs[r] // (148 * 12)) * (r + 6)
        if cost is None or 10 * c < 9 * cost:
            best, cost = r, c
    return best, next((r for r in (8, 12, 16, 24) if jobs[r] <= 148 * 16), 32)


@pytest.mark.parametrize("B,rows", [(1, (8, 8)), (20, (12, 8)), (28, (16, 12)), (36, (24, 16)), (52, (32, 24)),
                                    (70, (24, 32))])
def test_registration_loss_at_each_row_count(B, rows):
    from fvr.registration import biplanar_loss_per_candidate

    assert _rows(2 * B) == rows
    g = torch.Generator(device="cuda").manual_seed(B)
    y, x = torch.linspace(0, 3, H, device="cuda")[:, None], torch.linspace(0, 4, W, device="cuda")

    def image(n):
        ph = torch.rand((n, 1, 1, 1), generator=g, device="cuda")
        return 1.5 + torch.sin(2 * y + 6 * ph) * torch.cos(3 * x - 4 * ph) + 0.1 * torch.randn(
            (n, 1, H, W), generator=g, device="cuda")

    ims, refs = [image(B).requires_grad_(True) for _ in range(2)], [image(1) for _ in range(2)]
    loss = biplanar_loss_per_candidate(*ims, *refs)
    grads = torch.autograd.grad(loss.sum(), ims)
    i64 = [t.detach().double().requires_grad_(True) for t in ims]
    ref = _loss64(i64, [t.double() for t in refs])
    assert (loss.double() - ref).abs().max() < 2e-6
    for a, b in zip(grads, torch.autograd.grad(ref.sum(), i64)):
        assert rel_l2(a.cpu().numpy(), b.cpu().numpy()) < 1e-5


@pytest.mark.parametrize("B", [1, 3])
def test_edge_ncc_mean(B):
    from fvr.cone_beam_fvr import edge_dominant_ncc

    g = torch.Generator(device="cuda").manual_seed(B)
    a, b = (torch.rand((B, 2, 300, 97), generator=g, device="cuda") for _ in range(2))
    each, mean = edge_dominant_ncc(a, b, reduction="none"), edge_dominant_ncc(a, b)
    assert each.shape == (B,) and mean.shape == ()
    assert abs(float(mean) - float(each.double().mean())) < 1e-7
