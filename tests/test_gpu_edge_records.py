"""The edge NCC keeps 20 moments per (item, channel) for its backward, as its C
interface says, and writes nothing behind them; the registration loss has its
own count."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,C,H,W", [(1, 1, 20, 24), (3, 2, 33, 101)])
def test_edge_stats_are_twenty_moments_per_item(B, C, H, W):
    import fvr._lib as L
    from fvr.cone_beam_fvr import edge_dominant_ncc

    dev = torch.device("cuda", 0)
    g = torch.Generator(device=dev).manual_seed(1)
    a, b = (torch.rand((B, C, H, W), generator=g, device=dev) for _ in range(2))
    crop = max(4, W // 8)
    wsb = L.query("fvr_edge_ncc_workspace", B, C, H, W, crop)
    ws = torch.empty(wsb, dtype=torch.uint8, device=dev)
    buf = torch.full((40 * B * C,), -7.0, dtype=torch.float64, device=dev)
    out, up, grad = torch.empty(B, device=dev), torch.ones(B, device=dev), torch.empty_like(a)
    L.call("fvr_edge_ncc_forward", L.ptr(a), L.ptr(b), B, B, C, H, W, crop, 0.25, 0, L.ptr(ws), wsb, L.ptr(buf),
           L.ptr(out), L.stream_ptr(dev))
    L.call("fvr_edge_ncc_backward", L.ptr(a), L.ptr(b), B, B, C, H, W, crop, 0.25, 0, L.ptr(buf), L.ptr(up), 1, 0,
           L.ptr(grad), L.stream_ptr(dev))
    assert L.query("fvr_edge_ncc_stats_count") == 20 and L.query("fvr_reg_loss_stats_count") == 25
    assert bool((buf[20 * B * C:] == -7.0).all())
    x = a.clone().requires_grad_(True)
    want = edge_dominant_ncc(x, b, reduction="none")
    want.sum().backward()
    assert torch.equal(out, want.detach()) and torch.equal(grad, x.grad)
