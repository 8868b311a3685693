"""The separable warp adjoint on samples next to the far side of their image
cells: every corner's weight is formed by itself, so each element of dL/dimgs is
right to a few roundings of its own size (fractions 1 - 2^-10, positions and
weights exact in float32, one sample per cell: 4 x 2^-24 relative)."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("P,W,H,N", [(64, 20, 24, 1), (96, 47, 40, 2), (64, 30, 9, 300)])
def test_small_weights_are_not_differences(P, W, H, N):
    import fvr._lib as L

    eps = 2.0 ** -10
    B, d, c = 1, 512.0, float(P // 2)
    x, y = 2 * np.arange(W) + 1 - eps, 2 * np.arange(H) + 1 - eps  # image positions, all cells even
    rxc, ryr = ((x - c) / d).astype(np.float32), ((y - c) / d).astype(np.float32)
    assert np.array_equal(d * rxc.astype(np.float64) + c, x) and np.array_equal(d * ryr.astype(np.float64) + c, y)
    rng = np.random.default_rng(P + N)
    g = rng.standard_normal((N, H, W)).astype(np.float32)
    want = np.zeros((N, P, P))
    for dy in (0, 1):
        for dx in (0, 1):
            wt = ((1 - eps) if dy else eps) * ((1 - eps) if dx else eps)
            rows, cols = 2 * np.arange(H) + dy, 2 * np.arange(W) + dx
            r, k = rows < P, cols < P
            want[:, rows[r][:, None], cols[k][None]] += wt * g[:, r][:, :, k].astype(np.float64)
    dev = torch.device("cuda", 0)
    t = {k: torch.from_numpy(np.ascontiguousarray(v)).to(dev) for k, v in
         dict(imgs=rng.standard_normal((B, N, P, P)).astype(np.float32),
              offs=np.stack([np.full((B, N), d), np.zeros((B, N)), np.zeros((B, N))], -1), rxc=rxc, ryr=ryr,
              ic=np.ones((H, W), np.float32), g=g).items()}
    gim = torch.full((B, N, P, P), float("nan"), device=dev)
    goffs = torch.empty((3, B, N), dtype=torch.float64, device=dev)
    ws = torch.empty(L.query("fvr_pou_warp_sep_adjoint_workspace", N, H, W), dtype=torch.uint8, device=dev)
    L.call("fvr_pou_warp_sep_adjoint", L.ptr(t["imgs"]), B, N, P, L.ptr(t["offs"]), L.ptr(t["rxc"]), L.ptr(t["ryr"]),
           L.ptr(t["ic"]), H, W, 1.0, c, L.ptr(t["g"]), L.ptr(ws), ws.numel(), L.ptr(gim), L.ptr(goffs),
           L.stream_ptr(dev))
    got = gim.cpu().numpy()[0].astype(np.float64)
    assert np.abs(got - want).max() > 0 or np.array_equal(got, want)
    assert (np.abs(got - want) <= 4 * 2.0 ** -24 * np.abs(want)).all()
