"""The spectral-NCC epilogue on both sides of one chunk of 128 (view, candidate)
items: batches of 64 and 65 candidates in two views (one and two chunks), 129 in
one view and 300 in two give every candidate the gradient and the losses of
batches of one candidate (1/C of them), to the fp64 sums' rounding (1e-6 of
float32 values)."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("C,views", [(64, ("ap", "lateral")), (65, ("ap", "lateral")), (129, ("ap",)),
                                     (300, ("ap", "lateral"))])
def test_chunked_epilogue_matches_single_candidates(C, views):
    import fvr
    from fvr import synthetic

    eng = fvr.TorchDiffFVREngine(torch.from_numpy(synthetic.make_ellipsoid_volume(24, 2)))
    poses = torch.from_numpy(synthetic.make_poses(C, 3)).cuda()
    tp = torch.from_numpy(synthetic.make_poses(1, 4)).cuda()
    with torch.no_grad():
        fts = [eng.prepare_spectral_target(eng(tp, view=v, out_res=20)) for v in views]
    loss, grad = eng.spectral_ncc_value_and_grad(poses, fts, views)
    total = 0.0
    for c in (0, 1, 63, 64, C - 1):
        if c >= C:
            continue
        lo, g = eng.spectral_ncc_value_and_grad(poses[c:c + 1], fts, views)
        assert torch.allclose(grad[c] * C, g[0], rtol=1e-5, atol=1e-6 * float(g.abs().max()))
    total = sum(float(eng.spectral_ncc_value_and_grad(poses[c:c + 1], fts, views)[0]) for c in range(C)) / C
    assert abs(float(loss) - total) < 2e-6
