"""Lattices whose rays separate up to more than a rounding step: every pixel is
rendered at its own ray, not at its column's and row's midpoint."""
import pytest
import torch

from test_lattice_cache import _lattice


def _near(H, W, spread, device="cpu"):
    """rx of each column spread over the rows by a fraction of the largest |rx|."""
    lat = list(_lattice(H, W, device))
    lat[5] = lat[5] + 0.1 * spread * torch.linspace(-0.5, 0.5, H, device=device)[:, None]
    lat[8] = lat[5].reshape(-1)
    return tuple(lat)


@pytest.mark.parametrize("spread,tables,midpoints", [(0.0, True, True), (2.0 ** -21, True, False),
                                                     (0.9 * 2.0 ** -20, True, False), (2.0 ** -18, False, False)])
def test_limits_of_separable_lattices(spread, tables, midpoints):
    from fvr.cone_beam_fvr import _prepared_lattice

    entry = _prepared_lattice(_near(40, 60, spread), torch.device("cpu"))
    assert (entry[4] is not None) == tables and (entry[7] is not None) == midpoints


@pytest.mark.gpu
@pytest.mark.parametrize("H,W", [(40, 60), (33, 300)])
def test_lattice_near_the_limit_renders_at_its_own_rays(H, W, monkeypatch):
    import fvr.cone_beam_fvr as cb
    from fvr import synthetic

    m = cb.PerspectiveSlabFVR.from_volume(synthetic.make_ellipsoid_volume(40, 2), vox_mm=2.0, grid_blocks=(2, 2, 2),
                                          block_res=32, overlap=0.5)
    mats = synthetic.make_pinhole_mats(3, 5, device="cuda")
    lat = _near(H, W, 0.9 * 2.0 ** -20, "cuda")
    res = []
    for limit in (cb._SEPARABLE_REL, 0.0):  # 0: the per-pixel kernels
        monkeypatch.setattr(cb, "_SEPARABLE_REL", limit)
        cb._LATTICE_CACHE.clear()
        x = mats.clone().requires_grad_(True)
        out = m.forward_pinhole(x, lat)
        out.backward(out.detach())
        res.append((out.detach(), x.grad))
    cb._LATTICE_CACHE.clear()
    assert torch.equal(res[0][0], res[1][0])
    assert torch.allclose(res[0][1], res[1][1], rtol=1e-4, atol=1e-4 * float(res[1][1].abs().max()))
