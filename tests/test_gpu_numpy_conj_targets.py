"""Targets that torch conjugates lazily (t.conj(), t.mH) give the moments of
the conjugated values: equal to the last bit, the same kernel on the same
values."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def test_conjugated_views_are_read_conjugated():
    from fvr.diff_fvr import DifferentiableFourierVolumeRenderer
    from fvr.synthetic import make_ellipsoid_volume

    r = DifferentiableFourierVolumeRenderer(make_ellipsoid_volume(0, 4, shape=(12, 15, 10)).astype(np.float64))
    h, w = r._dims("ap")
    rng = np.random.default_rng(1)
    t = torch.from_numpy(rng.standard_normal((h, w)) + 1j * rng.standard_normal((h, w)))
    specs = [(3.0, -2.0, 1.0, 0.4, -0.3, "ap")]
    want, _ = r._ncc_moments(specs, [t.numpy().conj()])
    for target in (t.conj(), t.cuda().conj(), t.cuda().mT.contiguous().mH):
        assert target.is_conj()
        assert np.array_equal(r._ncc_moments(specs, [target])[0], want)
