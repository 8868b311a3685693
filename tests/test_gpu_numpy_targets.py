"""Item moments of the NumPy-convention NCC when items share targets: host
arrays, device tensors, views of them and both mixed give the moments of
separate calls with one target each (the same kernel on the same values: equal
to the last bit), and a target of the wrong size is refused."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def test_shared_host_and_device_targets():
    from fvr.diff_fvr import DifferentiableFourierVolumeRenderer
    from fvr.synthetic import make_ellipsoid_volume

    r = DifferentiableFourierVolumeRenderer(make_ellipsoid_volume(0, 4, shape=(12, 15, 10)).astype(np.float64))
    rng = np.random.default_rng(0)
    (ah, aw), (lh, lw) = r._dims("ap"), r._dims("lateral")
    ap = rng.standard_normal((ah, aw)) + 1j * rng.standard_normal((ah, aw))
    wide = rng.standard_normal((lh, 2 * lw)) + 1j * rng.standard_normal((lh, 2 * lw))
    lat = wide[:, ::2]  # not contiguous
    lat_dev = torch.from_numpy(wide).cuda()[:, ::2]
    specs = [(3.0, -2.0, 1.0, 0.4, -0.3, "ap"), (1.0, 2.0, -4.0, 0.1, 0.2, "lateral"),
             (2.0, 0.5, 0.0, -0.4, 0.9, "ap"), (-6.0, 2.5, 1.5, 0.0, 0.0, "lateral")]
    single = np.concatenate([r._ncc_moments([s], [ap if s[5] == "ap" else lat])[0] for s in specs])
    ap_dev = torch.from_numpy(ap).cuda()
    for a, b in ((ap, lat), (ap_dev, lat_dev), (ap, lat_dev), (ap_dev, lat)):
        got, sizes = r._ncc_moments(specs, [a, b, a, b])
        assert np.array_equal(got, single)
        assert [s[:2] for s in sizes] == [(ah, aw), (lh, lw), (ah, aw), (lh, lw)]
    with pytest.raises(RuntimeError):
        r._ncc_moments(specs[:1], [ap[:-1]])
