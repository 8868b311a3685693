"""The epilogue of the spectral-NCC step reads the poses of this step, whatever
wrote them right before it: the host-to-host graph, whose copy kernel lets its
successors start early, alternates between far-apart pose sets and returns
exactly the device step's loss and gradient of each, every time."""
import pytest
import torch

from oracle import torch_convention as tc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("C,R", [(1, 32), (8, 64), (70, 20)])
def test_host_step_uses_the_poses_of_the_step(C, R):
    import fvr
    from fvr.graphs import BiplanarSpectralNCCStep

    eng = fvr.TorchDiffFVREngine(torch.from_numpy(tc.make_ellipsoid_volume(32, 11)))
    tp = torch.from_numpy(tc.make_poses(1, 14)).cuda()
    f = [eng.prepare_spectral_target(eng(tp, view=v, out_res=R)) for v in ("ap", "lateral")]
    sets = [torch.from_numpy(tc.make_poses(C, 15)) * s for s in (1.0, -3.0)]
    want = []
    for p in sets:
        d = p.cuda()
        torch.cuda.synchronize()
        loss, grad = eng.spectral_ncc_value_and_grad(d, f)
        want.append((float(loss), grad.cpu()))
    step = BiplanarSpectralNCCStep(eng, *f, C, host_io=True)
    for i in range(400):
        loss, grad = step(sets[i % 2])
        assert float(loss) == want[i % 2][0] and torch.equal(grad, want[i % 2][1]), i
