"""Line FFTs at batches where the launch rule gives different lines per CTA
(unhalved, halved for too few CTAs, halved for a mostly empty second wave, a
last CTA with fewer lines): the unnormalised inverse 2-D transform against
torch's in float64.  The rounding grows with the passes of a line, about one
each: 1e-6 relative L2 in f32, 1e-14 in f64."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,H,W", [(1, 13, 7), (3, 150, 170), (32, 150, 170), (64, 96, 96), (128, 128, 128),
                                   (512, 50, 50), (512, 16, 16), (31, 64, 80)])
@pytest.mark.parametrize("dtype,tol", [(torch.complex64, 1e-6), (torch.complex128, 1e-14)])
def test_inverse_transform(B, H, W, dtype, tol):
    from fvr import _runtime as RT

    g = torch.Generator(device="cuda").manual_seed(B)
    x = torch.randn((B, H, W), generator=g, dtype=torch.complex128, device="cuda").to(dtype)
    want = torch.fft.ifft2(x.to(torch.complex128), norm="forward")
    got = RT.fft2d(x.clone(), inverse=True)
    assert float((got - want).norm() / want.norm()) < tol
