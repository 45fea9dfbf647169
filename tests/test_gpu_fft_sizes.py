"""gb_image_to_grid_f32 / gb_grid_to_image_f32 over the sizes of their two
routes (prime factors up to 7 and sizes up to 8192: the fused passes; others:
cuFFT) against torch's FP64 transforms.  An FP32 transform of n^2 points errs by
about 2^-24 times a few times sqrt(log2(n^2)) in the 2-norm, so 1e-6 leaves a
factor of two to four."""
import pytest

pytestmark = pytest.mark.gpu
TOL = 1e-6


def _shifted(f, a):
    import torch

    return torch.fft.fftshift(f(torch.fft.ifftshift(a)))


@pytest.mark.parametrize("n", [2, 14, 16, 18, 22, 30, 42, 64, 70, 96, 128, 250, 256, 486, 686, 1000,
                               1022, 2048, 3072, 4374, 6144, 6272, 8192, 8748])
@pytest.mark.parametrize("tapered", [True, False])
def test_transforms_match_fp64(n, tapered):
    import torch

    from rc_gb300.autograd import ImageToGrid, grid_to_image

    gen = torch.Generator(device="cuda").manual_seed(n)
    x = torch.randn(n, n, device="cuda", generator=gen)
    g = torch.randn(n, n, dtype=torch.complex64, device="cuda", generator=gen)
    t = torch.rand(n, device="cuda", generator=gen) + 0.5 if tapered else None
    tt = 1.0 if t is None else t.double()[:, None] * t.double()[None, :]
    got = ImageToGrid.apply(x, t)
    exp = _shifted(torch.fft.fft2, x.double() / tt)
    assert float(torch.linalg.norm(got - exp) / torch.linalg.norm(exp)) < TOL
    del exp
    keep = g.clone()
    img = grid_to_image(g, t)
    exp = _shifted(lambda a: torch.fft.ifft2(a, norm="forward"), g.to(torch.complex128)).real / tt
    assert float(torch.linalg.norm(img - exp) / torch.linalg.norm(exp)) < TOL
    assert torch.equal(g, keep)  # the grid is an input
