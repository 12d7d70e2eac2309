"""GPU test of the one-axis kernels' error in FP32 where a radix of their own
replaces the registered kernels' (fft_radix.cuh)."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [512, 1024])
def test_radix_32_is_as_exact_as_the_registered_kernels(cuda, n, monkeypatch):
    """The x pass of n = 32 x 16 or 32 x 32 points is no further from the 64-bit
    transform than that of the registered kernels (8 x 8 x 8, 16 x 8 x 8)."""
    import torch
    import gpu_fft_b200 as g

    grid = (n, 32, 128)
    gen = torch.Generator(device="cuda").manual_seed(n)
    x = torch.randn((n, 32, 65), generator=gen, dtype=torch.complex64, device="cuda")
    for forward in (True, False):
        want = torch.fft.fft(x.to(torch.complex128), dim=0) if forward else n * torch.fft.ifft(x.to(torch.complex128), dim=0)
        err = {}
        for form, choice in (("axisX{", "-1"), ("fastB{", "0")):
            monkeypatch.setenv("GPUFFT_VARIANT_B", choice)
            p = g.Plan(*grid, "float")
            assert form in p.describe()
            y = x.clone()
            p.pass_ptr(y.data_ptr(), torch.cuda.current_stream().cuda_stream, 1, forward)
            err[form] = ((y - want).norm() / want.norm()).item()
        assert err["axisX{"] <= err["fastB{"], err
