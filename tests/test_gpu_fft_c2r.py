"""The backward k pass of power-of-two FP32 grids (csrc/fft2.cu) against torch in
FP64: every split of the half length, rows that fill a CTA's group and grids
with fewer, and the row padding.  Tolerance: the FP32 bound of the grids' other
FFT tests, 2e-6 of the largest value."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def fg():
    from fftgal_gb300 import build
    build.build()
    import fftgal_gb300
    return fftgal_gb300


@pytest.mark.parametrize("Ng", [4, 8, 16, 32, 64, 128, 256, 512])
def test_backward(fg, Ng):
    import torch
    L, nh = 30.0, Ng // 2 + 1
    gen = torch.Generator(device="cuda")
    gen.manual_seed(Ng)
    f = torch.randn((Ng, Ng, nh, 2), generator=gen, device="cuda")
    z = torch.view_as_complex(f.double())
    want = torch.fft.ifft(torch.fft.ifft(z, dim=0), dim=1)
    pad = want[:, :, -1].clone()  # the transformed Nyquist column stays in the row padding
    want[:, :, 0].imag.zero_()
    want[:, :, -1].imag.zero_()
    want = torch.fft.irfft(want, n=Ng, dim=2) * (Ng / L) ** 3
    pad *= Ng ** 2 / L ** 3
    g = fg.Grid(Ng, L, precision="f32", host_view="lazy")
    g.copy_from(f.data_ptr())
    g.k2x(0)
    g.copy_to(f.data_ptr())
    got = f.view(Ng, Ng, 2 * nh).double()
    assert (got[:, :, :Ng] - want).abs().max() <= 2e-6 * want.abs().max()
    end = torch.view_as_complex(got[:, :, Ng:].contiguous())
    assert (end - pad).abs().max() <= 2e-6 * pad.abs().max()
