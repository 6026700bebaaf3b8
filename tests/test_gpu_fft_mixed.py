"""The mixed-radix FFT passes of FP32 grids (csrc/fft3.cu) against numpy in
FP64: forward and backward transforms at every kind of split (one factor, two
equal ones, the largest, odd and even lengths, each prime up to 13), and the
backward k pass at powers of two.  Round trips through fft_x2k / fft_k2x with
their normalisations.

Tolerance: the FP32 bound of the grids' FFT tests, 2e-6 of the largest value
(an L2 error of a few 1e-7, whose largest of 1e7 Gaussian values is about five
times as large); twice that after a transform there and back."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIZES = [5, 6, 13, 22, 25, 26, 27, 30, 33, 49, 65, 77, 81, 91, 96, 100, 121, 135, 169, 192, 225]


@pytest.fixture(scope="module")
def fg():
    from fftgal_gb300 import build
    build.build()
    import fftgal_gb300
    return fftgal_gb300


def _grid(fg, Ng, L, values):
    g = fg.Grid(Ng, L, precision="f32", host_view="lazy")
    f = np.zeros((Ng, Ng, g.Ng_pad))
    f[:, :, :Ng] = values
    g.importf(f.ravel())
    return g


@pytest.mark.parametrize("Ng", SIZES)
def test_forward_and_back(fg, Ng):
    L = 50.0
    rng = np.random.default_rng(Ng)
    x = rng.standard_normal((Ng, Ng, Ng)).astype(np.float32).astype(np.float64)
    g = _grid(fg, Ng, L, x)
    g.x2k(0)
    k = g.exportf().reshape(Ng, Ng, g.Ng_pad)
    want = np.fft.rfftn(x) * (L / Ng) ** 3
    got = k[..., 0::2] + 1j * k[..., 1::2]
    assert np.abs(got - want).max() <= 2e-6 * np.abs(want).max()
    g.k2x(0)
    back = g.exportf().reshape(Ng, Ng, g.Ng_pad)[:, :, :Ng]
    assert np.abs(back - x).max() <= 4e-6 * np.abs(x).max()


@pytest.mark.parametrize("Ng", [4, 8, 32, 128, 15, 48, 105])
def test_backward_ignores_imaginary_ends(fg, Ng):
    """Im X[0] and Im X[Ng/2] of every k row are ignored, as FFTW's c2r does."""
    L = 20.0
    rng = np.random.default_rng(Ng)
    nh = Ng // 2 + 1
    z = (rng.standard_normal((Ng, Ng, nh)) + 1j * rng.standard_normal((Ng, Ng, nh))).astype(np.complex64)
    g = fg.Grid(Ng, L, precision="f32", host_view="lazy")
    f = np.zeros((Ng, Ng, g.Ng_pad))
    f[..., 0::2], f[..., 1::2] = z.real, z.imag
    g.importf(f.ravel())
    g.k2x(0)
    got = g.exportf().reshape(Ng, Ng, g.Ng_pad)[:, :, :Ng]
    want = np.fft.irfft(np.fft.ifft(np.fft.ifft(z.astype(np.complex128), axis=0), axis=1), n=Ng, axis=2)
    want *= Ng ** 3 / L ** 3
    assert np.abs(got - want).max() <= 2e-6 * np.abs(want).max()
