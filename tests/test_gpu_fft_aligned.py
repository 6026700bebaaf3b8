"""Column passes whose rows share their alignment (csrc/fft2.cu: the tiles then
start on a boundary of memory, so the first holds fewer columns), against
numpy.fft in FP64: every kind of start and column count, one tile and several,
the CTA pairs of length 1024 among them.  What lies beside the columns stays,
and another launch shape gives the same bits.  Tolerance: that of the column
passes' other tests (an L2 error of about 1e-7 per two radix-2 levels)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def fg():
    from fftgal_gb300 import build
    build.build()
    import fftgal_gb300
    return fftgal_gb300


@pytest.mark.parametrize("N,other", [(4, 5), (32, 3), (256, 3), (512, 3), (1024, 3)])
@pytest.mark.parametrize("first,ncols", [(0, 1), (15, 1), (0, 16), (1, 16), (15, 18), (0, 33), (7, 33), (31, 34)])
def test_aligned_tiles(fg, N, other, first, ncols):
    import torch
    rng = np.random.default_rng(100 * ncols + first)
    pitch, nbatch, bs = 96, 2, 96 * N + 5  # a batch starts 5 columns further to the right in memory
    a = (rng.standard_normal(nbatch * bs) + 1j * rng.standard_normal(nbatch * bs)).astype(np.complex64)
    got = {}
    for shape in (-1, other):
        d = torch.from_numpy(a.view(np.float32)).cuda()
        torch.cuda.synchronize()
        st = fg.lib().fftgal_fft_columns_f32(N, d.data_ptr() + 8 * first, ncols, pitch, bs, nbatch, -1, shape, None)
        assert st == 0, fg.lib().fftgal_last_error()
        got[shape] = d.cpu().numpy().view(np.complex64)
    np.testing.assert_array_equal(got[-1], got[other])
    inside = np.zeros(nbatch * bs, bool)
    for b in range(nbatch):
        i = b * bs + first + pitch * np.arange(N)[:, None] + np.arange(ncols)
        inside[i] = True
        want = np.fft.fft(a[i].astype(np.complex128), axis=0)
        err = np.linalg.norm(got[-1][i] - want) / np.linalg.norm(want)
        assert err <= 3e-7 * np.log2(N) + 1e-7, err
    np.testing.assert_array_equal(got[-1][~inside], a[~inside])
