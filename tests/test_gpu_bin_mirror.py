"""Binning with mirrored modes summed first (csrc/bins.cu) against the FP64
oracle: lines of sight along an axis (four modes per slab element), with two
components (two, for (1, 1, 0) the jointly mirrored ones and the modes on the
Nyquist row that have no partner), with three (one) and a zero one, at even, odd
and small grid sizes, for the interlaced and the single-paint call under both host
views (finished field binned only, or stored too).  The parity criterion of the
FP32 path (tests/golden/parity.py)."""
import numpy as np
import pytest

import parity
from catalogs import clustered_box

pytestmark = pytest.mark.gpu

LOS = [(0, 0, 1), (0, 1, 0), (1, 0, 0), (0, 1, 1), (1, 0, 1), (1, 1, 0), (1, -1, 0), (0.3, 0.5, 1.0), (0, 0, 0)]


@pytest.fixture(scope="module")
def fg():
    from fftgal_gb300 import build
    build.build()
    import fftgal_gb300
    return fftgal_gb300


def _catalog(Ng, L):
    n = 60_000
    return [np.asarray(a, dtype=np.float32).astype(np.float64) for a in clustered_box(Ng, n, L, 600, 2.0)]


@pytest.mark.parametrize("Ng", [20, 27, 64, 65, 66, 98])
@pytest.mark.parametrize("los", LOS)
def test_interlaced(fg, oracle_lib, Ng, los):
    L = 200.0
    x, y, z = _catalog(Ng, L)
    V, dK, Nmu = L ** 3, 2 * np.pi / L, 4
    want = oracle_lib.power_spectrum(Ng, L, x, y, z, los, dK, Nmu=Nmu)
    for view in ("lazy", "sync"):
        g = fg.Grid(Ng, L, precision="f32", host_view=view)
        e = parity.errors(g.power_f32(x, y, z, V, los, dK, Nmu=Nmu), want, V / len(x), Ng, L)
        assert parity.passes(e), (view, e)
    o = oracle_lib.Oracle(Ng, L)
    o.p2k(x, y, z, V)
    got, ref = np.array(g.cplx), np.array(o.cplx)  # the stored field, every mode of it
    assert np.abs(got - ref).max() <= 1e-5 * np.abs(ref).max()


@pytest.mark.parametrize("Ng", [27, 64, 66])
@pytest.mark.parametrize("los", LOS[:7])
def test_single_paint(fg, oracle_lib, Ng, los):
    """The single paint under both views, against the oracle's p2g + x2k +
    deconvolution, P, Pl and Pmu."""
    L = 200.0
    x, y, z = _catalog(Ng, L)
    V, dK = L ** 3, 2 * np.pi / L
    o = oracle_lib.Oracle(Ng, L)
    o.p2g(x, y, z, V, (0.0, 0.0, 0.0))
    o.x2k(0)
    o.deconv()
    field = np.array(o.cplx)
    res = {}
    for view in ("lazy", "sync"):
        g = fg.Grid(Ng, L, precision="f32", host_view=view)
        res[view] = g.power_f32(x, y, z, V, los, dK, Nmu=3, interlace=False)
    got = np.array(g.cplx)
    assert np.abs(got - field).max() <= 1e-5 * np.abs(field).max()
    # the sums in FP64 from the oracle's field
    n = np.fft.fftfreq(Ng, 1.0 / Ng)
    n3 = np.arange(Ng // 2 + 1, dtype=float)
    n3[2 * n3 >= Ng] -= Ng
    n2 = n[:, None, None] ** 2 + n[None, :, None] ** 2 + n3[None, None, :] ** 2
    c = np.broadcast_to(1 + ((2 * np.arange(Ng // 2 + 1)) % Ng > 0), n2.shape).astype(float).copy()
    c[0, 0, 0] = 0
    b = np.floor(np.sqrt(n2)).astype(int)
    p = np.abs(field) ** 2 / V - V / len(x)
    h = np.array(los) / np.linalg.norm(los)
    mu2 = (n[:, None, None] * h[0] + n[None, :, None] * h[1] + n3 * h[2]) ** 2 / np.where(n2 > 0, n2, 1)
    NK = len(res["lazy"]["K"])
    N = np.bincount(b.ravel(), c.ravel(), NK)
    with np.errstate(all="ignore"):
        P0 = np.bincount(b.ravel(), (p * c).ravel(), NK) / N
        P2 = np.bincount(b.ravel(), (p * c * (1.5 * mu2 - 0.5)).ravel(), NK) * 5 / N
    den = np.abs(P0) + V / len(x)
    ok = N > 0
    for view in ("lazy", "sync"):
        for l, want in ((0, P0), (1, P2)):
            err = np.abs(res[view]["P"][:, l] - want)[ok] / den[ok]
            assert err.max() <= 1e-3, (view, l, err.max())
            assert err[: int(0.8 * Ng / 2)].max() <= 1e-4, (view, l)
