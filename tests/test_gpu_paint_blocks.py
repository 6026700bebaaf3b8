"""The per-block particle counts that set a tile's fixed-point scale
(csrc/paint.cu, tile_fixbits) have to place the particles that a tile takes from
the tile above it.  Two clumps of equal size: A, whose weight in the tile's last
cell is the largest there is, and B in a cell beyond the tile's upper edge, which
also reaches that cell.  A alone may just have 20 fraction bits; with B the cell's
32-bit sum needs 19, so a count that has B in another place overflows it by 2^12
unit weights.  Two tiles along an axis are where the periodic images of the tile
above are easily confused with cells below the tile: one grid (the next cell, at
the box edge) and both interlacing grids (two cells beyond, at either edge).

Tolerance of a painted grid: that of the other tile paints, 2e-5 of the largest
cell.  Of the interlaced field: every particle of a clump rounds alike, so a mode,
its window multiplied back on, may be off by all 64 cells' roundings of 2^-20 (19
bits) in units of the zeroth mode, plus 1e-6 of the FP32 weights and 2e-6 of the
FFT: 7e-5."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# n (16 2^20 + 28) <= 54 2^32 holds up to n = 13823: 20 fraction bits
N_CLUMP = 13_820


@pytest.fixture(scope="module")
def fg():
    from fftgal_gb300 import build
    build.build()
    import fftgal_gb300
    return fftgal_gb300


def _clumps(axis, a, b, other):
    """N_CLUMP particles at cell coordinate a along `axis` and as many at b, at
    `other` along the other axes (box and grid of the same size)."""
    p = np.full((3, 2 * N_CLUMP), float(other))
    p[axis, :N_CLUMP] = a
    p[axis, N_CLUMP:] = b
    return p


def _close(got, want, rel):
    err = np.abs(got - want).max() / np.abs(want).max()
    assert err <= rel, f"max error {err:.2e} of the largest value"


def _windowed(f, Ng):
    """The k-space field of a grid's values with the PCS window multiplied back on."""
    f = np.asarray(f).reshape(Ng, Ng, -1)
    n = np.arange(Ng)
    w = np.sinc(np.where(2 * n < Ng, n, n - Ng) / Ng) ** 4
    return (f[..., 0::2] + 1j * f[..., 1::2]) * w[:, None, None] * w[None, :, None] * w[None, None, :Ng // 2 + 1]


@pytest.mark.parametrize("Ng,axis", [(64, 0), (64, 1), (64, 2), (96, 0), (32, 0), (32, 1), (40, 2), (33, 2)])
def test_one_grid(fg, oracle_lib, Ng, axis):
    V = float(Ng) ** 3
    x, y, z = _clumps(axis, Ng - 1, 0, 8)
    g = fg.Grid(Ng, float(Ng), precision="f32", host_view="lazy")
    g.p2g(fg.Catalog(x, y, z, V), (0.0, 0.0, 0.0))
    o = oracle_lib.Oracle(Ng, float(Ng))
    o.p2g(x, y, z, V, (0.0, 0.0, 0.0))
    _close(g.exportf(), np.array(o.f), 2e-5)


@pytest.mark.parametrize("Ng,axis", [(64, 0), (64, 2), (66, 0), (96, 0), (32, 0), (40, 2)])
@pytest.mark.parametrize("edge", ["middle", "box"])
def test_both_grids(fg, oracle_lib, Ng, axis, edge):
    """The grid shifted by half a cell: A at 0.5 of the tile's last cell, B one and
    a half cells above."""
    V = float(Ng) ** 3
    last = Ng // 2 - 1 if edge == "middle" else Ng - 1
    x, y, z = _clumps(axis, last + 0.5, (last + 2) % Ng, 8.5)
    g = fg.Grid(Ng, float(Ng), precision="f32", host_view="lazy")
    g.p2k(fg.Catalog(x, y, z, V))
    o = oracle_lib.Oracle(Ng, float(Ng))
    o.p2k(x, y, z, V)
    _close(_windowed(g.exportf(), Ng), _windowed(o.f, Ng), 7e-5)
