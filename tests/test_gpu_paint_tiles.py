"""The tile paints of csrc/paint.cu against the FP64 oracle: FP64 grids
(test_paint_fp64) and FP32 grids with Ng >= 64, at the grid sizes where the tiles
differ: two tiles along an axis, extents that are odd or vary from tile to tile
(144 and 175: a CTA paints tiles of different widths along k in turn), rows that
start 16-byte aligned, 8 bytes off in turn, or neither (odd Ng), with catalogs that are uniform, wrapped over several
boxes, clumped (dense tiles) and empty, one grid with offsets and randoms and
both interlacing grids.

Tolerance: a deposit rounds by at most 2^-22 of a unit weight (21 fraction bits
or more) and its FP32 weights by about 1e-6 of itself, over at most 64 times
the particles per cell deposits in a cell: 2e-5 of the largest cell, the FP32
grids' stated tolerance."""
import numpy as np
import pytest

from catalogs import uniform_box

pytestmark = pytest.mark.gpu

SIZES = [64, 65, 66, 72, 75, 90, 91, 98, 105, 125, 128, 144, 175]


@pytest.fixture(scope="module")
def fg():
    from fftgal_gb300 import build
    build.build()
    import fftgal_gb300
    return fftgal_gb300


def _catalog(kind, Ng, L):
    rng = np.random.default_rng(Ng)
    if kind == "uniform":
        p = np.array(uniform_box(Ng, Ng ** 3 // 8, L))
    elif kind == "wrapped":
        p = (5 * rng.random((3, 20_000)) - 2) * L
    elif kind == "clump":
        p = 0.31 * L + 0.004 * L * rng.standard_normal((3, 60_000))
        p[:, ::2] = L * rng.random((3, 30_000))
    else:
        p = np.zeros((3, 0))
    return [np.asarray(a, dtype=np.float32).astype(np.float64) for a in p]


def _close(got, want, rel):
    scale = np.abs(want).max()
    err = np.abs(got - want).max() / scale
    assert err <= rel, f"max error {err:.2e} of the largest cell"


@pytest.mark.parametrize("Ng", SIZES)
@pytest.mark.parametrize("kind,offset", [("uniform", (0.0, 0.0, 0.0)), ("wrapped", (0.5, -0.3, 0.25)),
                                         ("clump", (0.5, 0.5, 0.5)), ("empty", (0.0, 0.5, 0.0))])
def test_paint_one_grid(fg, oracle_lib, Ng, kind, offset):
    L = 100.0
    V = L ** 3
    x, y, z = _catalog(kind, Ng, L)
    g = fg.Grid(Ng, L, precision="f32", host_view="lazy")
    cat = fg.Catalog(x, y, z, V)
    g.p2g(cat, offset)
    got = g.exportf()
    o = oracle_lib.Oracle(Ng, L)
    o.p2g(x, y, z, V, offset)
    if kind == "empty":  # the reference scales by 1/nbar = inf: NaN in every cell and the padding
        assert np.isnan(got).all()
        return
    _close(got, np.array(o.f), 2e-5)
    g.p2g(cat, offset)  # bit-reproducible, whatever the sort's order
    np.testing.assert_array_equal(g.exportf(), got)


@pytest.mark.parametrize("Ng", [64, 66, 75, 98])
def test_paint_with_randoms(fg, oracle_lib, Ng):
    """The randoms are painted into the catalog's grid with a negative weight."""
    L = 100.0
    V = L ** 3
    x, y, z = _catalog("clump", Ng, L)
    r = _catalog("uniform", Ng + 1, L)
    g = fg.Grid(Ng, L, precision="f32", host_view="lazy")
    rand = fg.Catalog(*r, V)
    g.p2g(fg.Catalog(x, y, z, V, rand=rand), (0.25, 0.0, 0.5))
    o = oracle_lib.Oracle(Ng, L)
    o.p2g(x, y, z, V, (0.25, 0.0, 0.5), rand=r)
    _close(g.exportf(), np.array(o.f), 2e-5)


@pytest.mark.parametrize("Ng", SIZES)
def test_paint_both_grids(fg, oracle_lib, Ng):
    """Both interlacing grids from one sort, through fft_p2k."""
    L = 100.0
    V = L ** 3
    x, y, z = _catalog("clump", Ng, L)
    g = fg.Grid(Ng, L, precision="f32", host_view="lazy")
    g.p2k(fg.Catalog(x, y, z, V))
    o = oracle_lib.Oracle(Ng, L)
    o.p2k(x, y, z, V)
    _close(g.exportf(), np.array(o.f), 2e-5)


@pytest.mark.parametrize("Ng", [5, 8, 9, 18, 24, 33, 66, 90])
@pytest.mark.parametrize("kind,offset", [("uniform", (0.0, 0.0, 0.0)), ("wrapped", (0.5, -0.3, 0.25)),
                                         ("clump", (0.5, 0.5, 0.5)), ("empty", (0.0, 0.5, 0.0))])
def test_paint_fp64(fg, oracle_lib, Ng, kind, offset):
    """FP64 grids: one warp per tile of up to 8 x 8 x 16 cells, boxes that wrap,
    tiles of more particles than one warp takes (30000 in a few cells).  A cell
    sums up to some 1e4 terms in another order than the oracle: 1e-12 of the
    largest cell, the FP64 grids' stated tolerance."""
    L = 100.0
    V = L ** 3
    x, y, z = _catalog(kind, Ng, L)
    g = fg.Grid(Ng, L, precision="f64", host_view="lazy")
    cat = fg.Catalog(x, y, z, V)
    g.p2g(cat, offset)
    o = oracle_lib.Oracle(Ng, L)
    o.p2g(x, y, z, V, offset)
    if kind == "empty":
        assert np.isnan(g.exportf()).all()
        return
    _close(g.exportf(), np.array(o.f), 1e-12)
    g.p2k(cat)
    o.p2k(x, y, z, V)
    _close(g.exportf(), np.array(o.f), 1e-12)


@pytest.mark.parametrize("Ng", [64, 96])
@pytest.mark.parametrize("edge", [0.0, 0.5])
def test_clump_at_a_tile_edge(fg, oracle_lib, Ng, edge):
    """A clump whose base cells are the first of a tile (the box edge, or the
    middle of the box where two tiles of Ng = 64 meet) reaches into the tile
    below, whose fixed-point scale has to count it: with 200000 particles near
    one cell an uncounted clump overflows that tile's 32-bit sums."""
    L = 100.0
    V = L ** 3
    rng = np.random.default_rng(3)
    p = L * edge + 0.2 * L / Ng * rng.random((3, 200_000)) + 0.1 * L / Ng
    x, y, z = (np.asarray(a, dtype=np.float32).astype(np.float64) for a in p)
    g = fg.Grid(Ng, L, precision="f32", host_view="lazy")
    g.p2g(fg.Catalog(x, y, z, V), (0.0, 0.0, 0.0))
    o = oracle_lib.Oracle(Ng, L)
    o.p2g(x, y, z, V, (0.0, 0.0, 0.0))
    _close(g.exportf(), np.array(o.f), 2e-5)
