"""Dense tiles of FP32 grids with Ng >= 64 (csrc/paint.cu, rot_deposit_wide): the
64-bit sums, 16 rows of a tile at a time, at tile extents that are even, odd and
uneven, rows of either alignment, clumps that cross tile corners, the box edge and
the two halves of a tile, one cell or several wide; cells beyond 2^32 units, so that
low words wrap.  Tolerance: the FP32 grids' 2e-5 of the largest cell.

And the time of the deposit does not depend on where in the tile the particles lie:
a clump in one cell, where all lanes of a warp want the same 64 cells, against the
same number of particles over 8 cells per axis (as dense a tile: both have 12
fraction bits).  Equal work, so a factor of two leaves room for noise; lanes that
walk the stencil in the same order took 4.7 times as long."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def fg():
    from fftgal_gb300 import build
    build.build()
    import fftgal_gb300
    return fftgal_gb300


@pytest.mark.parametrize("Ng", [64, 65, 66, 75, 98, 128])
@pytest.mark.parametrize("centre,width", [((0.5, 0.25, 0.5), 0.0), ((0.0, 0.0, 0.0), 1.0), ((0.25, 0.99, 0.6), 5.0)])
def test_dense_tiles(fg, oracle_lib, Ng, centre, width):
    L = 100.0
    rng = np.random.default_rng(Ng)
    n = 300_000
    p = np.array(centre)[:, None] * L + width * L / Ng * (rng.random((3, n)) - 0.5)
    p = np.concatenate([p, L * rng.random((3, 20_000))], 1).astype(np.float32).astype(np.float64)
    g = fg.Grid(Ng, L, precision="f32", host_view="lazy")
    cat = fg.Catalog(*p, L ** 3)
    for offset in ((0.0, 0.0, 0.0), (0.5, -0.3, 0.25)):
        g.p2g(cat, offset)
        got = g.exportf()
        o = oracle_lib.Oracle(Ng, L)
        o.p2g(*p, L ** 3, offset)
        want = np.array(o.f)
        err = np.abs(got - want).max() / np.abs(want).max()
        assert err <= 2e-5, f"offset {offset}: max error {err:.2e} of the largest cell"


def test_clump_takes_no_longer(fg):
    import torch
    Ng, L, n = 128, 128.0, 1_000_000
    gen = torch.Generator(device="cuda")
    gen.manual_seed(1)
    g = fg.Grid(Ng, L, precision="f32", host_view="lazy")
    g.set_timing(True)
    t = {}
    for width in (1.0, 8.0):
        x = 40.0 + width * (torch.rand((3, n), generator=gen, device="cuda") - 0.5)
        torch.cuda.synchronize()
        runs = []
        for _ in range(5):
            g.power_f32(*(x[a].data_ptr() for a in range(3)), L ** 3, (0, 0, 1), 2 * np.pi / L, where=fg.MEM_DEVICE,
                        Np=n)
            runs.append(g.stage_times()["paint_tile"])
        t[width] = min(runs)
    assert t[1.0] <= 2 * t[8.0], t
