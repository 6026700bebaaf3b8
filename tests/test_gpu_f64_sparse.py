"""Tile paint of FP64 grids (csrc/paint.cu, paint_warp_f64_kernel) where tiles are
empty or hold a few particles: against the FP64 oracle (1e-12 of the largest cell,
the FP64 grids' stated tolerance), randoms with their negative weights included.

And the time of a grid that is all but empty: clearing it and one launch.  Ten
particles on 384^3 may take four times as long as the clearing of as many bytes
plus 150 us (170 us measured, the clearing 70; 900 with a box of sums cleared and
read for every empty tile)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def fg():
    from fftgal_gb300 import build
    build.build()
    import fftgal_gb300
    return fftgal_gb300


@pytest.mark.parametrize("Ng", [2, 3, 4, 9, 16, 33, 66])
@pytest.mark.parametrize("randoms", [False, True])
def test_few_particles(fg, oracle_lib, Ng, randoms):
    L = 50.0
    V = L ** 3
    rng = np.random.default_rng(Ng)
    p = L * rng.random((3, 12))
    p[:, 0] = 0.0  # the corner of the box and a cell before its end
    p[:, 1] = L * (1 - 0.3 / Ng)
    r = L * rng.random((3, 7)) if randoms else None
    g = fg.Grid(Ng, L, precision="f64", host_view="lazy")
    rand = fg.Catalog(*r, V) if randoms else None
    for offset in ((0.0, 0.0, 0.0), (0.5, -0.3, 0.25)):
        g.p2g(fg.Catalog(*p, V, rand=rand), offset)
        o = oracle_lib.Oracle(Ng, L)
        o.p2g(*p, V, offset, **(dict(rand=r) if randoms else {}))
        want = np.array(o.f)
        assert np.abs(g.exportf() - want).max() <= 1e-12 * np.abs(want).max()
    if not randoms:
        g.p2k(fg.Catalog(*p, V))
        o.p2k(*p, V)
        want = np.array(o.f)
        assert np.abs(g.exportf() - want).max() <= 1e-12 * np.abs(want).max()


def test_an_empty_grid_takes_no_longer(fg):
    import time
    import torch
    Ng, L = 384, 100.0
    rng = np.random.default_rng(1)
    g = fg.Grid(Ng, L, precision="f64", host_view="lazy")
    cat = fg.Catalog(*(L * rng.random((3, 10))), L ** 3)
    z = torch.empty(Ng * Ng * g.Ng_pad, dtype=torch.float64, device="cuda")

    def best(call):
        t = []
        for _ in range(10):
            torch.cuda.synchronize()
            t0 = time.perf_counter()
            call()
            g.synchronize()
            torch.cuda.synchronize()
            t.append(time.perf_counter() - t0)
        return min(t)

    paint, clear = best(lambda: g.p2g(cat, (0.0, 0.0, 0.0))), best(z.zero_)
    assert paint <= 4 * clear + 150e-6, (paint, clear)
