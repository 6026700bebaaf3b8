"""The binning's slab shapes (csrc/bins.cu, slab_shape) where a grid fills few rounds
of CTAs and takes shorter slabs, and the one-mode kernel of full slabs: the tables of
power_f32 against FP64 sums over the field that the same call stores, for lines of
sight with one, two and three components, interlaced and single, the field stored and
not.  Tolerance: the parity bound of the FP32 path, 1e-4 of |P_0| + Pshot.

And the time of the one-mode kernel next to the four-mode one, which reads as much
and classifies a quarter: at Ng = 144 1.27 times as long (2.0 with slabs of 16 rows in
two rounds), at Ng = 512 1.94 (2.16 before its row loop was written for it)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

L = 100.0


@pytest.fixture(scope="module")
def fg():
    from fftgal_gb300 import build
    build.build()
    import fftgal_gb300
    return fftgal_gb300


def _positions(n):
    import torch
    gen = torch.Generator(device="cuda")
    gen.manual_seed(n)
    x = L * torch.rand((3, n), generator=gen, device="cuda")
    x[:, : n // 2] = (x[:, :50].repeat_interleave(n // 100, 1) + torch.randn((3, n // 2), generator=gen, device="cuda")) % L
    x.clamp_(0, 99.99)
    torch.cuda.synchronize()
    return x


def _multipoles(f, Ng, V, n, los, NK):
    import torch
    k = torch.arange(Ng, device="cuda", dtype=torch.float64)
    k = torch.where(2 * k < Ng, k, k - Ng)
    k3 = k[: Ng // 2 + 1]
    n2 = k[:, None, None] ** 2 + k[None, :, None] ** 2 + k3 ** 2
    c = (1.0 + ((2 * torch.arange(Ng // 2 + 1, device="cuda")) % Ng > 0).double()).expand(n2.shape).clone()
    c[0, 0, 0] = 0
    h = np.array(los) / np.linalg.norm(los)
    mu2 = (k[:, None, None] * h[0] + k[None, :, None] * h[1] + k3 * h[2]) ** 2 / torch.where(n2 > 0, n2, 1.0)
    b = torch.floor(torch.sqrt(n2)).long().reshape(-1)
    p = ((f.double() ** 2).sum(-1) / V - V / n) * c
    N = torch.bincount(b, c.reshape(-1), NK)
    leg = (torch.ones_like(mu2), 1.5 * mu2 - 0.5, (4.375 * mu2 - 3.75) * mu2 + 0.375)
    return torch.stack([torch.bincount(b, (p * q).reshape(-1), NK) * (4 * i + 1) / N for i, q in enumerate(leg)], 1)


@pytest.mark.parametrize("Ng", [128, 144, 160, 192, 225, 256, 300, 320])
@pytest.mark.parametrize("los", [(0, 0, 1), (1, 1, 0), (0, 1, 1), (1, 2, 3)])
@pytest.mark.parametrize("interlace", [True, False])
def test_tables(fg, Ng, los, interlace):
    import torch
    n, V = 200_000, L ** 3
    x = _positions(n)
    f = torch.empty((Ng, Ng, Ng // 2 + 1, 2), device="cuda")
    tables = {}
    for view in ("sync", "lazy"):
        g = fg.Grid(Ng, L, precision="f32", host_view=view)
        r = g.power_f32(*(x[a].data_ptr() for a in range(3)), V, los, 2 * np.pi / L, where=fg.MEM_DEVICE, Np=n,
                        interlace=interlace)
        tables[view] = r["P"][:, :3]
        if view == "sync":
            g.copy_to(f.data_ptr())
            g.synchronize()
            want = _multipoles(f, Ng, V, n, los, len(r["K"])).cpu().numpy()
    ok = np.isfinite(want[:, 0])
    den = np.abs(want[:, :1]) + V / n
    for view, got in tables.items():
        err = (np.abs(got - want) / den)[ok].max()
        assert err <= 1e-4, (view, err)


@pytest.mark.parametrize("Ng,most", [(144, 1.6), (512, 2.05)])
def test_one_mode_kernel_time(fg, Ng, most):
    n = 100_000
    x = _positions(n)
    g = fg.Grid(Ng, L, precision="f32", host_view="lazy")
    g.set_timing(True)
    t = {}
    for los in ((0, 0, 1), (1, 1, 1)):
        runs = []
        for _ in range(10):
            g.power_f32(*(x[a].data_ptr() for a in range(3)), L ** 3, los, 2 * np.pi / L, where=fg.MEM_DEVICE, Np=n)
            runs.append(g.stage_times()["finish_bin"])
        t[los] = min(runs)
    assert t[(1, 1, 1)] <= most * t[(0, 0, 1)], t
