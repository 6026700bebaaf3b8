"""Performance cases of the library: the calls its users make, over the range
of sizes that its configurations, tests and benchmark use.

Kinds of case (key "kind"):
  power   one FP32 catalog in GPU memory -> multipoles and mu wedges, in one
          call: interlaced (power_f32), redshift space (power_rsd_f32), one
          paint (power_f32(interlace=False)) or learned (power_learned_f32)
  batch   a list of FP32 catalogs of uneven sizes in page-locked host memory
          (power_batch_f32), as a covariance set is run
  p2k     the drop-in API on an FP64 grid: host doubles -> k-space field
  window  the drop-in API on an FP32 grid: a k-space power grid to
          configuration space, the sub-box window, back to k space (the loop
          of the sub-box driver): both directions of the FFT
  train   one training step of the aliasing perceptron

Every handle (grid, plan, trainer) is made in prepare(), as a program keeps
it.  The multipoles are sums over FP32 grids; they are returned as FP32 values,
the seven digits that the library's own text tables print.  Mean wavenumbers
are FP64 and mode counts are integers.
"""
import math

import numpy as np
import torch

import fftgal_gb300 as fg
from fftgal_gb300 import alias_mlp

L_BOX = 1000.0
AH = 1.0  # velocities in units of the displacement
# the reference driver's six lines of sight
LOS = {"001": (0.0, 0.0, 1.0), "010": (0.0, 1.0, 0.0), "100": (1.0, 0.0, 0.0),
       "011": (0.0, 1.0, 1.0), "101": (1.0, 0.0, 1.0), "110": (1.0, 1.0, 0.0)}


def _power(name, mode, Ng, Np, los="001", Nmu=3, fold=1, clustered=True):
    c = dict(kind="power", mode=mode, Ng=Ng, Np=Np, los=los, Nmu=Nmu, fold=fold, clustered=clustered)
    return dict(c, name=name) if name else c


def listed():
    return [
        # the smallest call: a quick look at a small catalog, all latency
        _power("tiny-ng64", "interlaced", 64, 40_000, los="011"),
        # a uniform box of 1e6 galaxies on 128^3
        _power("uniform-ng128", "interlaced", 128, 1_000_000, clustered=False),
        # an odd, ragged grid size (FFT lengths with factors 3 and 5)
        _power("odd-ng225", "interlaced", 225, 1_200_000, los="101"),
        # a mid-size mock of a mixed set: a size that is no power of two, folded twice
        _power("mock-ng384-fold2", "interlaced", 384, 6_000_000, los="100", fold=2),
        # a redshift-space mock with ten wedges
        _power("rsd-ng512-nmu10", "rsd", 512, 10_000_000, Nmu=10),
        # a quick single-paint measurement of the same size, folded four times
        _power("single-ng512-fold4", "single", 512, 10_000_000, los="110", fold=4),
        # single paint plus the learned aliasing correction
        _power("learned-ng256", "learned", 256, 3_000_000),
        # the headline: 1e8 galaxies on 1024^3
        _power("headline-ng1024", "interlaced", 1024, 100_000_000, clustered=False),
        # a covariance set streamed from host memory
        dict(name="batch-ng256", kind="batch", Ng=256, Np=1_500_000, ncat=8, los="001", Nmu=3),
        # FP64 throughout, host doubles in
        dict(name="p2k-f64-ng128", kind="p2k", Ng=128, Np=1_000_000, clustered=False),
        # the sub-box driver's k2x -> window -> x2k on 512^3
        dict(name="window-ng512", kind="window", Ng=512, Nsub=4),
        # the trainer's batch
        dict(name="train-n4096", kind="train", n=4096),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


_POW2 = (64, 128, 256, 512, 1024)
_EVEN = (72, 90, 96, 120, 144, 160, 192, 240, 300, 320, 360, 384, 448, 480, 500)
_ODD = (75, 105, 125, 175, 189, 225, 245)


def draw(rng):
    kind = rng.choice(("power",) * 7 + ("batch", "p2k", "window", "train"))
    los = rng.choice(sorted(LOS))
    if kind == "power":
        Ng = rng.choice(rng.choice((_POW2, _POW2, _EVEN, _EVEN, _ODD)))
        Np = _log_int(rng, max(2e4, 0.01 * Ng ** 3), min(8e7, max(4e4, 0.5 * Ng ** 3)))
        return _power(None, rng.choice(("interlaced", "interlaced", "rsd", "single", "learned")), Ng, Np, los=los,
                      Nmu=rng.choice((3, 4, 10)), fold=rng.choice((1, 2, 4)),
                      clustered=Ng < 192 or rng.random() < 0.6)  # unclustered boxes are the larger checks
    if kind == "batch":
        return dict(kind="batch", Ng=rng.choice((64, 96, 128, 192, 256, 384)), Np=_log_int(rng, 5e4, 3e6),
                    ncat=rng.randint(3, 10), los=los, Nmu=rng.choice((3, 10)))
    if kind == "p2k":
        return dict(kind="p2k", Ng=rng.choice((32, 48, 64, 75, 96, 128, 160, 192)), Np=_log_int(rng, 2e4, 2e6),
                    clustered=rng.random() < 0.5)
    if kind == "window":
        Nsub = rng.choice((2, 4, 8))
        return dict(kind="window", Ng=Nsub * rng.choice((16, 24, 32, 40, 60, 64)), Nsub=Nsub)
    return dict(kind="train", n=_log_int(rng, 500, 60_000))


# ---- inputs -------------------------------------------------------------------

def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    return g


def _catalog(Np, clustered, seed, velocities=False):
    """FP32 positions [3, Np] in the box (and velocities): uniform, or galaxies
    listed halo by halo around uniform centres (about 30 to a halo, with a
    smooth 30 %), wrapped into the box."""
    gen = _gen(seed)
    x = torch.rand((3, Np), generator=gen, device="cuda", dtype=torch.float32) * L_BOX
    if clustered:
        nc = max(50, Np // 30)
        nh = (7 * Np) // 10
        cen = torch.rand((3, nc), generator=gen, device="cuda", dtype=torch.float32) * L_BOX
        which = torch.sort(torch.randint(nc, (nh,), generator=gen, device="cuda"))[0]
        off = torch.randn((3, nh), generator=gen, device="cuda", dtype=torch.float32)
        x[:, :nh] = torch.remainder(cen[:, which] + 1.5 * off, L_BOX)
    v = 3.0 * torch.randn((3, Np), generator=gen, device="cuda", dtype=torch.float32) if velocities else None
    return x, v


def _batch_sizes(case):
    """Uneven catalog sizes around Np (between 0.6 and 1.4 of it)."""
    return [int(case["Np"] * (0.6 + 0.8 * ((7 * c + 3) % 11) / 10.0)) for c in range(case["ncat"])]


def _spectrum_grid(case, seed):
    """|FFT|^2 of white noise on the half spectrum: a power grid as P() leaves
    it (imaginary parts 0), complex64 [Ng, Ng, Ng/2 + 1]."""
    Ng = case["Ng"]
    w = torch.randn((Ng, Ng, Ng), generator=_gen(seed), device="cuda", dtype=torch.float32)
    d = torch.fft.rfftn(w) * (L_BOX / Ng) ** 1.5
    p = (d.real ** 2 + d.imag ** 2) / Ng ** 1.5
    return torch.complex(p, torch.zeros_like(p)).contiguous()


def _train_data(case, seed):
    gen = _gen(seed)
    n = case["n"]
    u = torch.rand((n, 5), generator=gen, device="cuda", dtype=torch.float32)
    X = torch.stack([1.7 * u[:, 0], u[:, 1], 0.6 * (u[:, 2] - 0.5), 0.4 * (u[:, 3] - 0.5), 6.0 * u[:, 4] - 5.0], 1)
    T = torch.randn((n, 3), generator=gen, device="cuda", dtype=torch.float32).clamp(-5, 5)
    return X.contiguous(), T.contiguous()


def _grid(Ng, L, precision):
    g = fg.Grid(Ng, L, precision=precision, host_view="lazy")
    g.set_stream(torch.cuda.current_stream().cuda_stream)
    return g


def prepare(case, seed):
    kind = case["kind"]
    s = dict(case=case)
    if kind == "power":
        L = L_BOX / case["fold"]
        s["x"], s["v"] = _catalog(case["Np"], case["clustered"], seed, case["mode"] == "rsd")
        s["grid"] = _grid(case["Ng"], L, "f32")
        s["dK"] = 2 * math.pi / L
        s["params"] = alias_mlp.load() if case["mode"] == "learned" else None
    elif kind == "batch":
        s["cats"] = []
        for c, n in enumerate(_batch_sizes(case)):
            x, _ = _catalog(n, c % 2 == 0, 1000 * seed + c)
            h = torch.empty((3, n), dtype=torch.float32, pin_memory=True)
            h.copy_(x)
            s["cats"].append(tuple(h[a].numpy() for a in range(3)))
        s["grid"] = _grid(case["Ng"], L_BOX, "f32")
    elif kind == "p2k":
        x = _catalog(case["Np"], case["clustered"], seed)[0].double().cpu().numpy()
        s["cat"] = fg.Catalog(x[0], x[1], x[2], L_BOX ** 3)
        s["grid"] = _grid(case["Ng"], L_BOX, "f64")
        Ng = case["Ng"]
        s["out"] = torch.empty((Ng, Ng, Ng // 2 + 1), dtype=torch.complex128, device="cuda")
    elif kind == "window":
        s["field"] = _spectrum_grid(case, seed)
        s["grid"] = _grid(case["Ng"], L_BOX, "f32")
        s["out"] = torch.empty_like(s["field"])
    else:
        s["X"], s["T"] = _train_data(case, seed)
        s["trainer"] = alias_mlp.Trainer(alias_mlp.init_params(7))
    return s


# ---- one pass -------------------------------------------------------------------

def _tables(r):
    return dict(K=r["K"], N=r["N"], P=r["P"].astype(np.float32), Kmu=r["Kmu"], Nmu=r["Nmu"],
                Pmu=r["Pmu"].astype(np.float32))


def run(s):
    c = s["case"]
    kind, g = c["kind"], s.get("grid")
    V = L_BOX ** 3
    if kind == "power":
        p = [s["x"][a].data_ptr() for a in range(3)]
        los, dK = LOS[c["los"]], s["dK"]
        kw = dict(Nmu=c["Nmu"], where=fg.MEM_DEVICE, Np=c["Np"])
        if c["mode"] == "rsd":
            v = [s["v"][a].data_ptr() for a in range(3)]
            return _tables(g.power_rsd_f32(*p, *v, V, los, AH, dK, **kw))
        if c["mode"] == "learned":
            return _tables(g.power_learned_f32(*p, V, los, dK, s["params"], **kw))
        return _tables(g.power_f32(*p, V, los, dK, interlace=c["mode"] == "interlaced", **kw))
    if kind == "batch":
        return [_tables(r) for r in g.power_batch_f32(s["cats"], V, LOS[c["los"]], 2 * math.pi / L_BOX, Nmu=c["Nmu"])]
    if kind == "p2k":
        g.p2k(s["cat"])
        g.copy_to(s["out"].data_ptr())
        return s["out"]
    if kind == "window":
        g.copy_from(s["field"].data_ptr())
        g.k2x(0)
        g.window_box(c["Ng"] // c["Nsub"])
        g.x2k(0)
        g.copy_to(s["out"].data_ptr())
        return s["out"]
    t = s["trainer"]
    loss = t.step(s["X"], s["T"], 2e-3)
    return dict(grad=t.g, params=t.p, loss=loss)


# ---- what a pass cannot do without ----------------------------------------------

def _table_bytes(Ng, Nmu):
    NK = int(3 ** 0.5 * (Ng // 2)) + 1
    return NK * 8 * (6 + 3 * Nmu)


def _power_flops(Ng, Np, grids):
    # paint 64 multiply-adds per particle and grid, 2.5 n log2 n per real FFT, 40 per mode for the bins
    n = float(Ng) ** 3
    return grids * (Np * 190 + 2.5 * n * math.log2(n)) + 20 * n


def work(case):
    kind = case["kind"]
    if kind == "power":
        Ng, Np = case["Ng"], case["Np"]
        per = 24 if case["mode"] == "rsd" else 12
        return dict(bytes=per * Np + _table_bytes(Ng, case["Nmu"]),
                    flops=_power_flops(Ng, Np, 2 if case["mode"] in ("interlaced", "rsd") else 1))
    if kind == "batch":
        n = _batch_sizes(case)
        return dict(bytes=12 * sum(n) + len(n) * _table_bytes(case["Ng"], case["Nmu"]),
                    flops=sum(_power_flops(case["Ng"], q, 2) for q in n))
    if kind == "p2k":
        Ng, Np = case["Ng"], case["Np"]
        return dict(bytes=24 * Np + 16 * Ng * Ng * (Ng // 2 + 1), flops=_power_flops(Ng, Np, 2) - 20.0 * Ng ** 3)
    if kind == "window":
        Ng = case["Ng"]
        n = float(Ng) ** 3
        return dict(bytes=16 * Ng * Ng * (Ng // 2 + 1), flops=5 * n * math.log2(n) + 8 * n / case["Nsub"] ** 3)
    n = case["n"]
    return dict(bytes=32 * n + 16 * alias_mlp.NPARAMS * 2, flops=6.0 * alias_mlp.NPARAMS * n)


# ---- the answer in 64 bits --------------------------------------------------------

def _paint64(x, Ng, L, off):
    """PCS density of positions x [3, Np] (FP64) on a grid shifted by `off` cells."""
    grid = torch.zeros(Ng ** 3, dtype=torch.float64, device="cuda")
    Np = x.shape[1]
    for p0 in range(0, Np, 12_500_000):
        cell, w = [], []
        for a in range(3):
            u = x[a, p0:p0 + 12_500_000] * (Ng / L) - off
            b = torch.floor(u)
            d = u - b
            e = 1 - d
            d2 = d * d
            w.append([e * e * e / 6, ((3 * d - 6) * d2 + 4) / 6, (((-3 * d + 3) * d + 3) * d + 1) / 6, d2 * d / 6])
            b = b.long()
            cell.append([torch.remainder(b + t - 1, Ng) for t in range(4)])
        for i in range(4):
            for j in range(4):
                wij, cij = w[0][i] * w[1][j], (cell[0][i] * Ng + cell[1][j]) * Ng
                for k in range(4):
                    grid.index_add_(0, cij + cell[2][k], wij * w[2][k])
    return grid.view(Ng, Ng, Ng)


def _phase64(Ng):
    n = torch.arange(Ng, device="cuda", dtype=torch.float64)
    n = torch.where(2 * n < Ng, n, n - Ng)  # the Nyquist entry is the conjugate's
    a = -2 * math.pi * n / Ng * 0.5
    return torch.complex(torch.cos(a), torch.sin(a))


def _winv64(Ng):
    n = torch.arange(Ng, device="cuda", dtype=torch.float64)
    n = torch.minimum(n, Ng - n)
    a = math.pi * n / Ng
    r = torch.where(n > 0, a / torch.sin(torch.where(n > 0, a, torch.ones_like(a))), torch.ones_like(a))
    return r ** 4


def _field64(x, Ng, L, V, interlace):
    """The deconvolved k-space field [Ng, Ng, Ng/2 + 1]."""
    H3 = (L / Ng) ** 3
    scale = V / x.shape[1] / H3 * H3  # density contrast of the box times the cell volume
    d = torch.fft.rfftn(_paint64(x, Ng, L, 0.0))
    nh = Ng // 2 + 1
    if interlace:
        e = torch.fft.rfftn(_paint64(x, Ng, L, 0.5))
        ph = _phase64(Ng)
        e *= ph[:, None, None]
        e *= ph[None, :, None]
        e *= ph[None, None, :nh]
        d += e
        del e
        d *= 0.5
    w = _winv64(Ng)
    d *= w[:, None, None] * scale
    d *= w[None, :, None]
    d *= w[None, None, :nh]
    return d


def _bins64(d, Ng, L, V, Np, los, dK, Nmu):
    los = np.array(los, dtype=np.float64)
    los = los / math.sqrt(los[0] * los[0] + los[1] * los[1] + los[2] * los[2])
    KF = 2 * math.pi / L
    inv = KF / dK
    NK = int(math.floor(1.73205080756887729352744634151 * (Ng // 2) * inv)) + 1
    W = Nmu + 1
    nh = Ng // 2 + 1
    dev = d.device
    n1 = torch.arange(Ng, device=dev, dtype=torch.float64)
    n1 = torch.where(2 * n1 < Ng, n1, n1 - Ng)
    n3 = n1[:nh]
    k3 = torch.arange(nh, device=dev)
    cnt3 = 1.0 + ((2 * k3) % Ng > 0).double()
    acc = torch.zeros((5, NK), device=dev, dtype=torch.float64)  # N is summed with the wedges
    wed = torch.zeros((3, NK * W), device=dev, dtype=torch.float64)
    step = max(1, (1 << 24) // (Ng * nh))
    for i0 in range(0, Ng, step):
        ki = n1[i0:i0 + step, None, None]
        kj, kk = n1[None, :, None], n3[None, None, :]
        amp = torch.sqrt(ki * ki + kj * kj + kk * kk)
        num = (ki * los[0] + kj * los[1]) + kk * los[2]
        if i0 == 0:
            amp[0, 0, 0] = 1.0
        mu = num / amp
        b = torch.floor(amp * inv).long()
        m = torch.floor(torch.abs(mu * Nmu)).long()
        f = d[i0:i0 + step]
        c = cnt3.expand(b.shape).clone()
        if i0 == 0:
            c[0, 0, 0] = 0.0
        p = ((f.real ** 2 + f.imag ** 2) / V - V / Np) * c
        ok = c.reshape(-1) > 0
        b, m, p, c, amp = (t.reshape(-1)[ok] for t in (b, m, p, c, amp))
        m2 = (mu * mu).reshape(-1)[ok]
        leg = (None, 1.5 * m2 - 0.5, (4.375 * m2 - 3.75) * m2 + 0.375,
               ((14.4375 * m2 - 19.6875) * m2 + 6.5625) * m2 - 0.3125)
        for q in range(4):
            acc[q] += torch.bincount(b, p if q == 0 else p * leg[q], NK)
        key = b * W + m
        for q, t in enumerate((p, c, c * amp)):
            wed[q] += torch.bincount(key, t, NK * W)
    acc, wed = acc.cpu().numpy(), wed.cpu().numpy().reshape(3, NK, W)
    with np.errstate(all="ignore"):
        Nf, Ks = wed[1].sum(1), wed[2].sum(1)
        N = np.round(Nf).astype(np.int64)
        K = Ks * (KF / Nf)
        P = np.stack([acc[q] * ((4 * q + 1.0) / Nf) for q in range(4)], 1)
        wed[:, :, Nmu - 1] += wed[:, :, Nmu]
        Pw, Nw, Kw = wed[0][:, :Nmu], wed[1][:, :Nmu], wed[2][:, :Nmu]
        has = Nw > 0
        Kmu = np.where(has, Kw * (KF / np.where(has, Nw, 1.0)), Kw)
        Pmu = np.where(has, Pw / np.where(has, Nw, 1.0), Pw)
    return dict(K=K, N=N, P=P, Kmu=Kmu, Nmu=np.round(Nw).astype(np.int64), Pmu=Pmu)


def _perceptron64(params, X):
    """Outputs and hidden activations of the 5-64-64-64-3 perceptron."""
    p = torch.as_tensor(np.asarray(params, dtype=np.float64), device="cuda")
    o, w, b = 0, [], []
    for a, z in ((5, 64), (64, 64), (64, 64), (64, 3)):
        w.append(p[o:o + a * z].view(a, z))
        b.append(p[o + a * z:o + a * z + z])
        o += a * z + z
    act = [X]
    for q in range(4):
        z = act[-1] @ w[q] + b[q]
        act.append(torch.tanh(z) if q < 3 else z)
    return w, act


def _learned64(r, Pshot, kNyq, params):
    K, P = r["K"], r["P"].copy()
    with np.errstate(all="ignore"):
        den = np.abs(P[:, 0]) + Pshot
        ok = np.isfinite(P[:, 0]) & np.isfinite(K) & (K > 0) & (den > 0)
        at = np.flatnonzero(ok)
        X = np.zeros((len(K), 5))
        lden, lk = np.log(den), np.log(K)
        for q, b in enumerate(at):
            lo, hi = at[max(q - 1, 0)], at[min(q + 1, len(at) - 1)]
            s = (lden[hi] - lden[lo]) / (lk[hi] - lk[lo]) if hi != lo and lk[hi] != lk[lo] else 0.0
            X[b] = K[b] / kNyq, Pshot / den[b], P[b, 1] / den[b], P[b, 2] / den[b], min(5.0, max(-5.0, s))
        y = _perceptron64(params, torch.as_tensor(X, device="cuda"))[1][-1].cpu().numpy()
        u6 = (K / kNyq) ** 6
        fix = np.isfinite(P[:, 0]) & (r["N"] > 0)
        P[fix, :3] += (den * (u6 / (1 + u6)))[fix, None] * y[fix]
    return dict(r, P=P)


def exact(case, seed):
    kind = case["kind"]
    V = L_BOX ** 3
    if kind == "power":
        Ng, Np, L = case["Ng"], case["Np"], L_BOX / case["fold"]
        x, v = _catalog(Np, case["clustered"], seed, case["mode"] == "rsd")
        x = x.double()
        los = LOS[case["los"]]
        if v is not None:
            h = torch.tensor(los, device="cuda", dtype=torch.float64)
            h = h / h.norm()
            x = x + h[:, None] * ((h[:, None] * v.double()).sum(0) / AH)
            del v
        d = _field64(x, Ng, L, V, case["mode"] in ("interlaced", "rsd"))
        del x
        r = _bins64(d, Ng, L, V, Np, los, 2 * math.pi / L, case["Nmu"])
        return _learned64(r, V / Np, math.pi * Ng / L, alias_mlp.load()) if case["mode"] == "learned" else r
    if kind == "batch":
        out = []
        for c, n in enumerate(_batch_sizes(case)):
            x, _ = _catalog(n, c % 2 == 0, 1000 * seed + c)
            d = _field64(x.double(), case["Ng"], L_BOX, V, True)
            out.append(_bins64(d, case["Ng"], L_BOX, V, n, LOS[case["los"]], 2 * math.pi / L_BOX, case["Nmu"]))
        return out
    if kind == "p2k":
        return _field64(_catalog(case["Np"], case["clustered"], seed)[0].double(), case["Ng"], L_BOX, V, True)
    if kind == "window":
        Ng = case["Ng"]
        xi = torch.fft.irfftn(_spectrum_grid(case, seed).to(torch.complex128), s=(Ng, Ng, Ng)) * (Ng / L_BOX) ** 3
        ns = Ng // case["Nsub"]
        n = torch.arange(Ng, device="cuda", dtype=torch.float64)
        n = torch.minimum(n, Ng - n)
        f = torch.where(n < ns, ns / torch.where(n < ns, ns - n, torch.ones_like(n)), torch.zeros_like(n))
        inside = (n < ns)
        box = f[:, None, None] * f[None, :, None] * f[None, None, :]
        both = inside[:, None, None] & inside[None, :, None] & inside[None, None, :]
        return torch.fft.rfftn(torch.where(both, xi * box, xi)) * (L_BOX / Ng) ** 3
    X, T = (t.double() for t in _train_data(case, seed))
    w, act = _perceptron64(alias_mlp.init_params(7), X)
    r = act[-1] - T
    loss = (r * r).sum() / X.shape[0]
    dl, parts = 2 * r / X.shape[0], []
    for q in (3, 2, 1, 0):
        parts.append(torch.cat([(act[q].T @ dl).reshape(-1), dl.sum(0)]))
        if q:
            dl = (dl @ w[q].T) * (1 - act[q] ** 2)
    grad = torch.cat(parts[::-1])
    p = torch.as_tensor(np.asarray(alias_mlp.init_params(7), dtype=np.float64), device="cuda")
    # the first Adam step: m / (1 - beta1) = g, v / (1 - beta2) = g^2
    return dict(grad=grad, params=p - 2e-3 * grad / (grad.abs() + 1e-8), loss=float(loss))
