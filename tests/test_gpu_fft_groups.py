"""FP32 FFT lengths that csrc/fft3.cu cuts into three groups of radix passes, whose
middle group goes from shared memory to shared memory: through a second buffer (245,
320, 384, 448: more tasks than a CTA's threads) and in place behind its own barrier
(1000, four columns per CTA); forward and backward against torch in FP64, and both
interlacing grids of one launch against the FP64 kernels.  (Lengths of a single group,
such as 13, 22 and 30, run the general kernels of csrc/fft.cu.)

Also the backward k pass of long power-of-two rows: 1024 = 32 x 16 packed pairs by
a whole grid with its row padding, 2048 = 32 x 32, two rows per CTA, by the rows of a
field of three plane waves along i and j.

Tolerance: the FP32 bound of the grids' other FFT tests, 2e-6 of the largest value;
the interlaced field 2e-5 of its largest, the stated tolerance of FP32 grids."""
import math

import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def fg():
    from fftgal_gb300 import build
    build.build()
    import fftgal_gb300
    return fftgal_gb300


@pytest.fixture(autouse=True)
def release():
    import torch
    yield
    torch.cuda.empty_cache()


def _gen(seed):
    import torch
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    return gen


@pytest.mark.parametrize("Ng", [245, 320, 384, 448, 1000])
def test_three_groups(fg, Ng):
    import torch
    L, nh = 30.0, Ng // 2 + 1
    g = fg.Grid(Ng, L, precision="f32", host_view="lazy")
    x = torch.randn((Ng, Ng, 2 * nh), generator=_gen(Ng), device="cuda")
    want = torch.fft.rfftn(x[..., :Ng].double()) * (L / Ng) ** 3
    torch.cuda.synchronize()
    g.copy_from(x.data_ptr())
    g.x2k(0)
    g.copy_to(x.data_ptr())
    g.synchronize()
    got = torch.view_as_complex(x.view(Ng, Ng, nh, 2))
    top = want.abs().max()
    assert max((got[i].to(want.dtype) - want[i]).abs().max() for i in range(Ng)) <= 2e-6 * top
    del got, want
    f = torch.randn((Ng, Ng, nh, 2), generator=_gen(Ng + 1), device="cuda")
    z = torch.view_as_complex(f.double())
    z = torch.fft.ifft(torch.fft.ifft(z, dim=0), dim=1)
    z[:, :, 0].imag.zero_()
    if Ng % 2 == 0:
        z[:, :, -1].imag.zero_()
    want = torch.fft.irfft(z, n=Ng, dim=2) * (Ng / L) ** 3
    del z
    torch.cuda.synchronize()
    g.copy_from(f.data_ptr())
    g.k2x(0)
    g.copy_to(f.data_ptr())
    g.synchronize()
    got = f.view(Ng, Ng, 2 * nh)[..., :Ng]
    top = want.abs().max()
    assert max((got[i].double() - want[i]).abs().max() for i in range(Ng)) <= 2e-6 * top


@pytest.mark.parametrize("Ng", [245, 320, 448])
def test_both_grids(fg, Ng):
    import torch
    L = 100.0
    p = torch.rand((3, 100_000), generator=_gen(Ng), device="cuda").double() * L
    p[:, ::2] = 31.0 + 0.4 * torch.randn((3, 50_000), generator=_gen(1), device="cuda").double()
    p = p.float().double().cpu().numpy()
    cat = fg.Catalog(*p, L ** 3)
    field = []
    for prec, dtype in (("f32", torch.float32), ("f64", torch.float64)):
        g = fg.Grid(Ng, L, precision=prec, host_view="lazy")
        g.p2k(cat)
        t = torch.empty((Ng, Ng, 2 * (Ng // 2 + 1)), dtype=dtype, device="cuda")
        g.copy_to(t.data_ptr())
        g.synchronize()
        field.append(t.double())
    assert (field[0] - field[1]).abs().max() <= 2e-5 * field[1].abs().max()


def test_backward_1024(fg):
    import torch
    Ng, L, nh = 1024, 30.0, 513
    f = torch.randn((Ng, Ng, nh, 2), generator=_gen(Ng), device="cuda")
    z = torch.fft.ifft(torch.view_as_complex(f.double()), dim=0)
    z = torch.fft.ifft(z, dim=1)
    pad = z[:, :, -1].clone() * (Ng ** 2 / L ** 3)  # the transformed Nyquist column stays in the row padding
    z[:, :, 0].imag.zero_()
    z[:, :, -1].imag.zero_()
    want = torch.fft.irfft(z, n=Ng, dim=2) * (Ng / L) ** 3
    del z
    g = fg.Grid(Ng, L, precision="f32", host_view="lazy")
    torch.cuda.synchronize()
    g.copy_from(f.data_ptr())
    g.k2x(0)
    g.copy_to(f.data_ptr())
    g.synchronize()
    got = f.view(Ng, Ng, 2 * nh)
    top = want.abs().max()
    assert max((got[i, :, :Ng].double() - want[i]).abs().max() for i in range(Ng)) <= 2e-6 * top
    end = torch.view_as_complex(got[:, :, Ng:].double().contiguous())
    assert (end - pad).abs().max() <= 2e-6 * pad.abs().max()


def test_backward_2048(fg):
    import torch
    Ng, L, nh = 2048, 30.0, 1025
    waves = [(0, 0), (1, 2045), (1024, 7)]
    F = torch.randn((3, nh, 2), generator=_gen(Ng), device="cuda")
    g = fg.Grid(Ng, L, precision="f32", host_view="lazy")
    f = torch.zeros((Ng, Ng, nh, 2), device="cuda")  # 34 GB
    for q, (a, b) in enumerate(waves):
        f[a, b] = F[q]
    torch.cuda.synchronize()
    g.copy_from(f.data_ptr())
    g.k2x(0)
    g.copy_to(f.data_ptr())
    g.synchronize()
    del g
    Z = torch.view_as_complex(F.double())
    y = torch.arange(Ng, device="cuda", dtype=torch.float64)
    err = err_pad = top = top_pad = 0.0
    for x in [0, 1, 2, 3, 511, 1023, 1024, 1025, 2046, 2047] + list(range(37, 2048, 97)):
        S = 0
        for q, (a, b) in enumerate(waves):
            turn = torch.remainder(a * x + b * y, Ng) * (2 * math.pi / Ng)
            S = S + torch.polar(torch.ones_like(turn), turn)[:, None] * Z[q] / L ** 3
        pad = S[:, -1].clone()
        S[:, 0].imag.zero_()
        S[:, -1].imag.zero_()
        want = torch.fft.irfft(S, n=Ng, dim=1) * Ng
        got = f[x].reshape(Ng, 2 * nh).double()
        err = max(err, float((got[:, :Ng] - want).abs().max()))
        err_pad = max(err_pad, float((torch.view_as_complex(got[:, Ng:].contiguous()) - pad).abs().max()))
        top, top_pad = max(top, float(want.abs().max())), max(top_pad, float(pad.abs().max()))
    assert err <= 2e-6 * top
    assert err_pad <= 2e-6 * top_pad
