"""Perceptron kernels (csrc/mlp.cu) where their tiles end: sample counts below, at
and above a warp and a tile of samples, several tiles per CTA, and a gradient
that is not 16-byte aligned, against the FP64 restatement oracle/mlp.py.
Tolerances: those of the kernels' other tests (1e-4 of the gradient's norm, 1e-5
of the loss and of the outputs)."""
import numpy as np
import pytest

from oracle import mlp as mlp_ref

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def fg():
    from fftgal_gb300 import build
    build.build()
    import fftgal_gb300
    return fftgal_gb300


def _data(n):
    from fftgal_gb300 import alias_mlp as a
    rng = np.random.default_rng(n)
    p = a.init_params(n)
    p[a.LAYOUT["W4"][0]:a.LAYOUT["W4"][0] + a.LAYOUT["W4"][1]] *= 10
    return p, rng.standard_normal((n, a.IN)).astype(np.float32), rng.standard_normal((n, a.OUT)).astype(np.float32)


@pytest.mark.parametrize("off", [0, 1])
@pytest.mark.parametrize("n", [1, 2, 31, 32, 33, 63, 65, 127, 129, 4864, 10007])
def test_gradient(fg, n, off):
    import torch
    p, X, T = _data(n)
    d = [torch.tensor(v, device="cuda") for v in (p, X, T)]
    buf = torch.zeros(len(p) + 8, device="cuda")
    loss = torch.zeros(1, device="cuda")
    torch.cuda.synchronize()
    st = fg.lib().fftgal_mlp_grad(d[0].data_ptr(), d[1].data_ptr(), d[2].data_ptr(), n, buf.data_ptr() + 4 * off,
                                  loss.data_ptr(), None)
    assert st == 0, fg.lib().fftgal_last_error()
    torch.cuda.synchronize()
    g = buf.cpu().numpy().astype(np.float64)
    g64, loss64 = mlp_ref.grad(p, X, T)
    assert abs(float(loss) - loss64) <= 1e-5 * loss64
    assert np.linalg.norm(g[off:off + len(p)] - g64) <= 1e-4 * np.linalg.norm(g64)
    assert not g[:off].any() and not g[off + len(p):].any()


@pytest.mark.parametrize("n", [1, 7, 8, 9, 33, 10007])
def test_forward(fg, n):
    from fftgal_gb300 import alias_mlp as a
    p, X, _ = _data(n)
    y = a.forward_gpu(p, X)
    y64, _ = mlp_ref.forward(p, X.astype(np.float64))
    assert np.abs(y - y64).max() <= 1e-5 * max(1.0, np.abs(y64).max())
