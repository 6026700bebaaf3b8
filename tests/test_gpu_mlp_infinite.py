"""The perceptron's gradient (csrc/mlp.cu) with weights of the first layer that are
infinite: they saturate their units, as 1e30 does, and the gradient is finite.  The
samples that fill up the last tile of 32 must not change that.  The saturated units'
values are the same in both, so the results agree to the roundings of a sum in
another order of atomics: 1e-5 of the gradient's norm."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def fg():
    from fftgal_gb300 import build
    build.build()
    import fftgal_gb300
    return fftgal_gb300


@pytest.mark.parametrize("n", [1, 31, 32, 33, 500])
def test_infinite_first_layer(fg, n):
    import torch
    from fftgal_gb300 import alias_mlp as a
    rng = np.random.default_rng(n)
    X = torch.tensor(rng.uniform(0.1, 1.0, (n, a.IN)).astype(np.float32), device="cuda")
    T = torch.tensor(rng.standard_normal((n, a.OUT)).astype(np.float32), device="cuda")
    out = []
    for big in (1e30, np.inf):
        p = a.init_params(5)
        w = a.LAYOUT["W1"][0]
        p[w + 3], p[w + 64 + 17] = big, -big
        d = torch.tensor(p, device="cuda")
        g, loss = torch.zeros(len(p), device="cuda"), torch.zeros(1, device="cuda")
        torch.cuda.synchronize()
        st = fg.lib().fftgal_mlp_grad(d.data_ptr(), X.data_ptr(), T.data_ptr(), n, g.data_ptr(), loss.data_ptr(), None)
        assert st == 0, fg.lib().fftgal_last_error()
        torch.cuda.synchronize()
        out.append((g.cpu().numpy().astype(np.float64), float(loss)))
    assert np.isfinite(out[1][0]).all()
    assert np.linalg.norm(out[1][0] - out[0][0]) <= 1e-5 * np.linalg.norm(out[0][0])
    assert abs(out[1][1] - out[0][1]) <= 1e-5 * out[0][1]
