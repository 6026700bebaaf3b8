"""The perceptron's forward pass (csrc/mlp.cu) over many samples, where a warp takes
four at a time: sample counts around the rule's line (four samples for each warp of
a full grid) and with one to three samples left over, against the FP64 restatement
oracle/mlp.py (1e-5, as the other forward tests) and bit for bit against the same
samples in a short call.  And its time: the forward pass has a third of the
gradient's multiply-adds, so half of the gradient's time is a bound with room (7e5
samples: 0.45 of 1.62 ms; 1.31 with one sample per warp)."""
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


@pytest.mark.parametrize("extra", [-1, 0, 1, 2, 3, 10_006])
def test_forward_many(fg, extra):
    import torch
    from fftgal_gb300 import alias_mlp as a
    n = 64 * torch.cuda.get_device_properties(0).multi_processor_count + extra
    p = a.init_params(3)
    X = np.random.default_rng(n).standard_normal((n, a.IN)).astype(np.float32)
    y = a.forward_gpu(p, X)
    y64, _ = mlp_ref.forward(p, X.astype(np.float64))
    assert np.abs(y - y64).max() <= 1e-5 * max(1.0, np.abs(y64).max())
    np.testing.assert_array_equal(y[:777], a.forward_gpu(p, X[:777]))
    np.testing.assert_array_equal(y[-777:], a.forward_gpu(p, X[-777:]))


def test_forward_is_cheaper_than_the_gradient(fg):
    import torch
    from fftgal_gb300 import alias_mlp as a
    n = 700_000
    p = torch.tensor(a.init_params(3), device="cuda")
    X, T, Y = torch.rand((n, a.IN), device="cuda"), torch.rand((n, a.OUT), device="cuda"), torch.zeros(
        (n, a.OUT), device="cuda")
    g, loss = torch.zeros(len(p), device="cuda"), torch.zeros(1, device="cuda")
    st = torch.cuda.current_stream().cuda_stream
    calls = dict(
        forward=lambda: fg.lib().fftgal_mlp_forward(p.data_ptr(), X.data_ptr(), n, Y.data_ptr(), st),
        gradient=lambda: fg.lib().fftgal_mlp_grad(p.data_ptr(), X.data_ptr(), T.data_ptr(), n, g.data_ptr(),
                                                  loss.data_ptr(), st))
    t = {}
    for name, call in calls.items():
        runs = []
        for _ in range(6):
            e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            e0.record()
            assert call() == 0
            e1.record()
            torch.cuda.synchronize()
            runs.append(e0.elapsed_time(e1))
        t[name] = min(runs)
    assert t["forward"] <= 0.5 * t["gradient"], t
