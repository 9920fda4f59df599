"""The closure network's kernels at the edges of their tiles and of the rules
that choose between them: training blocks of 64 samples (several tiles a block
beyond 152 x 64), the FP32 network with one row a thread below 100,000 rows and
two from there on, 16- and 128-row tensor-core tiles."""
import numpy as np
import pytest

from gpucode_gb300.capnet import CapNet
from test_gpu_capnet import _random_features, _t, mo

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 63, 64, 65, 152 * 64, 152 * 64 + 1, 30_001])
def test_gradient_at_tile_edges(cuda, n):
    """against the FP64 oracle, to the tolerances of the 700-sample test"""
    x, y, norm = _random_features(np.random.default_rng(n), max(n, 16))
    x, y = x[:n], y[:n]
    net = CapNet(seed=5)
    net.set(norm=norm)
    p, _ = net.get()
    g, loss = net.grad(_t(x), _t(y))
    lo, go = mo.loss_and_grad(p.astype(np.float64), x, y, norm.astype(np.float64))
    assert abs(loss - lo) <= 1e-5 * lo
    assert np.abs(g - go).max() < 1e-4 * np.abs(go).max()
    net.close()


@pytest.mark.parametrize("n", [1, 127, 128, 129, 99_999, 100_000, 100_257])
def test_inference_at_tile_edges(cuda, n):
    """FP32 against the oracle (both row counts a thread), and each row the same
    whatever rows come with it on the tensor-core paths"""
    x, y, norm = _random_features(np.random.default_rng(7), 100_257)
    net = CapNet(seed=6)
    p = mo.init_params(9).astype(np.float32)
    net.set(p, norm)
    want, _ = mo.forward(p.astype(np.float64), mo.std_inputs(x[:n], norm.astype(np.float64)))
    got = net.infer(_t(x[:n]), tensor_cores=False).cpu().numpy()
    assert np.abs((got - norm[8:10]) / norm[10:12] - want).max() < 1e-4
    for mode in ("warp", "tcgen05"):
        whole = net.infer(_t(x), tensor_cores=mode).cpu().numpy()
        np.testing.assert_array_equal(net.infer(_t(x[:n]), tensor_cores=mode).cpu().numpy(), whole[:n])
    net.close()


def test_parameters_set_after_an_inference_are_used(cuda):
    """every path reads the parameters of the last set()"""
    x, _, norm = _random_features(np.random.default_rng(8), 300)
    net = CapNet(seed=6)
    net.set(norm=norm)
    first = {m: net.infer(_t(x), tensor_cores=m).cpu().numpy() for m in (False, "warp", "tcgen05")}
    net.set(params=mo.init_params(2).astype(np.float32))
    fresh = CapNet(seed=1)
    fresh.set(mo.init_params(2).astype(np.float32), norm)
    for m, a in first.items():
        b = net.infer(_t(x), tensor_cores=m).cpu().numpy()
        assert not np.array_equal(a, b)
        np.testing.assert_array_equal(b, fresh.infer(_t(x), tensor_cores=m).cpu().numpy())
    net.close()
    fresh.close()
