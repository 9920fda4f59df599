"""The closure network's kernels at the edges of their tiles and of the rules
that choose between them: training blocks of 64 samples (several tiles a block
beyond 152 x 64), 16- and 128-row tensor-core tiles, the FP32 network's wide
layer in BF16 pieces and the rows and weights that those cannot hold."""
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
    """FP32 against the oracle, and each row the same
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


@pytest.mark.parametrize("n", [1, 128, 129, 4 * 152 * 128 + 1])
def test_fp32_network_in_three_pieces(cuda, n):
    """the wide layer as products of BF16 pieces: FP32's accuracy.  A dot product
    of 64 in FP32 is within 64 x 2^-24 of sum |w h|; with the random network's
    |w| < 1 and activations below 4 that is 64 x 64 x 4 x 2^-24 = 1e-3 at the very
    worst and two orders less for signs that mix: 1e-5"""
    x, _, norm = _random_features(np.random.default_rng(11), max(n, 16))
    x = x[:n]
    net = CapNet(seed=6)
    p = mo.init_params(9).astype(np.float32)
    net.set(p, norm)
    want, _ = mo.forward(p.astype(np.float64), mo.std_inputs(x, norm.astype(np.float64)))
    got = net.infer(_t(x), tensor_cores=False).cpu().numpy()
    assert np.abs((got - norm[8:10]) / norm[10:12] - want).max() < 1e-5
    net.close()


@pytest.mark.parametrize("tiny", [1e-30, 1e-36])
def test_fp32_network_beyond_the_pieces_range(cuda, tiny):
    """activations above the largest BF16 number (3.3895e38) and infinite ones,
    among ordinary rows, and weights whose pieces are subnormal (1e-36): the FP32
    result, not what is left of the pieces"""
    p = np.zeros(4610, np.float32)
    w1, w2, w3 = p[:256].reshape(64, 4), p[320:4416].reshape(64, 64), p[4480:4608].reshape(2, 64)
    w1[0, 2] = 3.399e38  # unit 0 = silu(3.399e38 x2)
    w2[:, 0] = tiny
    w3[0] = 1.0 / 64
    w3[1] = -1.0 / 64
    norm = np.array([0] * 4 + [1] * 4 + [0] * 2 + [1] * 2 + [-9] * 4 + [9] * 4, np.float32)
    x = np.ones((300, 4), np.float32)
    x[:, 2] = 0.5
    x[7, 2] = 1.0    # finite in FP32, infinite in BF16
    x[200, 2] = 2.0  # infinite in FP32 as well
    x[201, 2] = np.nan
    net = CapNet(seed=6)
    net.set(p, norm)
    y = net.infer(_t(x), tensor_cores=False).cpu().numpy()
    z = float(w1[0, 2]) * float(w2[0, 0]) * np.array([0.5, 1.0])  # above 100: silu(z) = z
    rest = np.delete(np.arange(300), [7, 200, 201])
    # a dozen FP32 roundings and 64 equal terms: below 2^-20
    np.testing.assert_allclose(y[rest, 0], z[0], rtol=1e-6)
    np.testing.assert_allclose(y[7], [z[1], -z[1]], rtol=1e-6)
    assert np.isposinf(y[200, 0]) and np.isneginf(y[200, 1])
    assert np.isnan(y[201]).all()
    net.close()
