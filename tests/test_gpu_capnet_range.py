"""The FP32 network where an activation's argument is as far below zero as FP32
goes: the SiLU and its derivative are 0 there, in every kernel that takes them."""
import numpy as np
import pytest

from gpucode_gb300.capnet import CapNet
from test_gpu_capnet import _t, mo

pytestmark = pytest.mark.gpu

NORM = np.array([0] * 4 + [1] * 4 + [0] * 2 + [1] * 2 + [-9] * 4 + [9] * 4, np.float32)


def _net(layer, rows):
    """unit 0 of the given layer has a large negative argument times feature 2; the
    sign after it turns what is left of the unit into a positive output.  rows: a
    weight too small for the BF16 pieces, so that the row kernel takes the network"""
    p = np.zeros(4610, np.float32)
    w1, w2, w3 = p[:256].reshape(64, 4), p[320:4416].reshape(64, 64), p[4480:4608].reshape(2, 64)
    if layer == 1:
        w1[0, 2] = -3.399e38
        w2[:, 0] = -1.0
    else:
        w1[0, 2] = 1e20
        w2[:, 0] = -1e15
    w3[0], w3[1] = -1.0 / 64, 1.0 / 64
    if rows:
        w2[3, 5] = 1e-36
    return p


def _features(n):
    x = np.ones((n, 4), np.float32)
    x[:, 2] = np.float32(10.0) ** np.linspace(-38, 0, n).astype(np.float32)
    return x


@pytest.mark.parametrize("rows", [False, True])
@pytest.mark.parametrize("layer", [1, 2])
def test_far_negative_activations_are_zero(cuda, layer, rows):
    """arguments from -3.4 to -3.4e38 (layer 1) and from 0 to -1e35 (layer 2);
    where the argument is of order one, 66 FP32 roundings of like terms: 1e-5"""
    x, p = _features(300), _net(layer, rows)
    net = CapNet(seed=0)
    net.set(p, NORM)
    y = net.infer(_t(x), tensor_cores=False).cpu().numpy()
    net.close()
    with np.errstate(over="ignore"):
        want, _ = mo.forward(p.astype(np.float64), mo.std_inputs(x, NORM.astype(np.float64)))
    np.testing.assert_allclose(y, want, rtol=1e-5, atol=1e-6)
    assert (y[x[:, 2] > 1e-30] == 0).all()


def test_gradient_of_far_negative_activations_is_zero(cuda):
    """the derivative of the SiLU at arguments to -3.4e38, against the FP64
    oracle's; tolerances of the other gradient tests"""
    x, p = _features(300)[150:], _net(1, False)
    y = np.tile(np.array([1, -1], np.float32), (len(x), 1))  # the two errors add up at layer 1
    net = CapNet(seed=0)
    net.set(p, NORM)
    g, loss = net.grad(_t(x), _t(y))
    net.close()
    with np.errstate(over="ignore"):
        lo, go = mo.loss_and_grad(p.astype(np.float64), x, y, NORM.astype(np.float64))
    assert abs(loss - lo) <= 1e-5 * lo
    assert np.abs(g - go).max() < 1e-4 * np.abs(go).max()
