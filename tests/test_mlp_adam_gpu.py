"""GPU: one Adam step of the warm-start network moves every parameter, at
parameter counts that leave 0 to 3 of them for the last, partly filled group of
four; the gradient is the network's own.

First step: m = (1 - b1) g, v = (1 - b2) g^2, so that the update is
lr (m / c1) / (sqrt(v / c2) + eps) with c1 = 1 - b1, c2 = 1 - b2.  About ten FP32
roundings of the update and one of the parameter: 16 x 2^-24 lr + 2^-24 |w|."""
import numpy as np
import pytest

import rootpwa_gb300 as R

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(9, 7, 5, 3), (1, 16, 8, 1), (2, 3, 2, 2), (3, 1, 1, 3), (1, 1, 1, 1), (33, 17, 9, 6)])
def test_one_step(shape):
    i, h, k, o = shape
    n = i * h + h + h * k + k + k * o + o
    rng = np.random.default_rng(n)
    net = R.pwaMLP(*shape, seed=5)
    p = (net.params() + 0.3 * rng.standard_normal(n)).astype(np.float32)
    net.setParams(p)
    X = rng.standard_normal((1, i)).astype(np.float32)
    T = rng.standard_normal((1, o)).astype(np.float32)
    _, g = net.gradient(X, T)
    lr = np.float32(0.01)
    net.train(X, T, batch=1, epochs=1, lr=float(lr))
    q = net.params().astype(np.float64)
    one, b1, b2 = np.float32(1), np.float32(0.9), np.float32(0.999)
    g = np.asarray(g, dtype=np.float64)
    m, v = float(one - b1) * g, float(one - b2) * g * g
    step = float(lr) * (m / float(one - b1)) / (np.sqrt(v / float(one - b2)) + float(np.float32(1e-8)))
    assert np.all(np.abs(q - (p - step)) <= 2.0 ** -24 * (16 * lr + np.abs(p)))
    assert np.any(step != 0) and np.any(step[-4:] != 0)
    # a second net with the new parameters computes the same output: the BF16
    # copy of the weights was refreshed with them
    other = R.pwaMLP(*shape, seed=6)
    other.setParams(net.params())
    assert np.array_equal(net.forward(X), other.forward(X))
