"""GPU test of the warm-start network at layer sizes and batches that fill no
tile: rows that need padding to 16 bytes, one value per layer side of a tile
edge, batches around the 128-row tile and the 256-row column sums.

Against oracle/mlp_oracle.py, which rounds to BF16 at the same points: the two
activations, the output's gradient and the two gradients passed back.  A value
on the other side of a rounding tie differs by 2^-8 of itself, so that even if
every value fell on the other side the output would stay within 2 x 2^-8 of its
norm, the squared error within 4 x 2^-8 and the gradient within 5 x 2^-8."""
import numpy as np
import pytest

import rootpwa_gb300 as R
from oracle import mlp_oracle as MO
import helpers

pytestmark = pytest.mark.gpu

TIE = 2.0 ** -8


@pytest.mark.parametrize("shape", [(9, 7, 5, 3), (1, 16, 8, 1), (127, 129, 131, 130), (65, 513, 40, 12)])
@pytest.mark.parametrize("B", [1, 129, 257, 512])
def test_shapes_that_fill_no_tile(shape, B):
    rng = np.random.default_rng(sum(shape) + B)
    net = R.pwaMLP(*shape, seed=3)
    p = net.params()
    # biases are zero at first: give them values
    p = (p + 0.1 * rng.standard_normal(p.size)).astype(np.float32)
    net.setParams(p)
    X = rng.standard_normal((B, shape[0])).astype(np.float32)
    T = rng.standard_normal((B, shape[3])).astype(np.float32)
    loss, g = net.gradient(X, T)
    l0, g0 = MO.loss_and_gradient(p, shape, X, T)
    assert abs(loss - l0) <= 4 * TIE * max(l0, np.mean(T * T))
    assert helpers.normwise(g, g0) <= 5 * TIE
    Y, Y0 = net.forward(X), MO.forward(p, shape, X)
    assert np.linalg.norm(Y - Y0) <= 2 * TIE * np.linalg.norm(Y0)
    # one training step over the whole batch reports the same error (the rows
    # come in another order: FP64 sums of the same terms)
    assert abs(net.train(X, T, batch=B, epochs=1)[0] - loss) <= 1e-10 * loss
