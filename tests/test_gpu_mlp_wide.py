"""Training of networks wider than the fused kernels take (2,048): a GEMM per layer.
The first Adam step moves a parameter by lr g / (|g| + eps), so with |g| > 1e-4 it
has to be lr sign(g) to 1e-3 of lr (eps = 1e-8 leaves 1e-4, the moments' rounding
in FP32 a few 1e-7) and the rounding of the parameter; and training lowers the
loss, which is the gradient call's at the final parameters."""
import numpy as np
import pytest

from conftest import pkg

pytestmark = pytest.mark.gpu


def test_training_of_a_wide_network():
    cs = pkg()
    rng = np.random.default_rng(7)
    X = rng.uniform(-2, 3, (96, 4)).astype(np.float32)
    Y = np.sin(X @ rng.standard_normal((4, 6))).astype(np.float32)
    net = cs.warmstart.Mlp(4, 6, width=2112, depth=3, seed=11)
    net.fit_normalization(X, Y)
    w0, (l0, g) = net.params(), net.gradient(X, Y)
    net.train(X, Y, epochs=1, batch=96, lr=1e-4)
    step, big = net.params().astype(float) - w0, np.abs(g) > 1e-4
    assert big.sum() > 1000
    np.testing.assert_array_less(np.abs(step + 1e-4 * np.sign(g))[big], 1e-7 + 2.0**-23 * np.abs(w0[big]) + 1e-12)
    last = net.train(X, Y, epochs=40, batch=96, lr=1e-4)
    l1, _ = net.gradient(X, Y)
    assert abs(last - l1) <= 1e-4 * l1 and l1 < 0.5 * l0
