"""The fused network kernels (csrc/cs_mlp.cu: one CTA carries a block of rows
through all layers) at the edges of their tiles and launch shapes, against the
numpy oracle with the same BF16 operand rounding.  Tolerances as in
test_gpu_mlp.py: gradient and prediction 2e-3 relative (L2), loss 1e-4."""
import numpy as np
import pytest

from conftest import pkg
from oracle import mlp_oracle as MO

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,n_in,width,depth,n_out", [
    (1, 1, 1, 1, 1), (1, 4, 256, 4, 322), (15, 3, 33, 2, 7), (16, 65, 8, 3, 64), (17, 4, 40, 5, 65), (129, 10, 100, 1, 300),
    (2432, 4, 64, 3, 20), (2433, 4, 64, 3, 20), (4865, 5, 48, 3, 9), (70, 4, 16, 2, 2100)])
def test_fused_network_matches_oracle(n, n_in, width, depth, n_out):
    cs = pkg()
    rng = np.random.default_rng(n + n_out)
    X = rng.uniform(-2, 3, (n, n_in)).astype(np.float32)
    Y = (np.sin(X @ rng.standard_normal((n_in, n_out))) + 0.1 * X.sum(1, keepdims=True)).astype(np.float32)
    net = cs.warmstart.Mlp(n_in, n_out, width=width, depth=depth, seed=3)
    net.set_normalization(rng.uniform(-1, 1, n_in), rng.uniform(0.5, 2, n_in), rng.uniform(-1, 1, n_out), rng.uniform(0.5, 2, n_out))
    norm = [a.astype(np.float64) for a in net.norm]
    par, X64, Y64 = net.params().astype(np.float64), X.astype(np.float64), Y.astype(np.float64)
    P, ref = net.predict(X), MO.predict(par, net.sizes, X64, *norm)
    assert np.linalg.norm(P - ref) <= 2e-3 * np.linalg.norm(ref)
    loss, g = net.gradient(X, Y)
    rl, rg = MO.loss_and_grad(par, net.sizes, X64, Y64, *norm)
    assert abs(loss - rl) <= 1e-4 * rl
    assert np.linalg.norm(g - rg) <= 2e-3 * np.linalg.norm(rg)
