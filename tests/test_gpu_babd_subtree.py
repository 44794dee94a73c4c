"""cs_babd_solve's subtree kernels (blocks up to 16 x 16) at the edges of their
chunks (16 rows, four levels), their register shapes (block sizes, columns per
lane) and beyond them, against a dense solve of the same system.  Tolerance:
1e-9 of the solution's scale (the systems' condition is below 1e6)."""
import numpy as np
import pytest

from conftest import pkg
from test_gpu_babd import babd_gpu, random_babd

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("fn", ["cs_babd_solve", "cs_babd_solve_noalloc"])
@pytest.mark.parametrize("ny,npar,n", [
    (1, 0, 1), (1, 1, 2), (2, 0, 16), (3, 2, 17), (4, 3, 31), (4, 20, 33), (5, 1, 255), (6, 2, 256), (6, 2, 257), (8, 7, 100),
    (8, 8, 48), (7, 32, 20), (9, 0, 64), (12, 4, 65), (16, 15, 40), (16, 16, 33), (13, 32, 18), (17, 2, 50)])
def test_subtree_solve_matches_dense_solve(fn, ny, npar, n):
    cs = pkg()
    A, C, H, b, B0, Bn, Vn, r = random_babd(ny, npar, n, seed=100 * ny + n)
    C = C + 0.1 * np.random.default_rng(n).standard_normal(C.shape)
    dy, dp, sing = babd_gpu(cs, fn, ny, npar, n, A, C, H, b, B0, Bn, Vn, r)
    size = (n + 1) * ny + npar
    M, g = np.zeros((size, size)), np.zeros(size)
    for i in range(n):
        q = slice(i * ny, (i + 1) * ny)
        M[q, i * ny:(i + 1) * ny], M[q, (i + 1) * ny:(i + 2) * ny], M[q, (n + 1) * ny:], g[q] = A[i], C[i], H[i], b[i]
    M[n * ny:, :ny] += B0
    M[n * ny:, n * ny:(n + 1) * ny] += Bn
    M[n * ny:, (n + 1) * ny:], g[n * ny:] = Vn, -r
    x = np.linalg.solve(M, g)
    scale = max(1.0, np.abs(x).max())
    assert sing == 0
    np.testing.assert_allclose(dy.ravel(), x[:(n + 1) * ny], rtol=0, atol=1e-9 * scale)
    np.testing.assert_allclose(dp, x[(n + 1) * ny:], rtol=0, atol=1e-9 * scale)
