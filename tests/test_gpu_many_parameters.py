"""Small block rows with many parameters: the top system is larger than the 16 x 16
that stay in registers, so the upper tree levels' kernel holds all of it in shared
memory.  Its direction (babd_path 0) has the bits of the per-level kernels
(babd_path 2), whose buffer is a launch of its own, and solves the condensed system.

The problem y' = M y + e p_0 with linear boundary rows R_0 y_0 + R_n y_n + V p = c
comes as generated source.  ny = 2 and 3 around the line (2 ny + np = 16, 17), the
sizes where the boundary rows alone would be too small a buffer (np >= 11), and
one whose top system takes more than 48 KB (np = 75)."""
import numpy as np
import pytest

from conftest import pkg

pytestmark = pytest.mark.gpu
NODES = [2, 3, 5, 16, 17, 18, 34, 70]


def linear_problem(cs, ny, npar, rng):
    M, e = 0.3 * rng.standard_normal((ny, ny)), rng.standard_normal(ny)
    R0, Rn = rng.standard_normal((ny + npar, ny)), rng.standard_normal((ny + npar, ny))
    V, c = rng.standard_normal((ny + npar, npar)), rng.standard_normal(ny + npar)
    D = np.hstack([M, e[:, None], np.zeros((ny, npar - 1))])
    DR = np.hstack([R0, Rn, V])
    pt = "const double* y, const double* z, const double* p, const double* th"
    bc = "const double* y0, const double* y1, const double* p, const double* th"
    fn = "__device__ __forceinline__ void"
    lines = ["%s cs_f(%s, double* f) {" % (fn, pt)]
    lines += ["  f[%d] = %s + %r*p[0];" % (a, " + ".join("%r*y[%d]" % (float(M[a, q]), q) for q in range(ny)), float(e[a])) for a in range(ny)]
    lines += ["}", "%s cs_Df(%s, double* Df) {" % (fn, pt)]
    lines += ["  Df[%d] = %r;" % (i, float(v)) for i, v in enumerate(D.ravel())]
    lines += ["}", "%s cs_g(%s, const double a, double* g) {}" % (fn, pt), "%s cs_Dg(%s, const double a, double* Dg) {}" % (fn, pt)]
    lines += ["%s cs_r(%s, double* r) {" % (fn, bc)]
    args = ["y0[%d]" % q for q in range(ny)] + ["y1[%d]" % q for q in range(ny)] + ["p[%d]" % q for q in range(npar)]
    lines += ["  r[%d] = %s - %r;" % (a, " + ".join("%r*%s" % (float(v), x) for v, x in zip(DR[a], args)), float(c[a])) for a in range(ny + npar)]
    lines += ["}", "%s cs_Dr(%s, double* Dr) {" % (fn, bc)]
    lines += ["  Dr[%d] = %r;" % (i, float(v)) for i, v in enumerate(DR.ravel())]
    lines += ["}", ""]
    return cs.GeneratedProblem("\n".join(lines), ny, 0, npar, 1, 0), DR, c


@pytest.mark.parametrize("ny,npar", [(2, 12), (2, 13), (2, 25), (3, 10), (3, 11), (2, 75)])
def test_direction_with_many_parameters(ny, npar):
    cs = pkg()
    rng = np.random.default_rng(100 * ny + npar)
    pr, DR, c = linear_problem(cs, ny, npar, rng)
    bt = cs.Batch(cs.CompiledProblem(pr, 3), len(NODES))
    y = [rng.standard_normal((n, ny)) for n in NODES]
    p = rng.standard_normal((len(NODES), npar))
    bt.set_guess([(np.linspace(0.0, 1.0, n), yi, None) for n, yi in zip(NODES, y)], p)
    d = {}
    for path in (0, 2):
        bt.set_opts(cs.default_opts(pr, babd_path=path))
        d[path] = bt.stage_newton_direction(0.1)
    for k in ("rows", "dy", "dydot", "dp"):
        np.testing.assert_array_equal(d[0][k], d[2][k])
    off = 0
    for i, n in enumerate(NODES):
        # the condensed system, densely; backward stable elimination of random
        # rows: 1e-9 of the solution's scale as for the standalone solve
        size = n * ny + npar
        S, g = np.zeros((size, size)), np.zeros(size)
        for j in range(n - 1):
            q, R = slice(j * ny, (j + 1) * ny), d[0]["rows"][off + j].reshape(-1, ny).T
            S[q, j * ny:(j + 1) * ny], S[q, (j + 1) * ny:(j + 2) * ny] = R[:, :ny], R[:, ny:2 * ny]
            S[q, n * ny], g[q] = R[:, 2 * ny], R[:, 2 * ny + 1]
        S[(n - 1) * ny:, :ny] += DR[:, :ny]
        S[(n - 1) * ny:, (n - 1) * ny:n * ny] += DR[:, ny:2 * ny]
        S[(n - 1) * ny:, n * ny:] = DR[:, 2 * ny:]
        g[(n - 1) * ny:] = c - DR @ np.concatenate([y[i][0], y[i][-1], p[i]])
        x = np.linalg.solve(S, g)
        scale = max(1.0, np.abs(x).max())
        np.testing.assert_allclose(d[0]["dy"][off:off + n].ravel(), x[:n * ny], rtol=0, atol=1e-9 * scale)
        np.testing.assert_allclose(d[0]["dp"][i], x[n * ny:], rtol=0, atol=1e-9 * scale)
        off += n
