"""The register condensation (small stage systems: algebraic unknowns
eliminated stage by stage, the reduced system in registers): Newton directions
at the sizes where a group of lanes, a warp's share of the work list or the
dealt-out right-hand side runs over its edge, and with control weights whose
h / r runs from far below to far above the limit that sends an interval back to
the pivoted elimination of its whole stage system.

Reference: the same Newton systems in extended precision on the host.
Tolerance: no less accurate than the elimination of the whole stage systems.
The blocked LU of the large-system layout is that, so its own error against the
reference, on the same inputs, is the measure (times 8: both are a few
roundings times the condition of the system, which differ by luck), with a
floor of 1e-12 of the direction's scale."""
import numpy as np
import pytest

from conftest import load_problem, pkg

pytestmark = pytest.mark.gpu
LD = np.longdouble


def _solve(A, B):
    """A X = B for stacks of systems, partial pivoting, in the arrays' type."""
    A, B = A.copy(), B.copy()
    n, i = A.shape[-1], np.arange(len(A))
    for k in range(n):
        p = k + np.argmax(np.abs(A[:, k:, k]), axis=1)
        for M in (A, B):
            t = M[:, k].copy()
            M[:, k] = M[i, p]
            M[i, p] = t
        f = A[:, k + 1:, k] / A[:, k, k, None]
        A[:, k + 1:] -= f[:, :, None] * A[:, None, k]
        B[:, k + 1:] -= f[:, :, None] * B[:, None, k]
    for k in range(n - 1, -1, -1):
        B[:, k] = (B[:, k] - np.einsum("bi,bic->bc", A[:, k, k + 1:], B[:, k + 1:])) / A[:, k, k, None]
    return B


def _reference_dy(m, rk, t, y, z, p, th, ydot, zt):
    """dy of the Van der Pol family's Newton system, extended precision."""
    A, b = np.asarray(rk.A, LD), np.asarray(rk.b, LD)
    n = len(t) - 1
    y, h, yd, u, r = y.astype(LD), np.diff(t.astype(LD)), ydot.astype(LD), zt[..., 0].astype(LD), LD(th[2])
    v = y[:-1, None] + h[:, None, None] * np.einsum("jk,nka->nja", A, yd)
    x1, x2, l1, l2 = (v[..., k] for k in range(4))
    q = x1 * x1 - 1
    f = np.stack([x2, -q * x2 - x1 + u, -x1 + l2 * (2 * x1 * x2 + 1), q * l2 - x2 - l1], axis=-1)
    F = np.zeros((n, m, 5, 5), LD)
    F[..., 0, 1] = 1
    F[..., 1, 0], F[..., 1, 1], F[..., 1, 4] = -(2 * x1 * x2 + 1), -q, 1
    F[..., 2, 0], F[..., 2, 1], F[..., 2, 3] = 2 * l2 * x2 - 1, 2 * x1 * l2, 2 * x1 * x2 + 1
    F[..., 3, 0], F[..., 3, 1], F[..., 3, 2], F[..., 3, 3] = 2 * x1 * l2, -1, -1, q
    F[..., 4, 3], F[..., 4, 4] = 1, r
    res = np.concatenate([f - yd, (r * u + l2)[..., None]], axis=-1)
    W = np.zeros((n, m, 5, m, 5), LD)
    for j in range(m):
        for k in range(m):
            W[:, j, :, k, :4] = h[:, None, None] * A[j, k] * F[:, j, :, :4]
        W[:, j, :, j, 4] = F[:, j, :, 4]
        W[:, j, :4, j, :4] -= np.eye(4, dtype=LD)
    R = np.concatenate([F[..., :4], res[..., None]], axis=-1)
    X = _solve(W.reshape(n, 5 * m, 5 * m), R.reshape(n, 5 * m, 5)).reshape(n, m, 5, 5)[:, :, :4]
    D = h[:, None, None] * np.einsum("j,njac->nac", b, X)
    fb = np.diff(y, axis=0) - h[:, None] * np.einsum("j,nja->na", b, yd)
    M, g = np.zeros((1, 4 * n + 6, 4 * n + 6), LD), np.zeros((1, 4 * n + 6, 1), LD)
    for i in range(n):
        M[0, 4 * i:4 * i + 4, 4 * i:4 * i + 4] = D[i, :, :4] - np.eye(4, dtype=LD)
        M[0, 4 * i:4 * i + 4, 4 * i + 4:4 * i + 8] = np.eye(4, dtype=LD)
        g[0, 4 * i:4 * i + 4, 0] = -fb[i] - D[i, :, 4]
    bc = [y[0, 0] - LD(th[0]), y[0, 1] - LD(th[1]), y[0, 2] + LD(p[0]), y[0, 3] + LD(p[1]), y[n, 2], y[n, 3]]
    for k, (c, e) in enumerate(zip((0, 1, 2, 3, 4 * n + 2, 4 * n + 3), bc)):
        M[0, 4 * n + k, c] = 1
        g[0, 4 * n + k, 0] = -e
    M[0, 4 * n + 2, 4 * n + 4] = M[0, 4 * n + 3, 4 * n + 5] = 1
    return _solve(M, g)[0, :4 * n + 4, 0].reshape(n + 1, 4)


def _direction(cs, pr, m, layout, meshes, p, th):
    cp = cs.CompiledProblem(pr, m, layout=layout)
    bt = cs.Batch(cp, len(meshes))
    bt.set_guess(meshes, p, th)
    return bt.stage_newton_direction(0.1)["dy"], bt.state()


@pytest.mark.parametrize("m", [2, 3, 4, 5, 6, 7, 8])
def test_reduced_condensation_is_as_accurate_as_the_whole_stage_system(m):
    cs = pkg()
    pr = load_problem("vdp_family")
    rng = np.random.default_rng(40 + m)
    nodes = [2, 3, 5, 8, 9, 10, 33, 34, 70]
    # h |f_z g_z^-1 g_y| = h / r: from far below to far above the limit of 2^5
    weights = [1.0, 0.1, 1e-3, 1e-5, 3.0, 1e-2, 1e-4, 1.0, 2e-4]
    meshes, th = [], []
    for N, r in zip(nodes, weights):
        t = np.concatenate([[0.0], np.cumsum(rng.uniform(0.02, 0.2, N - 1))])
        y = rng.standard_normal((N, 4)) * np.array([1.0, 1.0, r, r])
        meshes.append((t, y, 0.3 * rng.standard_normal((N, 1))))
        th.append([*rng.uniform(-1.0, 1.0, 2), r])
    p, th = rng.standard_normal((len(nodes), 2)), np.array(th)
    a, state = _direction(cs, pr, m, 1, meshes, p, th)
    b, _ = _direction(cs, pr, m, 2, meshes, p, th)
    o = 0
    for k, (t, y, z) in enumerate(meshes):
        n = len(t)
        ref = _reference_dy(m, cs.tables.lobatto(m), t, y, z, p[k], th[k], state["ydot"][o:o + n - 1], state["zt"][o:o + n - 1])
        scale = max(1.0, float(np.abs(ref).max()))
        err = [float(np.abs(x[o:o + n] - ref).max()) for x in (a, b)]
        assert err[0] <= max(8 * err[1], 1e-12 * scale), (k, err, scale)
        o += n
