"""Large-block tree and top system: blocked Householder panels, a merge shared by
the CTAs of a cluster where a level has few merges.  Sizes around the panel width
(16), the eight-column blocks and 256 rows; meshes from one interval up.

The direction has to satisfy the condensed system it was solved from.  Householder
elimination and back substitution are backward stable: the residual of a row is
at most about n eps times |row| |x| with n the reflectors an entry meets, 2 ny per
level and the top system's; allowed: 8 (2 ny) (levels + 2) eps of the largest
|row| |x|.  The split over CTAs is over columns only, so an instance's direction
has the same bits alone (eight CTAs per merge) and in a batch (one per merge)."""
import numpy as np
import pytest

from conftest import OracleProblem, pkg
from oracle import collocation_oracle as O

pytestmark = pytest.mark.gpu
NODES = [2, 3, 4, 5, 8, 17, 34]


@pytest.mark.parametrize("K,m,layout", [(2, 3, 2), (3, 3, 2), (4, 4, 2), (5, 3, 2), (6, 3, 2), (7, 3, 0), (9, 3, 0), (16, 3, 0), (33, 3, 0)])
def test_direction_solves_the_condensed_system_for_any_split(K, m, layout):
    cs = pkg()
    rng = np.random.default_rng(100 + K)
    pr = cs.ocp.Problem(cs.workloads.pendulum_ocp(K, rng.uniform(-0.5, 0.5, K), nodes=5), name="pend%d" % K)
    P, rk = OracleProblem(pr), cs.tables.lobatto(m)
    cp = cs.CompiledProblem(pr, m, layout=layout)
    Y0, Z0, p0 = np.asarray(pr.Y0, float), np.asarray(pr.Z0, float), np.asarray(pr.P0, float)
    states, ps = [], []
    for n in NODES:
        y, yd, zt = O.form_initial_input(P, m, n, np.repeat(Y0[:1], n, 0), np.repeat(Z0[:1], n, 0), p0, rk)
        states.append((np.concatenate([[0.0], np.cumsum(rng.uniform(0.05, 0.1, n - 1))]),
                       *(a + 0.05 * rng.standard_normal(a.shape) for a in (y, yd, zt))))
        ps.append(p0 + 0.05 * rng.standard_normal(p0.shape))
    ps = np.array(ps)

    def directions(idx):
        bt = cs.Batch(cp, len(idx))
        bt.set_state([states[i] for i in idx], ps[idx])
        return bt.stage_newton_direction(0.1)

    many = directions(list(range(len(NODES))) * 6)
    ny, off, eps = cp.ny, 0, np.finfo(float).eps
    for i, n in enumerate(NODES):
        one = directions([i])
        dy, dp = one["dy"][:n], one["dp"][0]
        rows = slice(off, off + n - 1)
        np.testing.assert_array_equal(many["rows"][rows], one["rows"][:n - 1])
        np.testing.assert_array_equal(many["dy"][off:off + n], dy)
        np.testing.assert_array_equal(many["dp"][i], dp)
        off += n
        t, y, yd, zt = states[i]
        two = (np.array([0.0, 1.0]), y[[0, -1]], yd[:m], zt[:m])
        r = O.compute_f_q(P, m, 2, rk, *two, ps[i], 0.1)[4]
        B_0, B_n, V_n = O.boundary_jacobian(P, 2, two[1], ps[i])
        R = one["rows"][:n - 1].reshape(n - 1, -1, ny).transpose(0, 2, 1)
        C, J, b = R[:, :, :ny], R[:, :, 2 * ny:-1], R[:, :, -1]
        res = np.einsum("iac,ic->ia", C, dy[:-1]) + dy[1:] + J @ dp[:cp.np_eff] - b
        size = np.einsum("iac,ic->ia", abs(C), abs(dy[:-1])) + abs(dy[1:]) + abs(J) @ abs(dp[:cp.np_eff]) + abs(b)
        rbc = B_0 @ dy[0] + B_n @ dy[-1] + V_n @ dp + r
        sbc = abs(B_0) @ abs(dy[0]) + abs(B_n) @ abs(dy[-1]) + abs(V_n) @ abs(dp) + abs(r)
        tol = 16 * ny * (np.ceil(np.log2(n)) + 2) * eps * max(size.max(), sbc.max())
        assert max(np.abs(res).max(), np.abs(rbc).max()) <= tol, (n, np.abs(res).max(), np.abs(rbc).max(), tol)
