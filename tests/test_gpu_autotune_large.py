"""The launch-shape tuner on large stage systems in FP64 (one CTA per interval,
its size fixed by the kernel): whatever shape it keeps, the direction has the
same bits as before.  Stage systems on both sides of the 128-row line between
the CTA sizes, 102 (K = 8, m = 4), 136 and 272 rows (K = 16, m = 3 and 5), and a
Van der Pol stage system of 15 rows on the large-system kernels."""
import numpy as np
import pytest

from conftest import load_problem, pkg

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("K,m", [(8, 4), (16, 3), (16, 5), (0, 4)])
def test_tuned_large_condensation_keeps_the_direction(K, m):
    cs = pkg()
    rng = np.random.default_rng(10 * K + m)
    if K:
        pr = cs.ocp.Problem(cs.workloads.pendulum_ocp(K, rng.uniform(-0.5, 0.5, K), nodes=41), name="pend%d" % K)
    else:
        pr = load_problem("vdp")
    cp = cs.CompiledProblem(pr, m, layout=2)
    s1 = (m - 1) * (cp.ny + cp.nz)
    N = 41
    bt = cs.Batch(cp, 3)
    t = np.linspace(0.0, 3.0, N)
    y, z = 0.1 * rng.standard_normal((3, N, cp.ny)), 0.1 * rng.standard_normal((3, N, cp.nz))
    p = 0.1 * rng.standard_normal((3, cp.np))
    bt.set_guess([(t, y[i], z[i]) for i in range(3)], p)
    before = bt.stage_newton_direction(0.1)
    r = bt.autotune(reps=2)
    after = bt.stage_newton_direction(0.1)
    assert r["block"] == (128 if s1 <= 128 else 256) and r["lanes"] == 0 and r["grid"] >= 1
    for k in ("rows", "dy", "dydot", "dzt", "dp"):
        assert np.isfinite(before[k]).all()
        np.testing.assert_array_equal(before[k], after[k])
