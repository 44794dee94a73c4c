"""The mesh phase inside the super-step (k_segres_list, k_mesh_decide) in batches
beyond one CTA's threads: more than 1,024 instances that converge in the same
super-step while their continuation goes on (the running offsets of the lists'
second chunk), and more than 4,096, where the Newton decisions have a launch of
their own (k_decide, k_lists mode 1).  One instance in forty starts from another
guess and keeps its own pace.

Each instance has the counts, the mesh and the solution of the same instance
solved alone (to 1e-10: one or a thousand instances may take other launches for
the block rows, with the same arithmetic), and the copies of an instance in the
batch have the same bits."""
import numpy as np
import pytest

from conftest import load_problem, pkg

pytestmark = pytest.mark.gpu
COUNTS = ("status", "newton_steps", "residual_evals", "segment_evals", "remeshes", "continuation_steps", "N")


@pytest.mark.parametrize("instances", [1500, 4100])
def test_large_batches_solve_as_single_instances(instances):
    cs = pkg()
    pr = load_problem("vdp_ineq")
    cp = cs.CompiledProblem(pr, 3)
    opts = cs.default_opts(pr)
    Y, Z, P = np.asarray(pr.Y0, float), np.asarray(pr.Z0, float), np.asarray(pr.P0, float).reshape(-1)
    guesses = [(np.asarray(pr.T0, float), Y * s, Z) for s in (1.0, 0.99)]

    def solve(k):
        bt = cs.Batch(cp, k.size)
        bt.set_guess([guesses[i] for i in k], np.tile(P, (k.size, 1)))
        bt.solve(opts)
        return bt.solution()

    alone = [solve(np.array([i]))[0] for i in range(2)]
    assert all(a["success"] and a["continuation_steps"] > 20 for a in alone)
    which = (np.arange(instances) % 40 == 1).astype(int)
    batch = solve(which)
    for i, s in enumerate(batch):
        a, first = alone[which[i]], batch[which[i]]
        assert tuple(s[k] for k in COUNTS) == tuple(a[k] for k in COUNTS), i
        for k in ("t", "y", "z", "p"):
            np.testing.assert_array_equal(s[k], first[k])
            np.testing.assert_allclose(s[k], a[k], rtol=0, atol=1e-10)
