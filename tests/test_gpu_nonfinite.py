"""A NaN or an infinity that a linear system holds shows in its solution: the
reflectors of cs_babd_solve (subtree kernels up to 16 x 16 blocks, level kernels
above) and of the Newton direction (boundary Jacobian in the top system, every
route to it) hand it on instead of leaving its column out."""
import re

import numpy as np
import pytest

from conftest import load_problem, pkg
from test_gpu_babd import babd_gpu, random_babd

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("fn", ["cs_babd_solve", "cs_babd_solve_noalloc"])
@pytest.mark.parametrize("ny,npar,n", [(1, 0, 2), (4, 2, 1), (4, 2, 2), (6, 2, 40), (8, 3, 9), (8, 7, 70), (12, 2, 20), (16, 4, 30), (17, 2, 20)])
def test_babd_solution_of_a_system_with_nan(fn, ny, npar, n):
    cs = pkg()
    good = random_babd(ny, npar, n, seed=ny)
    rng = np.random.default_rng(n)
    for value in (np.nan, np.inf, -np.inf):
        for which in range(8):  # A, C, H, b, B0, Bn, Vn, r
            if npar == 0 and which in (2, 6):
                continue
            system = [np.array(a) for a in good]
            if which == 0 and value != value and n > 1:
                system[0][1, :, 0] = np.where(np.arange(ny) == ny - 1, value, system[0][1, :, 0])
            else:
                system[which].reshape(-1)[rng.integers(system[which].size)] = value
            dy, dp, sing = babd_gpu(cs, fn, ny, npar, n, *system)
            assert sing == 0
            assert not np.isfinite(dy).any() and not np.isfinite(dp).any(), (value, which)


@pytest.mark.parametrize("layout,path", [(0, 0), (0, 1), (0, 2), (2, 0)])
@pytest.mark.parametrize("entry", [0, 11, 58])  # (row 0, y_0), (row 1, y_0), (last row, p)
def test_direction_with_nan_in_the_boundary_jacobian(layout, path, entry):
    cs = pkg()
    pr = load_problem("vdp")
    gp = cs.GeneratedProblem.from_problem(pr, name="vdp_nan")
    src, k = re.subn(r"Dr\[%d\] = [^;]*;" % entry, "Dr[%d] = __longlong_as_double(0x7ff8000000000000ll);" % entry,
                     gp.cuda_source)
    assert k == 1
    gp.cuda_source = src
    bt = cs.Batch(cs.CompiledProblem(gp, 4, layout=layout), 2)
    t = np.linspace(0.0, 4.0, 21)
    rng = np.random.default_rng(entry)
    bt.set_guess([(t, 0.1 * rng.standard_normal((21, 4)), 0.1 * rng.standard_normal((21, 1))) for _ in range(2)], np.ones((2, 2)))
    bt.set_opts(cs.default_opts(pr, babd_path=path))
    d = bt.stage_newton_direction(0.1)
    assert np.isfinite(d["rows"]).all()
    assert not np.isfinite(d["dy"]).any() and not np.isfinite(d["dp"]).any()
