"""cs_babd_solve's subtree kernels at the edges of their chunks of 8 rows and three
levels: the last system that one CTA solves alone (8 rows) and the first that it
does not, odd rows inside a chunk, and the edges of the second and third chunk
levels (64 and 512 rows).  Check and tolerance of test_gpu_babd_subtree.py."""
import pytest

import test_gpu_babd_subtree as subtree

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ny,npar", [(4, 2), (12, 3)])
@pytest.mark.parametrize("n", [3, 4, 5, 6, 7, 8, 9, 10, 15, 16, 63, 64, 65, 71, 72, 73])
def test_chunk_edges(ny, npar, n):
    subtree.test_subtree_solve_matches_dense_solve("cs_babd_solve", ny, npar, n)


@pytest.mark.parametrize("n", [511, 512, 513, 520, 521])
def test_third_chunk_level(n):
    subtree.test_subtree_solve_matches_dense_solve("cs_babd_solve", 3, 1, n)
