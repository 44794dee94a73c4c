"""Device memory that calls keep: the solution writer's text buffer stays with its
batch up to 256 MB and goes back to the device above."""
import numpy as np
import pytest

from conftest import load_problem, pkg

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
MB = 1 << 20


def free_memory():
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


def text_batch(cs, cp, instances, nodes):
    """A batch of full-length random numbers: about 120 bytes of text per node."""
    rng = np.random.default_rng(instances)
    T = instances * nodes
    bt = cs.Batch(cp, instances, node_capacity=T)
    t = np.tile(np.sort(rng.random(nodes)), instances)
    bt.set_guess_packed(np.full(instances, nodes, np.int32), t, rng.standard_normal((T, 4)), rng.standard_normal((T, 1)),
                        np.ones((instances, 2)), None)
    return bt


def test_large_text_buffers_go_back_to_the_device():
    cs = pkg()
    cp = cs.CompiledProblem(load_problem("vdp"), 3)
    text_batch(cs, cp, 2, 100).solution_text()  # the context's stacks grow once (2 KB a thread), whatever the batch
    small, large = text_batch(cs, cp, 64, 1000), text_batch(cs, cp, 1250, 2000)
    before = free_memory()
    text, _ = small.solution_text()
    first = bytes(text)
    kept = before - free_memory()
    assert len(first) < 256 * MB and kept < 64 * MB
    text, _ = small.solution_text()
    assert bytes(text) == first and before - free_memory() == kept
    before = free_memory()
    text, _ = large.solution_text()
    assert len(text) > 256 * MB
    assert before - free_memory() < 64 * MB
