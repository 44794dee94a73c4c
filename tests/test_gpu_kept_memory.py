"""Device memory that calls keep: the solution writer's text buffer stays with its
batch up to 256 MB and goes back to the device above, and so do the network's
copies of a call's host arrays."""
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


def test_large_training_sets_go_back_to_the_device():
    cs = pkg()
    rng = np.random.default_rng(0)
    X, Y = rng.random((66000, 4), dtype=np.float32), rng.random((66000, 1100), dtype=np.float32)  # Y: 290 MB
    net = cs.warmstart.Mlp(4, 1100, width=32, depth=3, seed=1)
    net.fit_normalization(X[:2048], Y[:2048])
    net.train(X[:2048], Y[:2048], epochs=1, batch=1024, lr=1e-3)  # training buffers, kernels
    first = net.predict(X[:2048])
    before = free_memory()
    net.train(X, Y, epochs=1, batch=1024, lr=0.0)
    assert before - free_memory() < 64 * MB
    whole = net.predict(X)  # 65,536 rows at a time: 288 MB of output
    assert before - free_memory() < 64 * MB
    np.testing.assert_array_equal(whole[:2048], first)
