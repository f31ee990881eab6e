"""Graph.launch: what it does to the arrays that the graph writes."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _doubling_graph(gpu, n_arrays):
    """A graph that doubles its arrays in place."""
    import vulkpy_gb300 as vk
    arrays = [vk.Array(gpu, data=np.full(300000, i + 1, np.float32)) for i in range(n_arrays)]
    g = vk.graph.Graph(gpu)
    with g:
        for a in arrays:
            a *= 2.0
    return g, arrays


def test_launch_is_one_operation(gpu):
    """However many arrays the graph writes (64 grouped models: 512), a launch
    takes one sequence number and every array waits for that one."""
    g, arrays = _doubling_graph(gpu, 5)
    before = gpu._dev.seq
    g.launch()
    assert gpu._dev.seq == before + 1
    assert {a.job.seq for a in arrays} == {gpu._dev.seq}
    for i, a in enumerate(arrays):
        a.wait()
        assert np.all(np.asarray(a) == 2.0 * (i + 1))


def test_a_read_back_begun_before_a_launch_is_not_used(gpu):
    """As for any other write after a prefetch."""
    g, (a,) = _doubling_graph(gpu, 1)
    g.launch()
    a.prefetch()
    g.launch()
    assert np.all(np.asarray(a) == 4.0)
