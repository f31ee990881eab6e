"""GroupedSequence and Sequence training on a stream that the caller has set
(vkc_device_set_stream): the same step as on the device's own stream."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture
def caller_stream(gpu):
    """Makes a stream of the caller's current; the device's own again after."""
    from vulkpy_gb300 import _lib
    lib, h = _lib.lib, gpu.handle
    s = C.c_void_p()
    assert lib.vkc_stream_create(h, C.byref(s)) == 0

    def use(on):
        gpu.wait()
        assert lib.vkc_device_set_stream(h, s if on else None) == 0

    yield use
    use(False)
    assert lib.vkc_stream_destroy(h, s) == 0


def _models(gpu, opt):
    from vulkpy_gb300 import nn
    rng = np.random.default_rng(5)
    nets = []
    for i, hid, o in ((7, 33, 3), (20, 64, 5)):
        d = [nn.Dense(gpu, n, m, w_opt=opt(), b_opt=opt()) for n, m in ((i, hid), (hid, o))]
        for q in d:
            q.w.value[:] = rng.standard_normal(q.w.value.shape).astype(np.float32) * 0.2
        nets.append(nn.Sequence([d[0], nn.ReLU(), d[1]], nn.MSELoss()))
    xs = [rng.standard_normal((b, i)).astype(np.float32) for b, i in ((9, 7), (40, 20))]
    ys = [rng.standard_normal((b, o)).astype(np.float32) for b, o in ((9, 3), (40, 5))]
    return nets, xs, ys


def _state(nets):
    return [np.array(p.value) for n in nets for k in (0, 2) for p in (n.L[k].w, n.L[k].b)]


def _grouped_step(gpu):
    import vulkpy_gb300 as vk
    from vulkpy_gb300 import nn
    nets, xs, ys = _models(gpu, lambda: nn.SGD(lr=1e-2))
    g = nn.GroupedSequence(nets)
    ax, ay = ([vk.Array(gpu, data=v) for v in a] for a in (xs, ys))
    for _ in range(3):
        preds, losses = g.train(ax, ay)
    return _state(nets) + [np.array(p) for p in preds] + [np.array(losses)]


def _sequence_step(gpu):
    import vulkpy_gb300 as vk
    from vulkpy_gb300 import nn
    opt = nn.SGD(lr=1e-2)
    nets, xs, ys = _models(gpu, lambda: opt)
    for n, x, y in zip(nets, xs, ys):
        ax, ay = vk.Array(gpu, data=x), vk.Array(gpu, data=y)
        for _ in range(3):
            n.train(ax, ay)
    return _state(nets)


@pytest.mark.parametrize("step", [_grouped_step, _sequence_step])
def test_training_step_on_a_callers_stream(gpu, caller_stream, step):
    own = step(gpu)
    caller_stream(True)
    got = step(gpu)
    caller_stream(False)
    for a, b in zip(own, got):
        np.testing.assert_array_equal(a, b)


def test_side_branch_where_the_gpu_is_waited_for(gpu, monkeypatch):
    """A step of small models run call by call waits for the host, and stays on
    one stream; the same values as on the branch, which a graph uses."""
    import vulkpy_gb300 as vk
    from vulkpy_gb300.nn.grouped import GroupedSequence
    used = []
    beside = GroupedSequence._beside
    monkeypatch.setattr(GroupedSequence, "_beside", lambda self, side, run: used.append(side) or beside(self, side, run))
    off = _grouped_step(gpu)
    assert not any(used)
    with monkeypatch.context() as m:
        m.setattr(GroupedSequence, "_gpu_bound", lambda self, batch: True)
        on = _grouped_step(gpu)
    assert any(used)
    for a, b in zip(off, on):
        np.testing.assert_array_equal(a, b)
    from vulkpy_gb300 import nn
    nets, xs, ys = _models(gpu, lambda: nn.SGD(lr=1e-2))
    group = GroupedSequence(nets)
    ax, ay = ([vk.Array(gpu, data=v) for v in a] for a in (xs, ys))
    group.train(ax, ay)
    used.clear()
    with vk.graph.Graph(gpu):
        group.train(ax, ay)
    assert used and all(used)
