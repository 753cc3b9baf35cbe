"""One network used by several host threads at a time: a net keeps its sample
buffers between calls, and calls that overlap must not share them."""
import threading

import numpy as np
import pytest

from ultraballpit_b200.closure import ClosureNet

from test_closure_gpu import _data

pytestmark = pytest.mark.gpu


def in_threads(*fs):
    errors = []

    def guarded(f):
        try:
            f()
        except Exception as e:  # noqa: BLE001 - any failure of a thread fails the test
            errors.append(e)
    ts = [threading.Thread(target=guarded, args=(f,)) for f in fs]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert not errors, errors


def test_forward_in_several_threads():
    net = ClosureNet(seed=5)
    xs = [_data(n, n)[0] for n in (100, 3000, 40000, 70001)]
    want = [net.forward(x) for x in xs]

    def reader(q):
        def go():
            for r in range(20):  # sizes that make the kept buffers grow, in another order per thread
                i = (q + r) % len(xs)
                np.testing.assert_array_equal(net.forward(xs[i]), want[i])
        return go
    in_threads(*[reader(q) for q in range(4)])


def test_forward_and_gradients_beside_training():
    x, t = _data(20000, 1)
    alone = ClosureNet(seed=6)
    want = alone.train(x, t, batch=1024, epochs=8, seed=2)
    net = ClosureNet(seed=6)
    got = []
    grads = []

    def forward():
        for _ in range(20):
            assert np.isfinite(net.forward(x[:5000])).all()

    def gradient():  # waits for a training that has begun, or is done before it
        loss, g = net.loss_grad(x[:333], t[:333])
        assert np.isfinite(loss)
        grads.append(g)
    before, after = (n.loss_grad(x[:333], t[:333])[1] for n in (ClosureNet(seed=6), alone))
    in_threads(lambda: got.append(net.train(x, t, batch=1024, epochs=8, seed=2)), forward, gradient)
    np.testing.assert_array_equal(got[0], want)
    np.testing.assert_array_equal(net.params(), alone.params())
    assert any(np.array_equal(grads[0], g) for g in (before, after))


def test_nets_that_come_and_go():
    """Kept buffers on both sides of 1 MB and 64 MB (what comes from the library's pool), given back by one net and
    taken by the next, and by several at a time."""
    sizes = (500, 3000, 60000, 400000)
    data = [_data(n, n) for n in sizes]
    net = ClosureNet(seed=8)
    want = [net.loss_grad(x, t) for x, t in data]
    net.close()

    def user(q):
        def go():
            for r in range(8):
                i = (q + r) % len(sizes)
                m = ClosureNet(seed=8)
                loss, g = m.loss_grad(*data[i])
                assert loss == want[i][0]
                np.testing.assert_array_equal(g, want[i][1])
                m.close()
        return go
    in_threads(*[user(q) for q in range(3)])
