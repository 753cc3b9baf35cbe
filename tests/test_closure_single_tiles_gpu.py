"""Each tile of 16 samples counts once in the gradient, whatever the size: the
targets are the network's own outputs except in one tile's rows, so that loss
and gradient come from that tile alone and a lost tile leaves nothing, a
doubled one twice as much. And large batches, whose kernel form is another, are
not slower by the sample."""
import time

import numpy as np
import pytest

from oracle import mlp_oracle as ref
from ultraballpit_b200.closure import ClosureNet

from test_closure_gpu import _data

pytestmark = pytest.mark.gpu


def tiles_of(n):
    """The first tiles (every place in a group of four), one in the middle, and those of the last group."""
    last = (n - 1) // 16
    return sorted({q for q in (0, 1, 2, 3, 4, last // 2, last - 4, last - 3, last - 2, last - 1, last) if 0 <= q <= last})


# parts of a tile, of a group of four and of k_adam's sixteen rows; 9,409 samples on are four tiles a block on 148 SMs
@pytest.mark.parametrize("n", [17, 100, 1009, 9408, 9409, 9473, 20001])
def test_every_tile_counts_once(n):
    net = ClosureNet(seed=6)
    params = net.params()
    x, t = _data(n, n)
    y = net.forward(x)  # what the training kernel computes too, bit for bit: same products in the same order
    for q in tiles_of(n):
        rows = slice(16 * q, min(16 * q + 16, n))
        target = y.copy()
        target[rows] = t[rows]
        loss, g = net.loss_grad(x, target)
        want_loss, want = ref.loss_grad(params, x[rows], t[rows])
        part = (rows.stop - rows.start) / n
        # both round to bfloat16 at the same points from values that agree to about 1e-6: few operands round apart,
        # each by 2^-8 of itself
        assert abs(loss - part * want_loss) <= 1e-2 * part * want_loss, q
        o = 0
        for name, shp in ref.SHAPES:
            k = int(np.prod(shp))
            a, b = g[o:o + k], part * want[o:o + k]
            assert np.linalg.norm(a - b) <= 3e-2 * max(np.linalg.norm(b), 1e-12), (q, name)
            o += k


def test_large_batches_are_not_slower():
    """Four tiles a block, from 9,409 samples on 148 SMs, leave fewer rows to add than one tile a block. With one
    row's load in flight they took 1.6 times as long."""
    net = ClosureNet(seed=6)
    x, t = _data(54000, 1)
    took = {}
    for batch in (9000, 18000):
        took[batch] = []
        for _ in range(8):
            t0 = time.perf_counter()
            net.train(x, t, batch=batch, epochs=4)
            took[batch].append(time.perf_counter() - t0)
    assert np.min(took[18000]) < 1.3 * np.min(took[9000]), took
