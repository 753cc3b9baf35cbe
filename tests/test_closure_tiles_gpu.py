"""The training kernel around its edges against the float64 oracle: parts of a
16-sample tile, of a group of four tiles and of k_adam's sixteen rows, and the
switch to four tiles per block (from 64 samples per SM: 9,409 on 148)."""
import numpy as np
import pytest

from oracle import mlp_oracle as ref
from ultraballpit_b200.closure import ClosureNet

from test_closure_gpu import _data

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 15, 16, 17, 63, 64, 65, 255, 256, 257, 1009, 9408, 9409, 9473, 20001])
def test_gradient_of_n_samples(n):
    net = ClosureNet(seed=6)
    x, t = _data(n, n)
    loss, g = net.loss_grad(x, t)
    want_loss, want = ref.loss_grad(net.params(), x, t)
    # both round to bfloat16 at the same points from values that agree to about 1e-6: few operands round apart, each
    # by 2^-8 of itself, so 3e-2 of a tensor's norm is a wide bound (a lost or doubled tile is of order 1 / tiles)
    assert abs(loss - want_loss) <= 1e-2 * want_loss
    o = 0
    for name, shp in ref.SHAPES:
        k = int(np.prod(shp))
        a, b = g[o:o + k], want[o:o + k]
        assert np.linalg.norm(a - b) <= 3e-2 * max(np.linalg.norm(b), 1e-12), name
        o += k


def test_samples_are_kept_between_calls_of_other_sizes():
    net = ClosureNet(seed=7)
    out = []
    for n in (300, 20000, 40, 300):
        x, t = _data(n, n)
        out.append((net.loss_grad(x, t), net.forward(x)))
    (l0, g0), y0 = out[0]
    (l3, g3), y3 = out[3]
    assert l0 == l3
    np.testing.assert_array_equal(g0, g3)
    np.testing.assert_array_equal(y0, y3)
