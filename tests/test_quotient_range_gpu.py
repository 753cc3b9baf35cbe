"""The pair sums' reciprocal and quotient (sph::rcp_rn, div_rn) against CUDA's
IEEE operations at the ends of what they are used for: divisors down to the
smallest normal number, and the XSPH quotient of the smallest masses allowed
by the largest density sums."""
import ctypes

import numpy as np
import pytest

from test_pair_sums_gpu import arith  # noqa: F401 - the module's compiled check

pytestmark = pytest.mark.gpu


# dividends scale * [1, 2), divisors in [2^lo, 2^hi]; every quotient is normal
@pytest.mark.parametrize("scale,lo,hi", [(2.0 ** -94, -126, -60), (1.0, -126, -100), (2.0 ** -93, -1, 31),
                                         (2.0 ** 20, -106, -60), (2.0 ** 41, 1, 31)])
def test_quotients_at_the_ends(arith, scale, lo, hi):  # noqa: F811
    rng = np.random.default_rng(hi - lo)
    m = np.concatenate([[1.0, 1.0 + 2.0 ** -23, 2.0 - 2.0 ** -23], rng.uniform(1.0, 2.0, 13)])
    b = np.concatenate([m * 2.0 ** e for e in (lo, lo + 1, (lo + hi) // 2, hi - 1)]).astype(np.float32)
    bad = (ctypes.c_ulonglong * 3)()
    assert arith.arith_check(np.float32(2.0 ** -126), np.float32(2.0 ** -100),
                             b.ctypes.data_as(ctypes.POINTER(ctypes.c_float)), len(b), scale, bad) == 0
    assert list(bad)[1:] == [0, 0]
