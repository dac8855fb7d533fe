"""The reciprocals of the fp32 cells (an approximation refined by one Newton step) against CUDA's division, bit for bit."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _bits(x):
    return int(np.float32(x).view(np.uint32))


ONE, MOST, INF, NAN = _bits(1.0), _bits(2.0 ** 126), _bits(np.inf), 0x7FC00000


@pytest.mark.parametrize("first,last,far", [
    (ONE, MOST, 0),                  # every denominator that is not divided: 1,056,964,609 values
    (MOST + 1, INF, 0),              # every one that is: the reciprocal is subnormal or 0
    (INF, 0x7FFFFFFF, 0),            # NaN
    # one such value among eleven that would not have been divided
    (ONE, _bits(4.0), MOST + 1), (ONE, _bits(4.0), INF), (ONE, _bits(4.0), NAN), (MOST - 4096, MOST, INF),
    (ONE, ONE, 0), (ONE, ONE + 11, 0), (ONE, ONE + 12, 0), (MOST - 6, MOST + 6, 0)])   # batches of one value, and across the limit
def test_reciprocals_are_those_of_the_division(cfx, gpu, first, last, far):
    differing = C.c_uint64(1)
    cfx.check(cfx.lib().cfx_selftest_reciprocals(0, first, last, far, C.byref(differing)))
    assert differing.value == 0
