"""A warp that waits as a whole gives up as a whole."""
import pytest

pytestmark = pytest.mark.gpu


def test_all_lanes_of_a_warp_give_up_together(cfx, gpu):
    """The self-test's warp waits with half of its lanes on a complete phase and half on one that never completes.  If the
    lanes decided one by one, half would go on alone, to instructions that take the whole warp."""
    assert cfx.lib().cfx_selftest_wait_timeout(0, 5) == cfx.ERR_DEVICE_TIMEOUT, cfx.lib().cfx_last_error()
    assert b"site %d," % 0x7E in cfx.lib().cfx_last_error()
