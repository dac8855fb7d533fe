"""Tiles of the fp32 encoder where a batch is many rounds of blocks: an SM holds two of them at a time, so that one block's start is under the other's sums.
Hidden sizes that are odd multiples of 64 have blocks of 16 records for each env of a lane: with 96 or more there is no room for a second block."""
import ctypes as C

import pytest


@pytest.mark.parametrize("hidden", [64, 192, 320, 448])
@pytest.mark.parametrize("num_envs", [65536, 131072, 262144])
def test_two_blocks_of_the_encoder_an_sm(cfx, num_envs, hidden):
    t = (C.c_int32 * 4)()
    cfx.check(cfx.lib().cfx_selftest_strict_tiles(num_envs, hidden, t))
    assert t[3] == 2 and t[2] <= 5
