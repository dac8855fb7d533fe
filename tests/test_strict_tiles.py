"""Which tiles the fp32 kernels take: the cases of test_strict_tiles_gpu.py reach every one that the rules can choose."""
import ctypes as C

from test_strict_tiles_gpu import HEIGHTS, SMALLEST, TILES

CASES = {**TILES, **HEIGHTS, **SMALLEST}


def _tiles(cfx, n, H):
    t = (C.c_int32 * 4)()
    cfx.check(cfx.lib().cfx_selftest_strict_tiles(n, H, t))
    return tuple(t)


def _kernels(tiles, H):
    """The instantiations behind a choice: how the warps of a block lie depends on the hidden size."""
    layers, deep, encoder, groups = tiles
    return ("layers", layers, deep, H % 64 == 0), ("encoder", encoder, groups, groups == 2 and H % 128 == 0)


def test_cases_take_the_tiles_that_stand_beside_them(cfx):
    for (n, H, _), tiles in CASES.items():
        assert _tiles(cfx, n, H) == tiles, (n, H)


def test_every_choice_has_a_case(cfx):
    reached = {k for (n, H, _), tiles in CASES.items() for k in _kernels(tiles, H)}
    for H in range(32, 513, 32):
        for n in range(32, 65537, 32):
            for k in _kernels(_tiles(cfx, n, H), H):
                assert k in reached, (n, H, k)


def test_sizes_that_the_mode_refuses_are_refused(cfx):
    t = (C.c_int32 * 4)()
    for n, H in ((0, 256), (33, 256), (32, 0), (32, 100), (32, 544)):
        assert cfx.lib().cfx_selftest_strict_tiles(n, H, t) == 1
    assert cfx.lib().cfx_selftest_strict_tiles(32, 256, None) == 1
