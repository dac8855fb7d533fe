"""Addresses of host arrays: the same by way of the buffer protocol as the array interface gives, for arrays that have no such buffer too."""
import numpy as np
import pytest


def _read_only():
    a = np.arange(8, dtype=np.int32)
    a.flags.writeable = False
    return a


@pytest.mark.parametrize("a", [
    np.zeros((3, 44), np.float32), np.zeros(96, np.uint8)[4:], np.zeros((4, 4), np.float32)[1:3], np.zeros((4, 4), np.float32)[:, 1:3],
    np.asfortranarray(np.zeros((3, 5))), np.zeros(8, np.float32)[::-1], np.zeros(0, np.int32), np.zeros((), np.int32), _read_only(),
    np.frombuffer(b"12345678", np.uint16)], ids=range(10))
def test_address(cfx, a):
    assert cfx.host_address(a) == a.__array_interface__["data"][0]
