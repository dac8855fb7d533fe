"""Addresses of host arrays: the same by way of the buffer protocol as the array interface gives, for arrays that have no such buffer too."""
import array

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


class Interface:
    """An array that is not numpy's."""

    def __init__(self, a):
        self.__array_interface__ = a.__array_interface__


def test_address_of_an_array_interface(cfx):
    a = np.zeros(8, np.int32)
    assert cfx.host_address(Interface(a)) == cfx.host_address(a)


@pytest.mark.parametrize("a", [bytearray(64), array.array("i", range(16)), memoryview(bytearray(64)), b"0" * 64, [1, 2]], ids=lambda a: type(a).__name__)
def test_what_is_no_array_is_refused(cfx, a):
    with pytest.raises(AttributeError):
        cfx.host_address(a)
