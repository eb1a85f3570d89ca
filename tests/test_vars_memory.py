"""Which vars arrays the library writes in place: plain arrays in its layout, nothing else."""
from types import SimpleNamespace

import numpy as np
import pytest

N = 16


class Logged(np.ndarray):
    """An array type with its own idea of assignment."""

    def __setitem__(self, key, value):
        self.assigned = True
        super().__setitem__(key, value)


def _memory(pkg, array):
    return pkg._vars_memory(SimpleNamespace(n=N, vars=SimpleNamespace(ux=array)), 0)


def test_plain_arrays_are_written_in_place(pkg):
    a = np.zeros((N, N, N), np.float32, order="F")
    assert _memory(pkg, a) == a.ctypes.data


def _read_only():
    a = np.zeros((N, N, N), np.float32, order="F")
    a.flags.writeable = False
    return a


@pytest.mark.parametrize("array", [
    np.zeros((N, N, N), np.float32),
    np.zeros((N, N, N), np.float64, order="F"),
    np.zeros((N, N, N), ">f4", order="F"),
    np.zeros((2 * N, N, N), np.float32, order="F")[::2],
    np.zeros((N, N), np.float32, order="F"),
    _read_only(),
    # assignment through numpy clears the mask of a masked array and is the type's own for any other
    np.ma.array(np.zeros((N, N, N), np.float32, order="F"), mask=True),
    np.zeros((N, N, N), np.float32, order="F").view(Logged),
], ids=["C", "f64", "swapped", "strided", "2d", "read-only", "masked", "subclass"])
def test_other_arrays_take_the_copy(pkg, array):
    assert _memory(pkg, array) is None
