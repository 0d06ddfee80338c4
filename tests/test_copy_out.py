"""The threaded copy of large outputs without a GPU (a stand-in for the device):
which outputs take it, what happens where a worker's pinned buffer or stream
cannot be had, and that an error of a copy is reported.
"""
import ctypes

import numpy as np
import pytest

from canard_b200 import api

MIB = 1 << 20


def copy(nbytes, before=0, cores=16, opens=8, bad=-1):
    L = api.lib()
    L.canard_copy_out_host.argtypes = [ctypes.c_void_p, ctypes.c_void_p, ctypes.c_int64, ctypes.c_int64, ctypes.c_int32,
                                       ctypes.c_int32, ctypes.c_int64, ctypes.POINTER(ctypes.c_int32)]
    src = np.random.default_rng(nbytes % 1000).integers(0, 255, max(nbytes, 1), np.uint8)
    dst = np.zeros_like(src)
    used = ctypes.c_int32(-1)
    rc = L.canard_copy_out_host(src.ctypes.data, dst.ctypes.data, nbytes, before, cores, opens, bad, ctypes.byref(used))
    return rc, used.value, np.array_equal(src[:nbytes], dst[:nbytes])


@pytest.mark.parametrize("opens,workers", [(0, 0), (1, 0), (2, 2), (5, 5), (8, 8)])
@pytest.mark.parametrize("nbytes", [64 * MIB, 65 * MIB + 12])
def test_falls_back_where_a_worker_cannot_be_had(opens, workers, nbytes):
    assert copy(nbytes, opens=opens) == (0, workers, True)


@pytest.mark.parametrize("nbytes,before,workers", [
    (2 * MIB + 4, 0, 0), (5 * MIB, 0, 0), (63 * MIB, 0, 0),   # first outputs: no set-up
    (5 * MIB, 58 * MIB, 0), (5 * MIB, 59 * MIB, 3),           # later ones, once 64 MiB have gone out
    (MIB, 64 * MIB, 0), (0, 64 * MIB, 0), (20 * MIB + 8, 64 * MIB, 8)])
def test_sizes(nbytes, before, workers):
    assert copy(nbytes, before) == (0, workers, True)


def test_one_core_goes_straight():
    assert copy(70 * MIB, cores=1) == (0, 0, True)
    assert copy(70 * MIB, cores=0) == (0, 0, True)  # unknown


@pytest.mark.parametrize("bad", [0, 17, 34])
def test_error_is_reported(bad):
    rc, used, _ = copy(70 * MIB, bad=bad)
    assert rc == 7 and used == 8
