"""The threaded copy of large outputs without a GPU (a stand-in for the device):
what happens where a worker's pinned buffer or stream
cannot be had, and that an error of a copy is reported.
"""
import ctypes

import numpy as np
import pytest

from canard_b200 import api

MIB = 1 << 20


def copy(nbytes, cores=16, opens=8, bad=-1):
    L = api.lib()
    L.canard_copy_out_host.argtypes = [ctypes.c_void_p, ctypes.c_void_p, ctypes.c_int64, ctypes.c_int32,
                                       ctypes.c_int32, ctypes.c_int64, ctypes.POINTER(ctypes.c_int32)]
    src = np.random.default_rng(nbytes % 1000).integers(0, 255, max(nbytes, 1), np.uint8)
    dst = np.zeros_like(src)
    used = ctypes.c_int32(-1)
    rc = L.canard_copy_out_host(src.ctypes.data, dst.ctypes.data, nbytes, cores, opens, bad, ctypes.byref(used))
    return rc, used.value, np.array_equal(src[:nbytes], dst[:nbytes])


@pytest.mark.parametrize("opens,workers", [(0, 0), (1, 0), (2, 2), (5, 5), (8, 8)])
@pytest.mark.parametrize("nbytes", [32 * MIB, 33 * MIB + 12])
def test_falls_back_where_a_worker_cannot_be_had(opens, workers, nbytes):
    assert copy(nbytes, opens=opens) == (0, workers, True)


def test_one_core_goes_straight():
    assert copy(40 * MIB, cores=1) == (0, 0, True)
    assert copy(40 * MIB, cores=0) == (0, 0, True)  # unknown


@pytest.mark.parametrize("bad", [0, 7, 19])
def test_error_is_reported(bad):
    rc, used, _ = copy(40 * MIB, bad=bad)
    assert rc == 7 and used == 8
