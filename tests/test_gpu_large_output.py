"""Recorded outputs above and below the size from which threads copy them: a
first output of more than 64 MiB, and small ones before and after 64 MiB have gone
out, equal the same outputs in pinned memory (one plain copy).
"""
import ctypes

import numpy as np
import pytest
import torch

from canard_b200 import api, cases

pytestmark = pytest.mark.gpu


def output_pinned(g):
    shape = (5,) + g.cases[0].blocks[0].shape
    pin = torch.empty(shape, dtype=torch.float32, pin_memory=True).numpy()
    ptr = (ctypes.POINTER(ctypes.c_float) * 1)(pin.ctypes.data_as(ctypes.POINTER(ctypes.c_float)))
    t = np.zeros(1)
    g._check(api.lib().canard_record_output(g.h, 0, ptr, api._dp(t)))
    return pin, float(t[0])


@pytest.mark.parametrize("n,outputs", [((152, 151, 149), 2), ((83, 71, 90), 8)])
def test_outputs_equal_plain_copies(n, outputs):
    cs = cases.tgv(nx=n[0], ny=n[1], nz=n[2])
    a, b = api.Context(cs), api.Context(cs)
    for g in (a, b):
        g.record_enable(True)
    total = 0
    for k in range(outputs):
        for g in (a, b):
            for _ in range(3 if k == 0 else 1):  # the first step's time step is zero
                g.step(1)
                g.record_accumulate()
        (x,), tx = a.record_output()
        y, ty = output_pinned(b)
        total += x.nbytes
        assert tx == ty and np.isfinite(x).all() and np.array_equal(x, y)
    assert total > 65 << 20
