"""The recording's launch over all blocks and the threaded copy of large outputs.

* several cases (and a case of several blocks) recorded in one context give the
  same bits as each case recorded alone, also after the recording was restarted
  (record_enable while it is on);
* an output larger than the copy's chunk (2 MiB, odd remainder) that lands in
  pageable memory through several threads equals the one that goes straight into
  pinned memory, also from two contexts on two threads at once.
"""
import ctypes
import threading

import numpy as np
import pytest
import torch

from canard_b200 import api, cases

pytestmark = pytest.mark.gpu


def recorded(ctx, steps, ncases):
    ctx.record_enable(True)
    for _ in range(steps):
        ctx.step(1)
        ctx.record_accumulate()
    return [ctx.record_output(c) for c in range(ncases)]


@pytest.mark.parametrize("precision", [api.FP64, api.FP32_MIXED])
def test_cases_recorded_together_equal_alone(precision):
    cl = [cases.tgv(nx=20, ny=26, nz=17), cases.curvilinear_4block(22, 14, 13, sponge_cells=4),
          cases.tgv(nx=33, ny=18, nz=15, mach=0.3)]
    g = api.Context(cl, precision=precision)
    recorded(g, 2, len(cl))
    got = recorded(g, 3, len(cl))
    for c, cs in enumerate(cl):
        a = api.Context(cs, precision=precision)
        recorded(a, 2, 1)
        (arrays, t), = recorded(a, 3, 1)
        assert t == got[c][1]
        for x, y in zip(arrays, got[c][0]):
            assert np.array_equal(x, y)


def run_large(cs, out):
    g = api.Context(cs)
    g.record_enable(True)
    for _ in range(3):
        g.step(1)
        g.record_accumulate()
    # straight into pinned memory, on a context that has seen the same steps
    h = api.Context(cs)
    h.record_enable(True)
    for _ in range(3):
        h.step(1)
        h.record_accumulate()
    shape = (5,) + cs.blocks[0].shape
    pin = torch.empty(shape, dtype=torch.float32, pin_memory=True).numpy()
    ptr = (ctypes.POINTER(ctypes.c_float) * 1)(pin.ctypes.data_as(ctypes.POINTER(ctypes.c_float)))
    t = np.zeros(1)
    h._check(api.lib().canard_record_output(h.h, 0, ptr, api._dp(t)))
    (a,), ta = g.record_output()
    out.append((a, ta, pin, float(t[0])))


def test_large_output_copy():
    cl = [cases.tgv(nx=83, ny=71, nz=90), cases.tgv(nx=64, ny=95, nz=77, mach=0.2)]
    got = [[], []]
    threads = [threading.Thread(target=run_large, args=(cs, o)) for cs, o in zip(cl, got)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for o in got:
        a, ta, pin, tp = o[0]
        assert ta == tp and a.nbytes > 2 << 20
        assert np.isfinite(a).all() and np.array_equal(a, pin)
