"""The one-lane line solve (k_line) at the line lengths where its code paths
meet: the shortest lines, every remainder of the blocks of eight rows, the
lengths where an xi tile goes from one tensor box to two (254 -> 255 FP64, 252
-> 253 FP32 points) and to bulk copies (508 -> 509, 504 -> 505), and the chunk
counts along eta and zeta; periodic lines and one-sided closures. The FP64 kind
of the plain path is compared bit for bit with the oracle, the fast mode's with
a few ulps of the field's scale, the FP32 ones with FP32 rounding (the bounds of
the two-ended solve's test).
"""
import numpy as np
import pytest

import pyoracle as po
from canard_b200 import api, cases
from test_gpu_mixed import rel_l2

pytestmark = pytest.mark.gpu

DIRS = ("xi", "eta", "zeta")
XI = [13, 14, 15, 16, 17, 18, 19, 20, 21, 28, 253, 254, 255, 256, 257, 508, 509, 510]
XI32 = [13, 16, 19, 22, 252, 253, 504, 505]
ETA = [13, 14, 15, 16, 17, 18, 19, 20, 36, 127, 128, 193, 260]


def one_block(nn, L, periodic):
    n = [17, 14, 13]
    n[nn - 1] = L - 1
    cs = cases.tgv(nx=n[0], ny=n[1], nz=n[2])
    if not periodic:
        cs.blocks[0].nbc[nn - 1] = [cases.BC_NON_REFLECTIVE] * 2
        cs.blocks[0].mbcd[nn - 1] = [-1, -1]
    return cs


def check(nn, L, prec, kind, op, tol, periodic):
    cs = one_block(nn, L, periodic)
    f = np.random.default_rng(L).standard_normal((2,) + cs.blocks[0].shape)
    g = api.Context(cs, precision=prec, setup=False, upload_state=False)
    g.set_line_kind("flux" if op == 0 else "filter", DIRS[nn - 1], kind)
    out, _ = g.line_bench(op, nn, f, reps=1)
    g.close()
    o = po.Oracle(cs, setup=False)
    for k in range(2):
        a = f[k].ravel().copy()
        if op == 0:
            o.mpigo([a], 0, 1, 0, k + 1, k + 1)
            ref = np.zeros_like(a)
            o.deriv(0, a, ref, nn, k + 1)
        else:
            o.mpigo([a], 1, 1, 0, k + 1, k + 1)
            o.filte(0, a, {2: 1, 3: 2, 1: 3}[nn], k + 1)
            ref = a
        err = rel_l2(out[k].ravel(), ref)
        if tol == 0:
            # the filter's third contracted value passes through the send chain: one
            # call from a zero chain is exact
            assert np.array_equal(out[k].ravel(), ref), (nn, L, kind, op, k, err)
        else:
            assert err <= tol, (nn, L, kind, op, k, err)


@pytest.mark.parametrize("periodic", [True, False])
@pytest.mark.parametrize("op", [0, 1])
def test_one_lane_plain_is_bit_exact(op, periodic):
    for L in XI:
        check(1, L, api.FP64, "fp64", op, 0, periodic)
    for nn in (2, 3):
        for L in ETA:
            check(nn, L, api.FP64, "fp64", op, 0, periodic)


@pytest.mark.parametrize("periodic", [True, False])
@pytest.mark.parametrize("op", [0, 1])
def test_one_lane_fast(op, periodic):
    for L in XI:
        check(1, L, api.FP64_FAST, "fp64-one-lane", op, 1e-13, periodic)
    for L in ETA:
        check(2, L, api.FP64_FAST, "fp64-one-lane", op, 1e-13, periodic)


@pytest.mark.parametrize("periodic", [True, False])
def test_one_lane_mixed(periodic):
    for L in XI32:
        check(1, L, api.FP32_MIXED, "fp32-one-lane", 0, 5e-6, periodic)
    for L in ETA:
        check(3, L, api.FP32_MIXED, "fp32-one-lane", 0, 5e-6, periodic)
