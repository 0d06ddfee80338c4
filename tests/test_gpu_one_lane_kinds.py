"""The one-lane line solve's other kinds at the line lengths where its code paths
meet (see test_gpu_one_lane): the filter of the FP64 state with an FP32
elimination along all directions (along xi its increments go out by one bulk add
per line, the odd lines' padding element among them; one tensor box up to 254
points, bulk copies above), the FP64 kind with contraction along zeta, the FP32
derivative along eta.

Bounds: those of the existing tests of FP64 solves with contraction (1e-13) and
FP32 solves (5e-6); what the FP32 elimination computes is the filter's
increment, so the increment is held to the latter.
"""
import numpy as np
import pytest

import pyoracle as po
from canard_b200 import api
from test_gpu_mixed import rel_l2
from test_gpu_one_lane import DIRS, ETA, check, one_block

pytestmark = pytest.mark.gpu

XI = [13, 14, 16, 19, 128, 253, 254, 255, 256, 257, 508, 509]


@pytest.mark.parametrize("periodic", [True, False])
@pytest.mark.parametrize("nn", [1, 2, 3])
def test_filter_with_fp32_elimination(nn, periodic):
    for L in XI if nn == 1 else ETA:
        cs = one_block(nn, L, periodic)
        f = np.random.default_rng(L).standard_normal((2,) + cs.blocks[0].shape)
        g = api.Context(cs, precision=api.FP32_MIXED, setup=False, upload_state=False)
        g.set_line_kind("filter", DIRS[nn - 1], "fp64-tile/fp32-one-lane")
        out, _ = g.line_bench(1, nn, f, reps=1)
        g.close()
        o = po.Oracle(cs, setup=False)
        for k in range(2):
            a = f[k].ravel().copy()
            o.mpigo([a], 1, 1, 0, k + 1, k + 1)
            o.filte(0, a, {2: 1, 3: 2, 1: 3}[nn], k + 1)
            err = rel_l2(out[k].ravel() - f[k].ravel(), a - f[k].ravel())
            assert err <= 5e-6, (nn, L, k, err)


@pytest.mark.parametrize("periodic", [True, False])
@pytest.mark.parametrize("op", [0, 1])
def test_fast_along_zeta(op, periodic):
    for L in ETA:
        check(3, L, api.FP64_FAST, "fp64-one-lane", op, 1e-13, periodic)


@pytest.mark.parametrize("periodic", [True, False])
def test_fp32_along_eta(periodic):
    for L in ETA:
        check(2, L, api.FP32_MIXED, "fp32-one-lane", 0, 5e-6, periodic)


@pytest.mark.parametrize("periodic", [True, False])
def test_longest_lines(periodic):
    """Lines whose tile leaves the CTA's shared memory no room, or little, for staged factors."""
    for nn, L in ((1, 905), (1, 906), (2, 895), (2, 896), (3, 896)):
        for op in (0, 1):
            check(nn, L, api.FP64, "fp64", op, 0, periodic)
            check(nn, L, api.FP64_FAST, "fp64-one-lane", op, 1e-13, periodic)
    for nn, L in ((1, 1800), (1, 1801), (2, 1801), (3, 1801)):
        check(nn, L, api.FP32_MIXED, "fp32-one-lane", 0, 5e-6, periodic)
