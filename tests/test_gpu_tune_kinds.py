"""The line kinds the autotuner tries: every one is a kind that
canard_set_line_kind takes for that precision, group and direction, and the
kinds the public header names as candidates are among them.
"""
import numpy as np
import pytest

from canard_b200 import api, cases

pytestmark = pytest.mark.gpu

NAME = {v: k for k, v in api.Context.LINE_KINDS.items()}


def candidates(g, grp, d):
    out = np.zeros(32, np.int32)
    n = api.lib().canard_tune_kinds(g.h, grp, d, out.ctypes.data_as(api.ctypes.POINTER(api.ctypes.c_int32)), 32)
    assert n > 0
    kinds = [NAME[int(k)] for k in out[:n]]
    assert len(set(kinds)) == n
    return kinds


def documented(prec, grp, d, L):
    """include/canard_gpu.h, canard_autotune."""
    two_ended, quad = 32 <= L <= 881, L >= 4 * 60  # 881: the FP64 tile
    if prec == api.FP64:
        want = {"fp64"} | ({"fp64-tmem"} if d != 0 and 16 <= L <= 257 else set())
    elif prec == api.FP64_FAST:
        want = {"fp64", "fp64-one-lane", "fp64-split"} | ({"fp64-twist"} if two_ended else set())
        want |= {"fp64-quad"} if quad and grp != 0 else set()
    elif grp == 0:
        want = {"fp64-tile/fp32-split", "fp64-tile/fp32-one-lane", "fp64", "fp64-one-lane", "fp64-split"}
        want |= {"fp64-twist", "fp64-tile/fp32-twist"} if two_ended else set()
    else:
        want = {"fp32-split", "fp32-one-lane"} | ({"fp32-twist"} if two_ended else set())
        want |= {"fp32-quad"} if quad else set()
    return want


@pytest.mark.parametrize("L", [16, 20, 40, 250, 600, 1000])
@pytest.mark.parametrize("prec", [api.FP64, api.FP64_FAST, api.FP32_MIXED])
def test_candidates(prec, L):
    if prec == api.FP64 and L > 896:
        pytest.skip("longer than the plain path's line tile")
    for d in range(3):
        n = [15, 13, 14]
        n[d] = L - 1
        cs = cases.tgv(nx=16, ny=14, nz=13)
        b = cs.blocks[0]
        b.lxi, b.let, b.lze = n
        cs.xyz = cs.qa = None
        g = api.Context(cs, precision=prec, setup=False, upload_state=False)
        for grp, group in enumerate(("filter", "viscous", "flux")):
            kinds = candidates(g, grp, d)
            missing = documented(prec, grp, d, L) - set(kinds)
            assert not missing, (prec, group, d, L, missing)
            for k in kinds:
                g.set_line_kind(group, ("xi", "eta", "zeta")[d], k)  # raises where it is refused
            g.set_line_kind(group, ("xi", "eta", "zeta")[d], "default")
        g.close()


def test_autotuned_mixed_step():
    """A tuned mixed context steps on FP32 kinds and stays at FP32 rounding of the untuned one."""
    cs = cases.tgv(nx=40, ny=36, nz=33)
    a, b = (api.Context(cs, precision=api.FP32_MIXED) for _ in range(2))
    for row in b.autotune(2):
        if row["group"] != "filter":
            assert row["kind"].startswith("fp32"), row
    a.step(3)
    b.step(3)
    x, y = a.state(0), b.state(0)
    assert np.linalg.norm(x - y) <= 1e-6 * np.linalg.norm(x)
