"""The line kernel a fast or mixed-precision context takes without tuning, at the
line lengths where the choice changes: the default's results are those of the
kind that measured faster there, bit for bit, and not those of the other one
(the kinds round differently).
"""
import numpy as np
import pytest

from canard_b200 import api, cases

pytestmark = pytest.mark.gpu

FAST, MIXED = api.FP64_FAST, api.FP32_MIXED
ONE32, SPLIT32 = "fp32-one-lane", "fp32-split"
ONE64, SPLIT64, TWIST64 = "fp64-one-lane", "fp64-split", "fp64-twist"

# (precision, derivative 0 / filter 1, direction, line lengths of the blocks, default, the other kind)
CHOICES = [
    # FP32 derivatives: one-lane while four tiles fit an SM, then split, one-lane again where
    # only one of its tiles fits along eta and zeta
    (MIXED, 0, 1, (425,), ONE32, SPLIT32), (MIXED, 0, 1, (449,), SPLIT32, ONE32),
    (MIXED, 0, 1, (1025,), SPLIT32, ONE32), (MIXED, 0, 1, (1801,), SPLIT32, ONE32),
    (MIXED, 0, 2, (417,), ONE32, SPLIT32), (MIXED, 0, 2, (433,), SPLIT32, ONE32),
    (MIXED, 0, 3, (1537,), SPLIT32, ONE32), (MIXED, 0, 3, (1801,), ONE32, SPLIT32),
    (MIXED, 0, 2, (65,), ONE32, SPLIT32),
    # FP64, lines longer than the two-ended tile
    (FAST, 0, 1, (880,), TWIST64, SPLIT64), (FAST, 0, 1, (897,), SPLIT64, ONE64),
    (FAST, 0, 2, (890,), SPLIT64, ONE64), (FAST, 1, 1, (897,), SPLIT64, ONE64),
    (FAST, 1, 3, (890,), ONE64, SPLIT64), (MIXED, 1, 1, (897,), SPLIT64, ONE64),
    (MIXED, 1, 2, (890,), ONE64, SPLIT64),
    # FP64, a block with lines too short for the two-ended solve beside long ones
    (FAST, 0, 2, (257, 20), ONE64, SPLIT64), (FAST, 0, 2, (321, 20), SPLIT64, ONE64),
    (FAST, 1, 1, (385, 20), ONE64, SPLIT64), (FAST, 1, 1, (513, 20), SPLIT64, ONE64),
    (FAST, 1, 2, (641, 20), ONE64, SPLIT64),
    # short lines and the two-ended solve's range
    (FAST, 0, 3, (200,), ONE64, TWIST64), (FAST, 0, 3, (201,), TWIST64, ONE64),
    (FAST, 1, 2, (160,), ONE64, TWIST64), (MIXED, 1, 2, (161,), TWIST64, ONE64),
]


def context(prec, nn, lengths):
    cs = cases.tgv(nx=16, ny=14, nz=13)
    blocks = []
    for k, L in enumerate(lengths):
        n = [16, 14, 13]
        n[nn - 1] = L - 1
        per = cases.BC_PERIODIC
        blocks.append(cases.BlockSpec(*n, [[per, per]] * 3, [[k, k]] * 3))
    cs.blocks, cs.xyz, cs.qa = blocks, None, None
    return api.Context(cs, precision=prec, setup=False, upload_state=False)


@pytest.mark.parametrize("prec,op,nn,lengths,kind,other", CHOICES)
def test_default(prec, op, nn, lengths, kind, other):
    g = context(prec, nn, lengths)
    f = np.random.default_rng(lengths[0]).standard_normal((2,) + g.cases[0].blocks[0].shape)
    out = {}
    for k in ("default", kind, other):
        g.set_line_kind("flux" if op == 0 else "filter", ("xi", "eta", "zeta")[nn - 1], k)
        out[k], _ = g.line_bench(op, nn, f, reps=1)
    g.close()
    assert np.array_equal(out["default"], out[kind])
    assert not np.array_equal(out["default"], out[other])
