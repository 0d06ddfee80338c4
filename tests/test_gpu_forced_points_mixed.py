"""The forced points' gather in mixed precision, and beside walls.

The mixed path's steps and phases form the fluxes differently (fused from the
primitives, or with stored stresses), so the step is compared with the FP64 step
within the mixed path's bound after a few steps (1e-5 per conserved variable);
with wall faces (their own branch of the wave amplitudes, edges where walls and
other boundaries meet) the FP64 step equals the phases bit for bit.
"""
import numpy as np
import pytest

from canard_b200 import api
from test_gpu_forced_points import CASES, by_phases
from test_gpu_mixed import state_errors
from test_gpu_parity import case_walls

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name", list(CASES))
def test_mixed_step_within_1e_5(name):
    cs = CASES[name]()
    a, b = api.Context(cs), api.Context(cs, precision=api.FP32_MIXED)
    a.step(4)
    b.step(4)
    for blk in range(len(cs.blocks)):
        errs = state_errors(b.state(blk), a.state(blk), 0.3)
        assert max(errs) <= 1e-5, (name, blk, errs)


def test_wall_step_equals_phases():
    cs = case_walls()
    a, b = api.Context(cs), api.Context(cs)
    a.step(4)
    by_phases(b, 4)
    assert np.array_equal(a.state(0), b.state(0))
    for f in (api.F_DE, api.F_DRVA[0], api.F_DRVA[1], api.F_DRVA[2]):
        assert np.array_equal(a.field(f, 0), b.field(f, 0)), f
