"""The step path's forced points (GCBC layers and sponge) against the phases.

On the step path the right-hand side is summed inside the RK update, except at
the points GCBC or sponge change, which one launch gathers from all faces. Run
phase by phase (canard_phase) the same context sums everywhere first. Both have
to leave the same bits: with faces of one direction only, with faces that meet
at edges and corners (up to three reach a point), with curved interfaces
(partner amplitudes), with and without a sponge, and with blocks that no face
or sponge touches.
"""
import numpy as np
import pytest

from canard_b200 import api, cases

pytestmark = pytest.mark.gpu


def corner_block(sponge):
    cs = cases.vortex(26, 22, 18, sponge_cells=4)
    cs.blocks[0].nbc = [[cases.BC_NON_REFLECTIVE] * 2 for _ in range(3)]
    cs.blocks[0].mbcd = [[-1, -1] for _ in range(3)]
    cs.szco = 1.0 if sponge else 0.0
    return cs


CASES = {
    "one direction, sponge": lambda: cases.vortex(40, 20, 14, sponge_cells=6),
    "edges and corners, sponge": lambda: corner_block(True),
    "edges and corners": lambda: corner_block(False),
    "curved interfaces, sponge": lambda: cases.curvilinear_4block(24, 16, 14, sponge_cells=6),
    "blocks without forced points": lambda: cases.reference_toy(18, 16, 13),
    "validation": lambda: cases.reference_validation(20, 18, 13),
}


def by_phases(g, steps):
    for _ in range(steps):
        g.phase(api.PH_FILTER)
        g.phase(api.PH_COPYQO)
        for nk in range(1, 5):
            g.phase(api.PH_MOVEF_A, nk)
            g.phase(api.PH_PRIM)
            if nk == 1:
                g.phase(api.PH_TIMESTEP, 1)
            g.phase(api.PH_VISCOUS, nk)
            g.phase(api.PH_FLUXES, nk)
            g.phase(api.PH_GCBC, nk)
            g.phase(api.PH_SPONGE)
            g.phase(api.PH_RKUPDATE, nk)
            g.phase(api.PH_WALL, nk)
            g.phase(api.PH_AVERAGE)
        g.phase(api.PH_ADVANCE)


@pytest.mark.parametrize("name", list(CASES))
def test_step_equals_phases(name):
    cs = CASES[name]()
    a, b = api.Context(cs), api.Context(cs)
    a.step(4)
    by_phases(b, 4)
    for blk in range(len(cs.blocks)):
        assert np.array_equal(a.state(blk), b.state(blk)), (name, blk)
        for f in (api.F_DE, api.F_DRVA[0], api.F_DRVA[1], api.F_DRVA[2]):
            assert np.array_equal(a.field(f, blk), b.field(f, blk)), (name, blk, f)
