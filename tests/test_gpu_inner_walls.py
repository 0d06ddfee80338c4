"""Whole steps against the phases where a point is both averaged and reset by a
wall: 2 x 2 blocks whose inner faces are walls (or non-reflecting faces) that
carry the neighbour's index, so that the edge they share is averaged though its
faces are not. The step stores the averaged state and redoes the primitives in
one launch, one thread per point; the phases form all primitives anew. Both leave
the same bits.
"""
import numpy as np
import pytest

from canard_b200 import api, cases
from test_average_tables import WALL_I, WALL_V, square
from test_gpu_forced_points import by_phases

pytestmark = pytest.mark.gpu

LAYOUTS = {
    "viscous walls": ((16, 16, 16), WALL_V, WALL_V),
    "uneven, viscous walls": ((40, 30, 20), WALL_V, WALL_V),
    "inviscid walls": ((21, 14, 13), WALL_I, cases.BC_NON_REFLECTIVE),
    "non-reflecting faces": ((16, 18, 13), cases.BC_NON_REFLECTIVE, WALL_V),
    "straight interfaces": ((17, 15, 13), cases.BC_INTER_STRAIGHT, WALL_V),
}


def flow(name):
    n, inner, outer = LAYOUTS[name]
    cs = square(n, inner, outer)
    cs.amach, cs.cfl, cs.reoo = (0.2, 0.0, 0.0), 0.5, 400.0
    cs.xyz, cs.qa = [], []
    for b, s in enumerate(cs.blocks):
        x, y, z = (np.linspace(o, o + 1.0, k + 1) for o, k in ((b % 2, s.lxi), (b // 2, s.let), (0.0, s.lze)))
        Z, Y, X = np.meshgrid(z, y, x, indexing="ij")
        cs.xyz.append(np.stack([X, Y, Z]))
        rho = 1.0 + 0.02 * np.cos(np.pi * X) * np.cos(np.pi * Y) + 0.01 * np.cos(2 * np.pi * Z)
        u, v, w = 0.02 * np.sin(np.pi * Y), 0.03 * np.sin(np.pi * X), 0.02 * np.sin(2 * np.pi * Z)
        p = rho ** 1.4 / 1.4
        cs.qa.append(np.stack([rho, rho * u, rho * v, rho * w, p / 0.4 + 0.5 * rho * (u * u + v * v + w * w)]))
    return cs


@pytest.mark.parametrize("name", list(LAYOUTS))
def test_step_equals_phases(name):
    cs = flow(name)
    a, b = api.Context(cs), api.Context(cs)
    a.step(4)
    by_phases(b, 4)
    for blk in range(len(cs.blocks)):
        assert np.isfinite(a.state(blk)).all()
        assert np.array_equal(a.state(blk), b.state(blk)), (name, blk)
        assert np.array_equal(a.field(api.F_P, blk), b.field(api.F_P, blk)), (name, blk)

