"""The averaging tables that the device reads (the list of points its last
averaging launch writes, one thread per point) without a GPU: every point stands
in the list once, the list holds exactly the averaged points and the other wall
points, and the averaging through the tables equals the averaging through the
plans bit for bit. Among the layouts are blocks whose faces carry a neighbour's
index without being averaged (walls or non-reflecting faces between blocks):
their shared edges are averaged points on no averaged face.
"""
import ctypes

import numpy as np
import pytest

from canard_b200 import api, cases

WALL_I, WALL_V = 20, 25
I64 = ctypes.POINTER(ctypes.c_int64)


def square(n, inner, outer=WALL_V, zeta_periodic=True):
    """2 x 2 blocks side by side in xi and eta; the faces between them carry the
    neighbour's index and code `inner`."""
    blocks = []
    for e in (0, 1):
        for x in (0, 1):
            me, nx, ne = 2 * e + x, 2 * e + 1 - x, 2 * (1 - e) + x
            nbc = [[inner, outer] if x else [outer, inner], [inner, outer] if e else [outer, inner],
                   [cases.BC_PERIODIC] * 2 if zeta_periodic else [WALL_I, cases.BC_NON_REFLECTIVE]]
            mbcd = [[nx, -1] if x else [-1, nx], [ne, -1] if e else [-1, ne], [me, me] if zeta_periodic else [-1, -1]]
            blocks.append(cases.BlockSpec(*n, nbc, mbcd))
    return cases.CaseSpec(blocks)


CASES = {
    "inner viscous walls": lambda: square((16, 16, 16), WALL_V),
    "inner inviscid walls": lambda: square((16, 16, 16), WALL_I, cases.BC_NON_REFLECTIVE),
    "inner non-reflecting faces": lambda: square((16, 16, 16), cases.BC_NON_REFLECTIVE),
    "inner code 40": lambda: square((16, 16, 16), 40),
    "uneven, inner viscous walls": lambda: square((40, 30, 20), WALL_V),
    "inner viscous walls, zeta ends": lambda: square((18, 13, 14), WALL_V, zeta_periodic=False),
    "straight interfaces, outer walls": lambda: square((17, 15, 13), cases.BC_INTER_STRAIGHT),
    "tgv": lambda: cases.tgv(nx=16, ny=18, nz=15),
    "toy": lambda: cases.reference_toy(18, 16, 13),
    "validation": lambda: cases.reference_validation(20, 18, 13),
    "curvilinear": lambda: cases.curvilinear_4block(24, 16, 14),
    "validation in sub-domains": lambda: cases.decompose(cases.reference_validation(48, 40, 12), [(2, 2, 1)]),
    "toy in sub-domains": lambda: cases.decompose(cases.reference_toy(52, 26, 12), [(4, 2, 1)] * 6),
}


def tables(cs, qa):
    _, blocks = api._structs([cs])
    _, args = keep = api._sub_args(cs)
    arrs = [np.ascontiguousarray(q).copy() for q in qa]
    ptrs = (ctypes.POINTER(ctypes.c_double) * len(arrs))(*[api._dp(a) for a in arrs])
    n, navg = ctypes.c_int64(), ctypes.c_int64()
    L = api.lib()
    L.canard_average_tables_host.argtypes = L.canard_average_host.argtypes + [I64, ctypes.c_int64, I64, I64]
    call = lambda out, cap: L.canard_average_tables_host(len(arrs), ctypes.cast(blocks, ctypes.c_void_p), *args, ptrs,
                                                         out, cap, ctypes.byref(n), ctypes.byref(navg))
    assert call(None, 0) == 0
    own = np.zeros(max(n.value, 1), np.int64)
    assert call(own.ctypes.data_as(I64), own.size) == 0
    del keep
    return arrs, own[:n.value].reshape(-1, 2), navg.value


def wall_points(cs):
    pts = set()
    for b, s in enumerate(cs.blocks):
        idx = np.arange(s.npts).reshape(s.shape)
        for d in range(3):
            for side in (0, 1):
                if s.nbc[d][side] in (WALL_I, WALL_V):
                    pts |= {(b, int(l)) for l in np.take(idx, -side, axis=2 - d).ravel()}
    return pts


@pytest.mark.parametrize("name", list(CASES))
def test_every_point_once(name):
    cs = CASES[name]()
    rng = np.random.default_rng(3)
    qa = [rng.standard_normal((5,) + s.shape) for s in cs.blocks]
    got, own, navg = tables(cs, qa)
    listed = [tuple(p) for p in own.tolist()]
    twice = len(listed) - len(set(listed))
    assert twice == 0, (name, twice)
    # a line's mean over the point alone is the point: the tables leave such targets out
    averaged = set()
    for kind in (api.PLAN_POINTS, api.PLAN_LINES, api.PLAN_SURFACE):
        src = api.plan_export(cs, kind + 3)
        for r, l, first, count in api.plan_export(cs, kind):
            if kind == api.PLAN_LINES and count in (1, 2, 4) and (src[first:first + count] == (r, l)).all():
                continue
            averaged.add((int(r), int(l)))
    assert set(listed[:navg]) == averaged
    assert set(listed[navg:]) == wall_points(cs) - averaged
    for a, b in zip(got, api.average_host(cs, qa)):
        assert np.array_equal(a, b)
