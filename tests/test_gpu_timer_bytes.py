"""The contraction timer's byte count: a face that a call exchanges reads 12 values
and writes 3 (filter) per line; one that it does not reads one value and advances
its send chain.
"""
import pytest

from canard_b200 import api, cases

pytestmark = pytest.mark.gpu


def test_contraction_bytes_of_the_plain_filter():
    cs = cases.tgv(nx=20, ny=17, nz=14)
    g = api.Context(cs)
    g.set_timers(True)
    g.phase(api.PH_FILTER)
    x, y, z = 21, 18, 15
    lines = [y * z, x * z, x * y]
    per_field = sum(2 * 8 * (15 * lines[d] + 3 * (sum(lines) - lines[d])) for d in range(3))
    t = g.timers()["mpigo"]
    assert t["launches"] == 15 and t["bytes"] == 5 * per_field
