"""The CG's scalars where the squares of a system's residuals leave the normal
range of a double."""
import math

import numpy as np
import pytest

import helpers as H
import hykkt_gb300 as hk

pytestmark = pytest.mark.gpu


def _scaled(s, f):
    for v in ("rx", "rs", "ry", "ryd"):
        setattr(s, v, getattr(s, v) * f)
    return s


@pytest.mark.parametrize("n_bus", [60, 460, 900])
def test_right_hand_sides_near_the_smallest_doubles(n_bus):
    """Right-hand sides times 2^-k change the solution by that factor: bit for
    bit while r.r stays normal to the end; where its last values are subnormal
    (30 bits or more of them left) the run still ends, within an iteration."""
    make = lambda: H.small_grid_system(n_bus=n_bus, seed=8)  # noqa: E731
    p = hk.Plan(make())
    p.set_accuracy(500, 1e-11, 0, 1e-10)
    assert p.solve(make()) == hk.OK
    x, its, err = p.solution(), p.info()["cg_iterations"], p.info()["cg_residual"]
    last = 2.0 * math.log2(err)  # log2 of the final r.r
    for k in (100, int((last + 1010) / 2)):
        assert p.solve(_scaled(make(), 2.0 ** -k)) == hk.OK
        assert p.info()["cg_iterations"] == its
        assert all(np.array_equal(a * 2.0 ** -k, b) for a, b in zip(x, p.solution()))
    for k in (int((last + 1026) / 2) + 1, int((last + 1026) / 2) + 9):
        assert last - 2 * k + 1074 > 25
        assert p.solve(_scaled(make(), 2.0 ** -k)) == hk.OK
        assert abs(p.info()["cg_iterations"] - its) <= 1
        assert all(np.all(np.isfinite(b)) for b in p.solution())
