"""Neighbor lists, classes and skin refreshes do not depend on the unit of length: any positive finite
radius is accepted, from where re^2 leaves the FP32 range at either end (1e-23, 2e19) to where it
nears the ends of the FP64 range, and radii about 1e18, the position the scan gives its empty lanes
in units of the radius. Lists and classes are integers: equal to the oracle's."""
import numpy as np
import pytest

import lsmps_b200 as lib
from _util import jittered_lattice
from oracle import Oracle

pytestmark = pytest.mark.gpu
SCALES = [1e-150, 1e-39, 1e-21, 1e-3, 3e17, 5e17, 1e18, 1e19, 1e39, 1e100, 1e150]


@pytest.mark.parametrize("l0", SCALES)
def test_scales(built, l0):
    re = 2.1 * l0
    xyz = (jittered_lattice(8, 0.2, seed=5) + np.array([0.0, 0.0, 1.0])) * l0
    t = np.where(np.arange(len(xyz)) % 5 == 4, lib.WALL, lib.INTERIOR).astype(np.uint8)
    moved = xyz + np.random.default_rng(1).uniform(-0.05, 0.05, xyz.shape) * l0
    row, col, trunc = Oracle.neighbors(xyz, re, 40)
    with lib.Context(0) as ctx:
        ctx.upload(xyz, t)
        st = ctx.build_neighbors(re, 40, l0)
        grow, gcol = ctx.neighbors(st.pairs)
        assert st.truncated == trunc and np.array_equal(grow, row) and np.array_equal(gcol, col)
        assert np.array_equal(ctx.types(), Oracle.classify(xyz, t, row, col, l0))
        ctx.build_neighbors_skin(re, 0.3 * l0, 128, 256, l0)
        ctx.update_positions(moved)
        st = ctx.refresh_neighbors()
        grow, gcol = ctx.neighbors(st.pairs)
        cls = ctx.types()
    row, col, _ = Oracle.neighbors(moved, re, 128)
    assert np.array_equal(grow, row)
    assert all(set(gcol[a:b]) == set(col[a:b]) for a, b in zip(row, row[1:]))
    assert np.array_equal(cls, Oracle.classify(moved, t, row, col, l0))
