"""The skin refresh keeps, of a particle's candidates within the radius, the first max_neighbors in
candidate order (the list order at the positions the candidates were built at) and counts the rest:
rows, truncated count and classes against the oracle's candidate lists filtered by the moved distances.
Integers: equal."""
import numpy as np
import pytest

import lsmps_b200 as lib
from _util import jittered_lattice
from oracle import Oracle

pytestmark = pytest.mark.gpu
RE, SKIN, L0 = 2.1, 0.3, 1.0


@pytest.mark.parametrize("n", [1, 3, 4, 5, 31, 125, 343])
@pytest.mark.parametrize("maxn", [1, 3, 8, 17, 128])
def test_refresh_keeps_the_first(built, n, maxn):
    xyz = (jittered_lattice(7, 0.1, seed=3) + np.array([0.0, 0.0, 2.0]))[:n]
    t = np.where(np.arange(n) % 7 == 3, lib.WALL, lib.INTERIOR).astype(np.uint8)
    moved = xyz + np.random.default_rng(n).uniform(-0.05, 0.05, xyz.shape)
    crow, ccol, trunc = Oracle.neighbors(xyz, RE + SKIN, 256)
    assert trunc == 0
    want_row, want_col, dropped = [0], [], 0
    for i in range(n):
        c = ccol[crow[i]:crow[i + 1]]
        d = moved[c] - moved[i]
        c = c[(d[:, 0] * d[:, 0] + d[:, 1] * d[:, 1]) + d[:, 2] * d[:, 2] < RE * RE]
        want_col.extend(c[:maxn])
        want_row.append(len(want_col))
        dropped += max(len(c) - maxn, 0)
    with lib.Context(0) as ctx:
        ctx.upload(xyz, t)
        ctx.build_neighbors_skin(RE, SKIN, maxn, 256, L0)
        ctx.update_positions(moved)
        st = ctx.refresh_neighbors()
        row, col = ctx.neighbors(st.pairs)
        cls = ctx.types()
    assert np.array_equal(row, want_row) and np.array_equal(col, want_col)
    assert st.truncated == dropped
    assert np.array_equal(cls, Oracle.classify(moved, t, row, col, L0))
