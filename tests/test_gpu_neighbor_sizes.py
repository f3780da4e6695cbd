"""Neighbor lists and classes where the one-warp-per-cell scan changes its course: cells of 1, 2,
31, 32, 33 and 65 particles (one or two queries at a time, blocks of 32 queries), candidates just
below, at and above the 320 it holds at once, lists cut at max_neighbors within and across its
groups, pairs at the cut-off radius and with tied sectors; and the refresh of skin lists (four
particles per warp) of 1 to 9 particles and cut lists. Lists and classes are integers: equal to
the oracle's."""
import numpy as np
import pytest

import lsmps_b200 as lib
from _util import jittered_lattice
from oracle import Oracle

pytestmark = pytest.mark.gpu
RE, L0 = 2.1, 1.0


def check(ctx, xyz, t, maxn, re=RE):
    row, col, trunc = Oracle.neighbors(xyz, re, maxn)
    st = ctx.build_neighbors(re, maxn, L0)
    grow, gcol = ctx.neighbors(st.pairs)
    assert np.array_equal(grow, row) and np.array_equal(gcol, col) and st.truncated == trunc
    assert np.array_equal(ctx.types(), Oracle.classify(xyz, t, row, col, L0))


def cloud(per_cell, cells, seed):
    """cells of side RE along x with per_cell particles each, above the wall layer"""
    r = np.random.default_rng(seed)
    corner = np.repeat(np.arange(cells), per_cell)[:, None] * np.array([[RE, 0.0, 0.0]]) + np.array([[0.0, 0.0, 2 * RE]])
    xyz = corner + r.uniform(0.01, RE - 0.01, (per_cell * cells, 3))
    return xyz, np.where(np.arange(len(xyz)) % 5 == 4, lib.WALL, lib.INTERIOR).astype(np.uint8)


@pytest.mark.parametrize("per_cell", [1, 2, 31, 32, 33, 65, 106, 107, 120])
@pytest.mark.parametrize("maxn", [7, 40, 128])
def test_cell_scan_sizes(built, per_cell, maxn):
    xyz, t = cloud(per_cell, 3, seed=per_cell)
    with lib.Context(0) as ctx:
        ctx.upload(xyz, t)
        check(ctx, xyz, t, maxn)


@pytest.mark.parametrize("re", [2.0, 5.0 ** 0.5, 3.0])
def test_cut_off_and_ties(built, re):
    """an exact lattice: pairs at distance re, equal and zero components"""
    xyz = jittered_lattice(7, 0.0) + np.array([0.0, 0.0, 3.0])
    with lib.Context(0) as ctx:
        t = np.full(len(xyz), lib.INTERIOR, np.uint8)
        ctx.upload(xyz, t)
        check(ctx, xyz, t, 128, re)


@pytest.mark.parametrize("n", [1, 2, 3, 4, 5, 8, 9, 125])
@pytest.mark.parametrize("maxn", [3, 128])
def test_refresh_sizes(built, n, maxn):
    xyz = (jittered_lattice(5, 0.1, seed=3) + np.array([0.0, 0.0, 2.0]))[:n]
    t = np.where(np.arange(n) % 7 == 3, lib.WALL, lib.INTERIOR).astype(np.uint8)
    moved = xyz + np.random.default_rng(n).uniform(-0.05, 0.05, xyz.shape)
    with lib.Context(0) as ctx:
        ctx.upload(xyz, t)
        ctx.build_neighbors_skin(RE, 0.3, maxn, 128, L0)
        ctx.update_positions(moved)
        st = ctx.refresh_neighbors()
        row, col = ctx.neighbors(st.pairs)
        cls = ctx.types()
    full, fcol, _ = Oracle.neighbors(moved, RE, 128)
    # the same neighbors; the candidates' order is that of the positions the skin lists were built at
    for i in range(n):
        want, got = set(fcol[full[i]:full[i + 1]]), list(col[row[i]:row[i + 1]])
        assert len(set(got)) == len(got) == min(len(want), maxn) and set(got) <= want
    assert np.array_equal(cls, Oracle.classify(moved, t, row, col, L0))
