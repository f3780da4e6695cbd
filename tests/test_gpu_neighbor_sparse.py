"""List builds on grids with far more cells than particles: isolated particles, pairs across cell faces
and a crowded cell (several blocks of 32 queries) in the corners of a grid of millions of cells. Lists
and classes are integers: equal to the oracle's."""
import numpy as np
import pytest

import lsmps_b200 as lib
from oracle import Oracle

pytestmark = pytest.mark.gpu
RE = 2.1


@pytest.mark.parametrize("side", [1, 30, 250])
@pytest.mark.parametrize("n", [1, 31, 33, 257, 5000])
def test_sparse_grid(built, n, side):
    r = np.random.default_rng(n)
    far = side * RE
    xyz = r.uniform(0, far, (n, 3))
    crowd = np.clip(far - RE, 0, None) + r.uniform(0.01, RE - 0.01, (100, 3))
    faces = np.stack([np.full(8, RE * (side // 2)) + np.linspace(-0.4, 0.4, 8), np.full(8, 0.5), np.full(8, 3.0)], 1)
    xyz = np.concatenate([xyz, crowd, faces])
    t = np.where(np.arange(len(xyz)) % 5 == 4, lib.WALL, lib.INTERIOR).astype(np.uint8)
    row, col, trunc = Oracle.neighbors(xyz, RE, 40)
    with lib.Context(0) as ctx:
        ctx.upload(xyz, t)
        st = ctx.build_neighbors(RE, 40, 1.0)
        grow, gcol = ctx.neighbors(st.pairs)
        assert np.array_equal(grow, row) and np.array_equal(gcol, col) and st.truncated == trunc
        assert np.array_equal(ctx.types(), Oracle.classify(xyz, t, row, col, 1.0))
