"""All-particle WLS of caller fields at the edges of its one-warp blocks (1, 31, 32, 33, 95 and
125 particles) for one to three fields, in the caller's order: solutions against the oracle to
1e-8 relative per particle (as test_gpu_projection), zeros where there is no system; and the
analytic fields of both precisions on the same sets reproduce the quadratic's derivatives."""
import numpy as np
import pytest

import lsmps_b200 as lib
from _util import jittered_lattice
from oracle import Oracle

pytestmark = pytest.mark.gpu
RE, L0 = 2.1, 1.0


@pytest.mark.parametrize("fields", [1, 2, 3])
@pytest.mark.parametrize("n", [1, 31, 32, 33, 95, 125])
def test_wls_fields_sizes(built, n, fields):
    xyz = jittered_lattice(5, 0.1, seed=3)[np.random.default_rng(n).permutation(125)][:n]
    t = np.where(np.arange(n) % 7 == 3, lib.WALL, lib.INTERIOR).astype(np.uint8)
    f = np.random.default_rng(1).normal(size=(n, fields))
    quads = np.array([lib.REF_QUADRATIC, [0, 1, 0, 2, 0, 0.3, 0, 0.1, 0, 0], [1, 0, -1, 0, 0.2, 0, 0.4, 0, 0.3, 0]])
    row, col, _ = Oracle.neighbors(xyz, RE, 128)
    cls = Oracle.classify(xyz, t, row, col, L0)
    want, st = Oracle.wls_fields(xyz, cls, row, col, RE, L0, f)
    ok = (st == 0) | (st == 1)
    with lib.Context(0) as ctx:
        ctx.upload(xyz, t)
        ctx.build_neighbors(RE, 128, L0)
        assert np.array_equal(cls, ctx.types())
        got = ctx.wls_fields(f).cpu().numpy()
        analytic = []
        for precision in (0, 1):
            ctx.wls(RE, L0, mode=1, coef=quads[:fields], precision=precision, store=True)
            analytic.append(ctx.wls_result(fields, with_x=True)[:2])
    assert got.shape == (n, fields, 9) and np.all(got[~ok] == 0)
    scale = np.abs(want).max(axis=(1, 2))[:, None, None] + 1e-30
    assert np.all(np.abs(got - want)[ok] <= 1e-8 * scale[ok])
    x, y, z = xyz.T
    for sol, status in analytic:
        assert np.array_equal((status == 0) | (status == 1), ok) and np.all(sol[~ok] == 0)
        good = status == 0
        for k, c in enumerate(quads[:fields]):
            grad = np.stack([c[1] + 2 * c[4] * x + c[7] * y + c[8] * z, c[2] + 2 * c[5] * y + c[7] * x + c[9] * z,
                             c[3] + 2 * c[6] * z + c[8] * x + c[9] * y], 1)
            # 1e-6: rounding of the moments times the condition of one-sided stencils (<= 1e9)
            assert np.all(np.abs(sol[good, k, :3] - grad[good]) <= 1e-6 * (1 + np.abs(grad[good]).max(initial=0)))
