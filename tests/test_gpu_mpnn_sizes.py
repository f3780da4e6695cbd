"""Loss and gradient of the network at the edges of the backward kernels' tiles: 16-node tiles of
the layers, 64-node tiles of the weight gradient (one more than its 296 blocks hold at once),
eight rows per block of the per-node sums. Against the numpy oracle, to BF16 rounding (the
tolerances of test_gpu_mpnn: 2e-2 for the loss, 3e-2 of the gradient's norm)."""
import numpy as np
import pytest

import lsmps_b200 as lib
import mpnn_oracle as mo
from _util import jittered_lattice
from test_gpu_mpnn import oracle_graph

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("unknowns", [1, 2, 15, 17, 63, 64, 65, 300, 64 * 296 + 65])
def test_gradient_at_tile_edges(built, unknowns):
    xyz = jittered_lattice(11 if unknowns <= 300 else 30, 0.1, seed=4)
    with lib.Context(0) as ctx:
        ctx.upload(xyz, np.zeros(len(xyz), np.uint8))
        ctx.build_neighbors(2.1, 128, 1.0)
        ctx.wls(2.1, 1.0, mode=1)
        st = ctx.ppe_assemble("wls", unknowns, 2.1, 1.0, diag_shift=0.0)
        assert st.unknowns == unknowns
        ctx.ppe_manufacture(0.3, 0.05, [(1.0, 0.2, -0.1, 0.15, 0.3)])
        assert ctx.ppe_solve("jacobi", 20000, 1e-10).converged
        ctx.mpnn_init(7)
        ctx.mpnn_add_sample()
        ctx.mpnn_train(steps=0, loss=2)
        loss, g = ctx.mpnn_grad(0)
        G, r, t = oracle_graph(ctx, st)
        for k in ("src", "dst"):
            G[k] = G[k].astype(np.int64)
        l_orc, g_orc, _ = mo.loss_and_grad(ctx.mpnn_weights(), G, r, t, kind=2)
    assert loss == pytest.approx(l_orc, rel=2e-2)
    assert np.linalg.norm(g - g_orc) <= 3e-2 * np.linalg.norm(g_orc)
