"""A node whose input is not a number is masked by the encoder's ReLU (max(NaN, 0) = 0), so it adds
nothing to the gradient: the gradient of the error loss stays finite."""
import numpy as np
import pytest

import lsmps_b200 as lib
from _util import jittered_lattice

pytestmark = pytest.mark.gpu


def test_masked_nodes_add_nothing(built):
    xyz = jittered_lattice(11, 0.1, seed=4)
    with lib.Context(0) as ctx:
        ctx.upload(xyz, np.zeros(len(xyz), np.uint8))
        ctx.build_neighbors(2.1, 128, 1.0)
        ctx.wls(2.1, 1.0, mode=1)
        st = ctx.ppe_assemble("wls", 10**9, 2.1, 1.0, diag_shift=0.0)
        ctx.ppe_manufacture(0.0, 1e307)  # b = A p* leaves the FP64 range in the upper layers
        b = ctx.ppe(st.unknowns, st.nnz)[3]
        assert 0 < np.count_nonzero(~np.isfinite(b)) < st.unknowns
        ctx.ppe_solve("jacobi", 0, 1e-10)  # x = 0: with |b| not finite the inputs are 0, and NaN where b is not finite
        ctx.mpnn_init(7)
        ctx.mpnn_add_sample()
        ctx.mpnn_train(steps=0, loss=0)
        _, g = ctx.mpnn_grad(0)
    assert np.isfinite(g).all() and np.count_nonzero(g)
