"""The row product's kernel bench at a solve's blocks: a system without unknowns (no slice to cut),
fewer slices than one block's warps, and blocks on every SM."""
import numpy as np
import pytest

import lsmps_b200 as lib
from _util import jittered_lattice
from test_gpu_krylov_sizes import system

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kernel", [lib.KB_SPMV32, lib.KB_SPMV64])
def test_no_unknowns(built, kernel):
    xyz = jittered_lattice(4, 0.1)
    for n in (0, len(xyz)):  # nobody, walls only
        with lib.Context(0) as ctx:
            ctx.upload(xyz[:n], np.full(n, lib.WALL, np.uint8))
            ctx.build_neighbors(2.1, 128, 1.0)
            assert ctx.ppe_assemble("shifted", 10**9, 2.1, 1.0).unknowns == 0
            ms, nbytes = ctx.kernel_bench(kernel, 2)
            assert ms >= 0 and nbytes == 0


@pytest.mark.parametrize("kernel", [lib.KB_SPMV32, lib.KB_SPMV64])
@pytest.mark.parametrize("n", [1, 257, 200001])
def test_sizes(built, kernel, n):
    row, col, val, b = system(n, 50, n)
    with lib.Context(0) as ctx:
        ctx.ppe_load_csr(row, col, val, b)
        ms, nbytes = ctx.kernel_bench(kernel, 2)
        assert ms > 0 and nbytes > 0
        assert ctx.ppe_solve("mixed", 500, 1e-10).converged
