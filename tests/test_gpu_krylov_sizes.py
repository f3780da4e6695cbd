"""The one-launch BiCGStab (krylov.cu) at the edges of its row partition: fewer slices than warps or
blocks, one row, a partial last slice, an odd number of rows (pairwise vector updates), a system
over all 148 blocks, 16-bit and 32-bit columns. Each solver reaches the solution of a diagonally
dominant system (against numpy's) to the residual tolerance times the condition number bound of a
dominant matrix, repeats its bits, and stops at an iteration cap."""
import numpy as np
import pytest

import lsmps_b200 as lib

pytestmark = pytest.mark.gpu
TOL = 1e-12


def system(n, spread, seed):
    """Rows of up to 12 entries: |j - i| <= spread, diagonal 1.5 times the row's off-diagonal sum."""
    rng = np.random.default_rng(seed)
    k = min(11, n - 1)
    off = rng.integers(1, max(spread, 2), (n, k)) * rng.choice([-1, 1], (n, k))
    col = (np.arange(n)[:, None] + off) % n
    val = -rng.uniform(0.1, 1.0, (n, k))
    val[col == np.arange(n)[:, None]] = 0
    keep = np.arange(k)[None, :] < rng.integers(min(1, k), k + 1, n)[:, None]
    diag = 1.5 * np.abs(np.where(keep, val, 0)).sum(1) + 1.0
    col = np.concatenate([np.where(keep, col, -1), np.arange(n)[:, None]], 1)
    val = np.concatenate([val, diag[:, None]], 1)
    live = col >= 0
    row = np.concatenate([[0], np.cumsum(live.sum(1))]).astype(np.int64)
    return row, col[live].astype(np.int32), val[live], rng.normal(size=n)


@pytest.mark.parametrize("solver", ["fp64", "jacobi", "mixed"])
@pytest.mark.parametrize("n", [1, 2, 31, 32, 33, 255, 257, 8191, 148 * 8 * 32 + 1, 200001])
def test_sizes(built, n, solver):
    import scipy.sparse as sp

    row, col, val, b = system(n, 50 if n % 2 else 10**9, n)
    A = sp.csr_matrix((val, col, row), shape=(n, n))  # sums duplicates, as the library does
    with lib.Context(0) as ctx:
        ctx.ppe_load_csr(row, col, val, b)
        st = ctx.ppe_solve(solver, 500, TOL)
        x = ctx.pressure(n)
        assert st.converged and st.iterations > 0
        bn = np.linalg.norm(b)
        # the FP64 residual, to rounding of A x (|A| |x| <= 3 |b| here)
        assert np.linalg.norm(b - A @ x) <= TOL * max(1.0, bn) + 1e-14 * bn
        for mode in (0, 1, 2):
            again = ctx.ppe_solve(solver, 500, TOL, use_graph=mode)
            assert again.iterations == st.iterations and np.array_equal(ctx.pressure(n), x)
        if st.iterations > 2:
            cap = ctx.ppe_solve(solver, 2, TOL)
            assert not cap.converged and cap.iterations == 2
        warm = ctx.ppe_solve(solver, 500, TOL)
        warm = ctx.ppe_solve(solver, 500, TOL, warm_start=True)
        assert warm.converged and warm.iterations <= 1
        none = ctx.ppe_solve(solver, 0, TOL)
        assert none.iterations == 0 and not none.converged
