"""The solvers' matrix copies where their build changes its course: rows of 1 to 70 entries with the
diagonal first, last and in the middle of its row, slices longer and shorter than what is staged,
and sizes around a slice of 32 rows. Every solver's solution of a diagonally dominant system
against a dense solve: with rows of |a_ii| >= 2 sum |a_ij| the error is at most
2 |residual| / min |a_ii|, and the residual at most 1e-11 |b|."""
import numpy as np
import pytest

import lsmps_b200 as lib

pytestmark = pytest.mark.gpu


def system(n, long_rows, seed):
    r = np.random.default_rng(seed)
    a = np.zeros((n, n))
    for i in range(n):
        k = min(n - 1, 70 if i < long_rows else int(r.integers(0, 6)))
        j = r.choice(np.delete(np.arange(n), i), k, replace=False)
        a[i, j] = r.uniform(-1, 1, k)
        a[i, i] = 2 * np.abs(a[i]).sum() + 1
    return a, r.normal(size=n)


@pytest.mark.parametrize("solver", ["fp64", "jacobi", "mixed"])
@pytest.mark.parametrize("n,long_rows", [(1, 0), (31, 31), (32, 0), (33, 32), (97, 97), (1000, 40), (1000, 0)])
def test_copies(built, solver, n, long_rows):
    a, b = system(n, long_rows, seed=n + long_rows)
    row = np.concatenate([[0], np.cumsum((a != 0).sum(1))]).astype(np.int64)
    i, j = np.nonzero(a)
    with lib.Context(0) as ctx:
        ctx.ppe_load_csr(row, j.astype(np.int32), a[i, j], b)
        p = ctx.ppe_solve(solver, 500, 1e-11)
        x = ctx.pressure(n)
    assert p.converged
    # converged: |r| <= tol max(1, |b|)
    bound = 2 * 1e-11 * max(1.0, np.linalg.norm(b)) / np.abs(np.diag(a)).min() + 1e-13 * np.abs(x).max()
    assert np.abs(x - np.linalg.solve(a, b)).max() <= bound
