"""A one-launch solve whose barriers give up: every block leaves, the call returns the timeout
status, and the context goes on as before. The wait is made to run out by a limit of no polls."""
import numpy as np
import pytest

import lsmps_b200 as lib
from test_gpu_krylov_sizes import TOL, system

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("solver", ["fp64", "jacobi", "mixed"])
@pytest.mark.parametrize("n", [33, 8191, 148 * 8 * 32 + 1])
def test_wait_runs_out(built, n, solver):
    """one, a few and all blocks"""
    row, col, val, b = system(n, 50, n)
    with lib.Context(0) as ctx:
        ctx.ppe_load_csr(row, col, val, b)
        want = ctx.ppe_solve(solver, 500, TOL)
        x = ctx.pressure(n)
        ctx.set_wait_limit(0)
        for _ in range(2):
            with pytest.raises(lib.LsmpsError) as e:
                ctx.ppe_solve(solver, 500, TOL)
            assert e.value.code == lib.ERR_TIMEOUT
        ctx.set_wait_limit()
        again = ctx.ppe_solve(solver, 500, TOL)
        assert again.converged and again.iterations == want.iterations
        assert np.array_equal(ctx.pressure(n), x)
        with pytest.raises(lib.LsmpsError):
            ctx.set_wait_limit(-1)


@pytest.mark.parametrize("solver", ["fp64", "jacobi", "mixed"])
def test_no_solution_after_a_failed_solve(built, solver):
    """what a failed solve leaves is a partial (column-scaled) iterate: it is neither handed out as a
    solution nor continued by a warm start"""
    n = 8191
    row, col, val, b = system(n, 50, n)
    with lib.Context(0) as ctx:
        ctx.ppe_load_csr(row, col, val, b)
        cold = ctx.ppe_solve(solver, 500, TOL)
        x = ctx.pressure(n)
        for warm in (False, True):
            ctx.set_wait_limit(0)
            with pytest.raises(lib.LsmpsError):
                ctx.ppe_solve(solver, 500, TOL, warm_start=warm)
            ctx.set_wait_limit()
            with pytest.raises(lib.LsmpsError) as e:
                ctx.pressure(n)
            assert e.value.code == lib.ERR_STATE
            again = ctx.ppe_solve(solver, 500, TOL, warm_start=True)  # nothing to start from
            assert again.iterations == cold.iterations and np.array_equal(ctx.pressure(n), x)
            with pytest.raises(lib.LsmpsError):  # refused before anything is written: the solution stays
                ctx.ppe_solve(solver, 500, TOL, precond="multigrid")
            assert np.array_equal(ctx.pressure(n), x)
