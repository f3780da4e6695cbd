"""Separate contexts are independent: one-launch solves issued from several threads at the same time,
each on its own context, give the bits of solves issued one after another, whether the launches fit
the GPU together (32 blocks each) or each takes all of it (one block per SM); and a context whose
solves leave SMs free does not keep another one waiting."""
import threading

import numpy as np
import pytest

import lsmps_b200 as lib
from test_gpu_krylov_sizes import TOL, system

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [8191, 100001])
@pytest.mark.parametrize("solvers", [("fp64", "mixed"), ("jacobi", "mixed", "fp64")])
def test_concurrent_solves(built, n, solvers):
    row, col, val, b = system(n, 50, n)
    ctxs = [lib.Context(0) for _ in solvers]
    try:
        alone = []
        for ctx, solver in zip(ctxs, solvers):
            ctx.ppe_load_csr(row, col, val, b)
            st = ctx.ppe_solve(solver, 500, TOL)
            alone.append((st.iterations, ctx.pressure(n)))
            ctx.set_wait_limit(1 << 21)  # about a second
        together = [[] for _ in solvers]
        errors = []
        gate = threading.Barrier(len(solvers))

        def work(k):
            try:
                gate.wait(30)
                for _ in range(20):
                    st = ctxs[k].ppe_solve(solvers[k], 500, TOL)
                    together[k].append((st.iterations, ctxs[k].pressure(n)))
            except Exception as e:  # noqa: BLE001 (reported below)
                errors.append((solvers[k], e))

        threads = [threading.Thread(target=work, args=(k,)) for k in range(len(solvers))]
        for t in threads:
            t.start()
        for t in threads:
            t.join()
        assert not errors, errors
        for want, got in zip(alone, together):
            assert len(got) == 20
            for its, x in got:
                assert its == want[0] and np.array_equal(x, want[1])
    finally:
        for ctx in ctxs:
            ctx.close()


def test_free_sms_let_another_context_work(built):
    """a solve of some 150 ms (5,000 iterations on a 1-D Laplacian); list builds on another context, a
    millisecond each, end long before it"""
    n = 200_000
    i = np.arange(n)
    row = np.concatenate([[0], np.cumsum(np.where((i == 0) | (i == n - 1), 2, 3))]).astype(np.int64)
    col = np.concatenate([[0, 1], np.stack([i[1:-1] - 1, i[1:-1] + 1, i[1:-1]], 1).ravel(), [n - 2, n - 1]]).astype(np.int32)
    val = np.where(col == np.repeat(i, np.diff(row)), 2.0, -1.0)
    xyz, t, _ = lib.generate(None, case="rain_plate", particles=20_000, l0=1.0, seed=2)
    with lib.Context(0) as busy, lib.Context(0) as other:
        busy.ppe_load_csr(row, col, val, np.random.default_rng(0).normal(size=n))
        busy.set_free_sms(2)
        busy.ppe_solve("fp64", 10, 1e-12)
        other.upload(xyz, t)
        pairs = other.build_neighbors(2.1, 128, 1.0).pairs
        out = []
        solve = threading.Thread(target=lambda: out.append(busy.ppe_solve("fp64", 5000, 1e-12)))
        solve.start()
        for _ in range(5):
            assert other.build_neighbors(2.1, 128, 1.0).pairs == pairs
        during = solve.is_alive()
        solve.join()
        assert out[0].iterations == 5000 and during
        with pytest.raises(lib.LsmpsError):
            busy.set_free_sms(-1)
        with pytest.raises(lib.LsmpsError):
            busy.set_free_sms(10**6)


@pytest.mark.parametrize("free", [1, 2, 40, 147])
def test_free_sms_solve(built, free):
    import scipy.sparse as sp

    n = 100001
    row, col, val, b = system(n, 50, n)
    A = sp.csr_matrix((val, col, row), shape=(n, n))
    bn = np.linalg.norm(b)
    with lib.Context(0) as ctx:
        ctx.ppe_load_csr(row, col, val, b)
        ctx.set_free_sms(free)
        for solver in ("fp64", "jacobi", "mixed"):
            assert ctx.ppe_solve(solver, 500, TOL).converged
            assert np.linalg.norm(b - A @ ctx.pressure(n)) <= TOL * max(1.0, bn) + 1e-14 * bn
