"""The decisions of the one-launch BiCGStab (krylov.cu): chunks, residual replacement, restart after a
stop that the FP64 residual denies, |s| test, breakdown, iteration cap and warm start, against a
numpy restatement of the loop on small diagonally dominant systems. Sums run in other orders there,
so a case is usable only where no decision is close: every comparison of a residual with its limit is
at least 1e-3 away (the two iterations drift apart by about 1e-6 of a residual that has fallen to 1e-10
of |b|), which the restatement asserts. Then iterations, replacements and restarts are equal; iterates stopped
by the cap agree to 1e-9 (up to six iterations of a system of condition 4 amplify 1e-16 by far less).

And the network's start: a guess or a correction worse than none is discarded, finite or not, from a cold
and from a warm start, after which the solve is the one without the network, bit for bit."""
import numpy as np
import pytest

import lsmps_b200 as lib
import mpnn_oracle as mo
from _util import jittered_lattice

pytestmark = pytest.mark.gpu


class Loop:
    """The iteration with A (FP64) or, MIXED, with the FP32 copy of A D^-1 and FP64 true residuals."""

    def __init__(self, A, b, solver):
        d = np.diag(A)
        self.b, self.mixed = b, solver == "mixed"
        self.dinv = np.ones_like(d) if solver == "fp64" else 1.0 / d
        self.A64 = A * self.dinv[None, :]
        self.A = self.A64.astype(np.float32).astype(np.float64) if self.mixed else self.A64

    def below(self, value, limit):
        assert value == 0 or abs(value / limit - 1) > 1e-3, "decision too close"
        return value <= limit

    def solve(self, max_iter, tol, x0=None, delta=0.01, chunk=8):
        b, A = self.b, self.A
        y = np.zeros_like(b) if x0 is None else x0 / self.dinv
        thresh = tol * max(1.0, np.linalg.norm(b))
        total = outer = guard = 0
        most = max_iter // chunk + 4 + max_iter
        left, start = max_iter, True
        while True:
            if start:  # (re)start from the true residual
                r = b - self.A64 @ y
                r0, p, v = r.copy(), np.zeros_like(b), np.zeros_like(b)
                rho = beta = r @ r
                rho0 = alpha = omega = 1.0
                rn = upd = np.sqrt(rho)
                it = base = in_chunk = 0
                start = False
                if self.below(rn, thresh):
                    return total, outer, True, y * self.dinv
                if abs(rho) < 1e-30:
                    return total, outer, False, y * self.dinv
                done = "cap" if left <= 0 else None
                if done and not (self.mixed and outer == 0):
                    return total, outer, False, y * self.dinv
            else:
                done = None
            if not done:
                p = r + beta * (p - omega * v)
                v = A @ p
                den = r0 @ v
                if abs(den) < 1e-30:
                    done = "break"
                else:
                    alpha = rho / den
                    s = r - alpha * v
                    if self.below(np.linalg.norm(s), thresh):
                        y, r, it, done = y + alpha * p, s, it + 1, "conv"
                    else:
                        t = A @ s
                        tt = t @ t
                        if tt < 1e-30:
                            done = "break"
                        else:
                            omega = (t @ s) / tt
                            y, r, it = y + (alpha * p + omega * s), s - omega * t, it + 1
                            rn, new = np.linalg.norm(r), r0 @ r
                            if self.below(rn, thresh):
                                done = "conv"
                            elif it >= left:
                                done = "cap"
                            elif abs(new) < 1e-30:
                                done = "break"
                            else:
                                beta = (new / rho) * (alpha / omega)
                                rho0, rho = rho, new
                in_chunk += 1
                if not done and in_chunk < chunk:
                    continue
                in_chunk = 0
                if not self.mixed:
                    if done:
                        return it, outer, done == "conv", y * self.dinv
                    continue
                total += it - base
                base = it
                if not done and not self.below(rn, delta * upd):
                    continue
            last = done == "cap" or total >= max_iter
            if done in (None, "cap") or last:  # replacement
                r = b - self.A64 @ y
                rn, new = np.linalg.norm(r), r0 @ r
                conv = self.below(rn, thresh)
                if last or conv:
                    return total, outer + (not last), conv, y * self.dinv
                beta, rho = (new / rho0) * (alpha / omega), new
                outer, upd, done = outer + 1, rn, "break" if abs(new) < 1e-30 else None
            if done:  # restart
                outer, guard, left, start = outer + 1, guard + 1, max_iter - total, True
                if guard >= most:
                    return total, outer, False, y * self.dinv


def system(n, seed, dominance=1.5):
    rng = np.random.default_rng(seed)
    A = np.where(rng.uniform(size=(n, n)) < 10 / n, -rng.uniform(0.1, 1.0, (n, n)), 0.0)
    np.fill_diagonal(A, 0)
    np.fill_diagonal(A, dominance * np.abs(A).sum(1) + rng.uniform(0.5, 1.5, n))
    return A, rng.normal(size=n)


def load(ctx, A, b):
    """rows with the diagonal last, as the library stores them"""
    rows = [[j for j in np.nonzero(A[i])[0] if j != i] + [i] for i in range(len(b))]
    row = np.concatenate([[0], np.cumsum([len(r) for r in rows])]).astype(np.int64)
    col = np.concatenate(rows).astype(np.int32)
    ctx.ppe_load_csr(row, col, A[np.repeat(np.arange(len(b)), np.diff(row)), col], b)


def compare(st, x, want, A, b, tol):
    its, outer, conv, xw = want
    assert (st.iterations, st.outer_iterations, bool(st.converged), st.fallback) == (its, outer, conv, 0)
    if conv:  # both residuals are below the limit
        assert np.linalg.norm(x - xw) <= 2 * tol * max(1.0, np.linalg.norm(b)) * np.linalg.norm(np.linalg.inv(A), 2)
    else:
        assert np.linalg.norm(x - xw) <= 1e-9 * np.linalg.norm(xw)


@pytest.mark.parametrize("n", [33, 300])
@pytest.mark.parametrize("delta", [0.5, 1e-2, 1e-30])  # often, sometimes, never replaced (denied, restarted)
@pytest.mark.parametrize("chunk", [1, 3, 8])
@pytest.mark.parametrize("cap", [0, 1, 3, 6, 500])
def test_mixed_decisions(built, n, delta, chunk, cap):
    A, b = system(n, 5)
    tol = 1e-9
    want = Loop(A, b, "mixed").solve(cap, tol, delta=delta, chunk=chunk)
    with lib.Context(0) as ctx:
        load(ctx, A, b)
        st = ctx.ppe_solve("mixed", cap, tol, inner_tol=delta, check_every=chunk)
        compare(st, ctx.pressure(n), want, A, b, tol)


@pytest.mark.parametrize("solver", ["fp64", "jacobi"])
@pytest.mark.parametrize("cap", [0, 1, 3, 500])
def test_plain_decisions(built, solver, cap):
    A, b = system(300, 5)
    want = Loop(A, b, solver).solve(cap, 1e-9)
    with lib.Context(0) as ctx:
        load(ctx, A, b)
        compare(ctx.ppe_solve(solver, cap, 1e-9), ctx.pressure(300), want, A, b, 1e-9)


@pytest.mark.parametrize("solver", ["jacobi", "mixed"])
def test_warm_start_decisions(built, solver):
    A, b = system(300, 5)
    loop = Loop(A, b, solver)
    with lib.Context(0) as ctx:
        load(ctx, A, b)
        ctx.ppe_solve(solver, 500, 1e-3)
        x = ctx.pressure(300)
        want = loop.solve(500, 1e-9, x0=x)
        compare(ctx.ppe_solve(solver, 500, 1e-9, warm_start=True), ctx.pressure(300), want, A, b, 1e-9)


def test_s_test_and_breakdown(built):
    """exact arithmetic: A = I stops at |s| = 0 and a restart confirms it; a singular A breaks down
    (r0.v = 0) at every restart until their number is bounded"""
    for A, b in ((np.eye(40), np.arange(1.0, 41.0)), (np.ones((2, 2)), np.array([1.0, -1.0]))):
        want = Loop(A, b, "mixed").solve(5, 1e-9, chunk=2)
        with lib.Context(0) as ctx:
            load(ctx, A, b)
            st = ctx.ppe_solve("mixed", 5, 1e-9, check_every=2)
            x = ctx.pressure(len(b))
        assert (st.iterations, st.outer_iterations, bool(st.converged)) == want[:3]
        assert np.array_equal(x, want[3])


@pytest.mark.parametrize("precond", ["jacobi", "multigrid"])
@pytest.mark.parametrize("warm", [False, True])
@pytest.mark.parametrize("bad", [1e6, np.inf, np.nan])
def test_bad_network_leaves_the_solve_without_it(built, precond, warm, bad):
    xyz = jittered_lattice(14, 0.1, seed=9)
    with lib.Context(0) as ctx:
        ctx.upload(xyz, np.zeros(len(xyz), np.uint8))
        ctx.build_neighbors(2.1, 128, 1.0)
        ctx.wls(2.1, 1.0, mode=1)
        st = ctx.ppe_assemble("wls", 10**9, 2.1, 1.0, diag_shift=0.0)
        ctx.mpnn_init(3)
        w = ctx.mpnn_weights()
        w[mo.OFF_WD:mo.OFF_WD + 64] *= bad
        ctx.mpnn_set_weights(w)
        out = {}
        for solver in ("mixed", "learned"):
            first = ctx.ppe_solve("mixed", 20000, 1e-2)
            assert first.converged
            s = ctx.ppe_solve(solver, 20000, 1e-10, warm_start=warm, precond=precond)
            assert s.converged and s.relative_l2_error <= 1e-8 and s.fallback == (solver == "learned")
            out[solver] = s.iterations, s.outer_iterations, ctx.pressure(st.unknowns).tobytes()
        assert out["learned"] == out["mixed"]
