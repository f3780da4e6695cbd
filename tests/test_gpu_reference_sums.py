"""The REFERENCE solver's sequential-order sums, formed in parallel, keep the bits of sums added
one by one: BiCGStab on small systems against a numpy restatement whose dots are cumulative sums
and whose row products run in entry order. Sizes sit at the edges of the parallel sum (64 first
elements one by one, 1,024 threads, 7,168 elements per pass, several passes) and the entries'
lengths at those of the row product (32 entries per step); the right-hand sides cross binades,
tie, cancel, vanish and spread over many orders of magnitude."""
import numpy as np
import pytest

import lsmps_b200 as lib

pytestmark = pytest.mark.gpu


def seq(a):
    return np.cumsum(a)[-1]


def rows_times(lens, col, val, x):
    """Row products in entry order (col, val: rows x longest, padded)."""
    s = np.zeros(len(lens))
    for k in range(col.shape[1]):
        s = np.where(k < lens, s + val[:, k] * x[col[:, k]], s)
    return s


def bicgstab(lens, col, val, b, tol, most):
    """The reference's iteration; (iterations, converged, |b|, |Ax - b|, x)."""
    x, p, v = np.zeros_like(b), np.zeros_like(b), np.zeros_like(b)
    r, r0 = b.copy(), b.copy()
    bn = np.sqrt(seq(b * b))
    thresh = tol * max(1.0, bn)
    rho0 = alpha = omega = 1.0
    iters, conv = 0, False
    for it in range(most):
        rho = seq(r0 * r)
        if abs(rho) < 1e-30:
            break
        beta = (rho / rho0) * (alpha / omega)
        p = r + beta * (p - omega * v)
        v = rows_times(lens, col, val, p)
        den = seq(r0 * v)
        if abs(den) < 1e-30:
            break
        alpha = rho / den
        s = r - alpha * v
        if np.sqrt(seq(s * s)) <= thresh:
            x = x + alpha * p
            iters, conv = it + 1, True
            break
        t = rows_times(lens, col, val, s)
        tt = seq(t * t)
        if tt < 1e-30:
            break
        omega = seq(t * s) / tt
        x = x + (alpha * p + omega * s)
        r = s - omega * t
        iters = it + 1
        if np.sqrt(seq(r * r)) <= thresh:
            conv = True
            break
        if abs(omega) < 1e-30:
            break
        rho0 = rho
    d = rows_times(lens, col, val, x) - b
    return iters, conv, bn, np.sqrt(seq(d * d)), x


def rhs(kind, n, rng):
    if kind == "smooth":
        return np.sin(0.01 * np.arange(n)) + 0.3
    if kind == "signed":
        return rng.normal(size=n)
    if kind == "ties":  # few significant bits: half-way cases and exact cancellations
        return rng.integers(-64, 65, n) * 2.0 ** rng.integers(-27, 1, n)
    if kind == "spread":
        return rng.normal(size=n) * 10.0 ** rng.uniform(-60, 60, n)
    b = np.zeros(n)  # zero up to the last element
    b[-1] = 1.5
    return b


@pytest.mark.parametrize("kind", ["smooth", "signed", "ties", "spread", "last"])
@pytest.mark.parametrize("n", [1, 31, 64, 65, 1023, 1025, 3072, 7167, 7168, 7169, 16000])
def test_sequential_sums_bitwise(built, n, kind):
    rng = np.random.default_rng(n)
    lens = rng.integers(1, 4, n) if n < 40 else rng.choice([1, 2, 8, 27, 32, 33, 41], n)
    lens = np.minimum(lens, n)
    most = int(lens.max())
    col = rng.integers(0, n, (n, most))
    col[np.arange(n), lens - 1] = np.arange(n)  # the diagonal last, as the assembly stores it
    off = np.arange(most)[None, :] < (lens - 1)[:, None]
    col[off & (col == np.arange(n)[:, None])] = (np.nonzero(off & (col == np.arange(n)[:, None]))[0] + 1) % n
    if n == 1:
        off[:] = False
    val = np.where(off, -rng.uniform(0.1, 1.0, (n, most)), 0.0)
    val[np.arange(n), lens - 1] = 1.1 * lens + rng.uniform(0, 1, n)
    b = rhs(kind, n, rng)
    keep = np.arange(most)[None, :] < lens[:, None]
    row = np.concatenate([[0], np.cumsum(lens)]).astype(np.int64)
    with np.errstate(all="ignore"):
        want = bicgstab(lens, col, val, b, 1e-13, 6)
    with lib.Context(0) as ctx:
        ctx.ppe_load_csr(row, col[keep], val[keep], b)
        st = ctx.ppe_solve("reference", 6, 1e-13)
        x = ctx.pressure(n)
    assert (st.iterations, bool(st.converged)) == want[:2]
    assert st.initial_residual.hex() == float(want[2]).hex()
    assert st.final_residual.hex() == float(want[3]).hex()
    assert np.array_equal(x.view(np.int64), want[4].view(np.int64))
