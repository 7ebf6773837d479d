"""The cluster PCG kernels of small reduced systems (at most 16 tile rows, 128
cameras) at the sizes where a class of kernel begins and ends, against the
FP64 iteration they restate; one size past the last goes to the persistent
kernel."""

from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def system(n, keep, seed):
    """A random SPD block system of n nodes, each pair coupled with
    probability `keep`, its condition number about 50."""
    rng = np.random.default_rng(seed)
    edges, off = [], []
    diag = np.zeros((n, 6, 6))
    for a in range(n):
        for b in range(a + 1, n):
            if rng.random() > keep:
                continue
            ga, gb = (np.eye(6) + 0.3 * rng.standard_normal((6, 6)) for _ in range(2))
            diag[a] += ga.T @ ga
            diag[b] += gb.T @ gb
            edges.append((a, b))
            off.append(-(gb.T @ ga))
    diag += np.eye(6) * (1.0 + 0.05 * np.trace(diag.mean(0)) / 6)
    off = np.array(off, np.float32).reshape(-1, 6, 6)
    edges = np.array(edges, np.uint32).reshape(-1, 2)
    return diag, edges, off, rng.standard_normal((n, 6))


def dense(diag, edges, off):
    n = len(diag)
    S = np.zeros((n, 6, n, 6))
    S[np.arange(n), :, np.arange(n), :] = diag
    for (a, b), o in zip(edges, off.astype(np.float64)):
        S[b, :, a, :] = o
        S[a, :, b, :] = o.T
    return S.reshape(6 * n, 6 * n)


def pcg64(S, diag, rhs, tol, cap):
    n = len(diag)
    inv = np.linalg.inv(diag)
    prec = lambda r: np.einsum("nab,nb->na", inv, r.reshape(n, 6)).reshape(-1)  # noqa: E731
    b = rhs.reshape(-1)
    x, r = np.zeros_like(b), b.copy()
    z = prec(r)
    p, rz = z.copy(), r @ z
    for k in range(cap):
        q = S @ p
        alpha = rz / (p @ q)
        x += alpha * p
        r -= alpha * q
        if np.linalg.norm(r) <= tol * np.linalg.norm(b):
            return x, k + 1
        z = prec(r)
        new = r @ z
        p, rz = z + (new / rz) * p, new
    return x, cap


@pytest.mark.parametrize("n", [1, 2, 5, 8, 15, 16, 17, 31, 32, 33, 63, 64, 65, 71, 127, 128, 129])
@pytest.mark.parametrize("keep", [1.0, 0.15])
def test_matches_the_fp64_iteration(solver, n, keep):
    diag, edges, off, rhs = system(n, keep, 7 * n)
    S = dense(diag, edges, off)
    x, it, rr = solver.reduced_solve(diag, edges, off, rhs, 1e-5, 300)
    ref, it_ref = pcg64(S, diag, rhs, 1e-5, 300)
    assert abs(it - it_ref) <= 1 and rr <= 1e-5
    # Both stop within 1e-5 |b| of the solution's residual: they differ by
    # at most twice that over the smallest eigenvalue, and FP32 rounding.
    lmin = np.linalg.eigvalsh(S)[0]
    bound = 2e-5 * np.linalg.norm(rhs) / lmin + 1e-5 * np.linalg.norm(ref)
    assert np.linalg.norm(x.reshape(-1) - ref) <= bound
    # A few iterations only: the iterates themselves, before rounding grows.
    if n >= 5:
        x3, it3, _ = solver.reduced_solve(diag, edges, off, rhs, 0.0, 3)
        ref3, _ = pcg64(S, diag, rhs, -1.0, 3)
        assert it3 == 3
        assert np.linalg.norm(x3.reshape(-1) - ref3) <= 1e-5 * np.linalg.norm(ref3)
    # The same bits on a repeated call.
    again, _, _ = solver.reduced_solve(diag, edges, off, rhs, 1e-5, 300)
    assert np.array_equal(again, x)


@pytest.mark.parametrize("n", [3, 20, 50, 100, 140])
def test_stopping_rules(solver, n):
    """Zero right-hand side, iteration cap 0 and 1, non-positive curvature
    (x stays at the last iterate) and NaN: as the persistent kernel."""
    diag, edges, off, rhs = system(n, 0.5, n)
    x, it, _ = solver.reduced_solve(diag, edges, off, 0.0 * rhs, 1e-6, 50)
    assert it == 0 and not x.any()
    x, it, _ = solver.reduced_solve(diag, edges, off, rhs, 1e-6, 0)
    assert it == 0 and not x.any()
    x, it, _ = solver.reduced_solve(diag, edges, off, rhs, 1e-12, 1)
    assert it == 1 and x.any()
    # Indefinite beyond the block diagonal: large couplings.
    x, it, _ = solver.reduced_solve(diag, edges, 100.0 * off, rhs, 1e-6, 50)
    assert it < 50 and np.isfinite(x).all()
    bad = rhs.copy()
    bad[0, 0] = np.nan
    x, it, _ = solver.reduced_solve(diag, edges, off, bad, 1e-6, 50)
    assert it == 0 and not x.any()
