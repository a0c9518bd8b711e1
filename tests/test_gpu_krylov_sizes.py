"""The Krylov solvers' reductions over awkward row counts.

The reductions take one block per 256 rows up to 912 blocks, and a thread
takes several rows beyond that; the cooperative BiCGSTAB forms p and s on the
fly up to 20000 rows and holds one, two or three rows a thread up to 77824,
155648 and 233472 (on 152 SMs).  The counts here sit on both sides of a warp,
a block, and each of those lines.  The system is tridiagonal (-1/4, 1, -1/4): its
inverse's norm is at most 2 and ||A|| at most 1.5, so a stop at ||r|| <= 1e-12
||b|| leaves x within 2 * 1.5 * 1e-12 of the solution; 4e-12 leaves room for
the recurrences' drift.
"""
import numpy as np
import pytest

from beach_slope_confined_gb300 import Solver, scenario as sc, setup_tank, solve_csr

pytestmark = pytest.mark.gpu


def tridiagonal(n):
    row = np.repeat(np.arange(n), 3)
    col = row + np.tile([-1, 0, 1], n)
    val = np.tile([-0.25, 1.0, -0.25], n)
    keep = (col >= 0) & (col < n)
    rowptr = np.zeros(n + 1, np.int32)
    rowptr[1:] = np.cumsum(np.bincount(row[keep], minlength=n))
    return rowptr, col[keep].astype(np.int32), val[keep]


def apply(n, x):
    y = x.copy()
    y[1:] -= 0.25 * x[:-1]
    y[:-1] -= 0.25 * x[1:]
    return y


@pytest.mark.parametrize("solver", ["bicgstab", "fgmres"])
@pytest.mark.parametrize("n", [1, 31, 33, 255, 257, 1025, 12000, 20000, 20001, 77824, 77825, 131071, 155648, 155649, 912 * 256,
                               912 * 256 + 257])
def test_solve_over_row_counts(n, solver):
    x = np.random.default_rng(n).standard_normal(n)
    b = apply(n, x)
    P = sc.make_params(sc.TankSpec(), solver=solver, tol=1e-12, maxit=400, restart=30)
    rc, got, info = solve_csr(P, *tridiagonal(n), b, np.zeros(n))
    assert rc == 0 and info.converged
    assert np.linalg.norm(got - x) <= 4e-12 * np.linalg.norm(x)


def test_rows_too_long_for_shared_memory():
    """Row 0 couples to every unknown: its warp reads its rows from memory."""
    n = 5000
    rng = np.random.default_rng(1)
    rowptr, col, val = tridiagonal(n)
    w = rng.standard_normal(n - 2) * (0.1 / n)
    col = np.concatenate([col[:2], np.arange(2, n, dtype=np.int32), col[2:]])
    val = np.concatenate([val[:2], w, val[2:]])
    rowptr = rowptr + np.int32(n - 2) * (np.arange(n + 1) > 0).astype(np.int32)
    x = rng.standard_normal(n)
    b = apply(n, x)
    b[0] += w @ x[2:]
    P = sc.make_params(sc.TankSpec(), solver="bicgstab", tol=1e-12, maxit=400)
    rc, got, info = solve_csr(P, rowptr, col, val, b, np.zeros(n))
    assert rc == 0 and info.converged
    # row 0 changes A by less than 0.1 in norm: ||A^-1|| <= 2 / (1 - 0.2)
    assert np.linalg.norm(got - x) <= 5e-12 * np.linalg.norm(x)


@pytest.mark.parametrize("dx", [0.02, 0.009, 0.0075, 0.0038])
def test_cooperative_bicgstab_has_the_kernels_bits(dx, monkeypatch):
    """The per-kernel profiling keeps the five-kernel iteration: same pressures, bit for bit (tanks up to
    20000 rows, up to 77824, and beyond)."""
    spec = sc.TankSpec(dx=dx)
    scen = sc.build(spec)
    P = sc.make_params(spec, scen.bounds, solver="bicgstab", tol=1e-10, maxit=20000)
    out = []
    for profile in ("0", "1"):
        monkeypatch.setenv("BSC_PROFILE_ITER", profile)
        g = Solver(P)
        setup_tank(g, scen)
        info = g.step(2)
        out.append((info.iterations, g.download_state()))
        g.close()
    assert out[0][0] == out[1][0]
    for f in ("p", "vx", "vy", "x", "y"):
        assert np.array_equal(out[0][1][f], out[1][1][f]), f
