"""The Krylov solvers' reductions over awkward row counts.

The reductions take one block per 256 rows up to 912 blocks, and a thread
takes several rows beyond that; the counts here sit on both sides of a warp, a
block, and the largest grid.  The system is tridiagonal (-1/4, 1, -1/4): its
inverse's norm is at most 2 and ||A|| at most 1.5, so a stop at ||r|| <= 1e-12
||b|| leaves x within 2 * 1.5 * 1e-12 of the solution; 4e-12 leaves room for
the recurrences' drift.
"""
import numpy as np
import pytest

from beach_slope_confined_gb300 import scenario as sc, solve_csr

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
@pytest.mark.parametrize("n", [1, 31, 33, 255, 257, 1025, 131071, 912 * 256 - 1, 912 * 256 + 257])
def test_solve_over_row_counts(n, solver):
    x = np.random.default_rng(n).standard_normal(n)
    b = apply(n, x)
    P = sc.make_params(sc.TankSpec(), solver=solver, tol=1e-12, maxit=400, restart=30)
    rc, got, info = solve_csr(P, *tridiagonal(n), b, np.zeros(n))
    assert rc == 0 and info.converged
    assert np.linalg.norm(got - x) <= 4e-12 * np.linalg.norm(x)
