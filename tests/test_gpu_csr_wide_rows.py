"""CSR systems whose entries do not fit the cooperative BiCGSTAB's shared memory:
a quarter of it holds rows, the others are read from memory.

Band matrices, 1 on the diagonal and -1/(4 k) on k diagonals each side: the
off-diagonal part has norm 1/2 at most, so ||A^-1|| <= 2, ||A|| <= 1.5, and a
stop at ||r|| <= 1e-12 ||b|| leaves x within 3e-12 of the solution; 4e-12 leaves
room for the recurrences' drift.  The row counts take each form of the kernel
(up to 20000, 77824, 155648 and 233472 rows) and the kernels beyond, with bands
that leave ragged batches of a row's entries.
"""
import numpy as np
import pytest

from beach_slope_confined_gb300 import scenario as sc, solve_csr

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,k", [(12000, 61), (30000, 53), (125000, 30), (160000, 27), (235000, 22)])
def test_wide_bands(n, k):
    rows = np.repeat(np.arange(n), 2 * k + 1)
    cols = rows + np.tile(np.arange(-k, k + 1), n)
    ok = (cols >= 0) & (cols < n)
    rowptr = np.zeros(n + 1, np.int32)
    rowptr[1:] = np.cumsum(np.bincount(rows[ok], minlength=n))
    val = np.where(rows == cols, 1.0, -0.25 / k)[ok]
    x = np.random.default_rng(n).standard_normal(n)
    s = np.concatenate([[0.0], np.cumsum(x)])  # band sums by differences of the running sum
    lo, hi = np.maximum(np.arange(n) - k, 0), np.minimum(np.arange(n) + k + 1, n)
    b = x - (0.25 / k) * (s[hi] - s[lo] - x)
    P = sc.make_params(sc.TankSpec(), solver="bicgstab", tol=1e-12, maxit=400)
    rc, got, info = solve_csr(P, rowptr, cols[ok].astype(np.int32), val, b, np.zeros(n))
    assert rc == 0 and info.converged
    assert np.linalg.norm(got - x) <= 4e-12 * np.linalg.norm(x)
