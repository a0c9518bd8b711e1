"""Row pointers that go backwards: such a row is empty, as a loop from rowptr[i]
to rowptr[i + 1] takes it.

The leading rows are a tridiagonal system (-1/4, 1, -1/4); the rows after them
have pointers that fall by two a row, a right-hand side of zero and a guess of
zero, so the solution is the leading system's.  The counts give every block of
the cooperative BiCGSTAB two 32-row units with entries and one without (14592
rows), and a form of one row per thread without the merged vectors (24320).  A
stop at ||r|| <= 1e-12 ||b|| leaves x within 2 * 1.5 * 1e-12 of the solution
(||A^-1|| <= 2, ||A|| <= 1.5); 4e-12 leaves room for the recurrences' drift.
"""
import numpy as np
import pytest

from beach_slope_confined_gb300 import scenario as sc, solve_csr_noalloc
from test_gpu_krylov_sizes import apply, tridiagonal

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,empty", [(9728, 4864), (16000, 8320)])
def test_rows_with_falling_pointers_are_empty(n, empty):
    import torch

    rowptr, col, val = tridiagonal(n)
    rowptr = np.concatenate([rowptr, rowptr[-1] - 2 * np.arange(1, empty + 1, dtype=np.int32)]).astype(np.int32)
    assert rowptr.min() >= 0
    x = np.random.default_rng(n).standard_normal(n)
    b = np.concatenate([apply(n, x), np.zeros(empty)])
    d = [torch.from_numpy(a).cuda() for a in (rowptr, col, val, b, np.zeros(n + empty))]
    P = sc.make_params(sc.TankSpec(), solver="bicgstab", tol=1e-12, maxit=400)
    rc, info = solve_csr_noalloc(P, n + empty, *(t.data_ptr() for t in d), stream=torch.cuda.current_stream().cuda_stream)
    got = d[4].cpu().numpy()
    assert rc == 0 and info.converged
    assert np.linalg.norm(got[:n] - x) <= 4e-12 * np.linalg.norm(x) and not got[n:].any()
