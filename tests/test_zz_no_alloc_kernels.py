"""The first bsc_csr_solve_noalloc call brings in every kernel that a later one
runs.

Under lazy module loading a kernel's code takes device memory when the kernel is
first used, and the solve takes other kernels for other sizes (and after a
barrier that gave up, or a breakdown).  A host makes one call and then gives the
rest of the device to its pool, so later calls must leave the free memory alone.
In a process of its own: elsewhere other tests have loaded the kernels.
"""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

SCRIPT = """
import ctypes, numpy as np, torch
from beach_slope_confined_gb300 import scenario as sc, solve_csr_noalloc
from test_gpu_krylov_sizes import apply, tridiagonal

def call(n, P):
    rowptr, col, val = tridiagonal(n)
    x = np.random.default_rng(n).standard_normal(n)
    d = [torch.from_numpy(a).cuda() for a in (rowptr, col, val, apply(n, x), np.zeros(n))]
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    rc, info = solve_csr_noalloc(P, n, *(t.data_ptr() for t in d), stream=torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    assert rc == 0 and info.converged
    return free - torch.cuda.mem_get_info()[0]

P = sc.make_params(sc.TankSpec(), solver="bicgstab", tol=1e-12, maxit=400)
call(FIRST, P)
print("changes", [call(n, P) for n in (12000, 40000, 131072)])
"""


@pytest.mark.parametrize("first", [300, 131072])
def test_later_sizes_leave_the_free_memory_alone(first):
    here = os.path.dirname(os.path.abspath(__file__))
    env = dict(os.environ, CUDA_MODULE_LOADING="LAZY",
               PYTHONPATH=os.pathsep.join([os.path.dirname(here), here, os.path.join(os.path.dirname(here), "oracle")]))
    r = subprocess.run([sys.executable, "-c", SCRIPT.replace("FIRST", str(first))], env=env, capture_output=True,
                       text=True, timeout=300)
    assert r.returncode == 0, r.stderr
    assert "changes [0, 0, 0]" in r.stdout, r.stdout
