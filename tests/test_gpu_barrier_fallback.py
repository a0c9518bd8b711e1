"""A cooperative BiCGSTAB launch whose grid barrier gives up (csrc/bicg_coop.cuh).

BSC_BARRIER_POLLS bounds the polls of a wait.  With 0 the first barrier runs
out in (almost) every block: x has not moved, and the five kernels that go on
from it have to give their own run's iterations and bits.  With a few polls
some barriers hold and the launch may end anywhere; the solve still converges,
to a pressure that both stops at 1e-10 put within 600 * 2e-10 of the other
(600: the Jacobi-scaled matrix's condition number at these spacings).  The
tanks take the merged form, and the forms with one and two rows per thread.
"""
import numpy as np
import pytest

from beach_slope_confined_gb300 import Solver, scenario as sc, setup_tank

pytestmark = pytest.mark.gpu


def pressure(dx):
    spec = sc.TankSpec(dx=dx)
    scen = sc.build(spec)
    g = Solver(sc.make_params(spec, scen.bounds, solver="bicgstab", tol=1e-10, maxit=20000))
    setup_tank(g, scen)
    info = g.step(1)
    p = g.download_state()["p"]
    g.close()
    assert info.converged
    return info.iterations, p


@pytest.mark.parametrize("dx", [0.02, 0.0075, 0.0038])
def test_the_kernels_go_on_from_x(dx, monkeypatch):
    monkeypatch.setenv("BSC_PROFILE_ITER", "1")  # the five kernels alone
    it, want = pressure(dx)
    monkeypatch.setenv("BSC_PROFILE_ITER", "0")
    for polls in (0, 2, 20):
        monkeypatch.setenv("BSC_BARRIER_POLLS", str(polls))
        k, p = pressure(dx)
        if polls == 0:
            assert k == it and np.array_equal(p, want)
        else:
            assert np.linalg.norm(p - want) <= 600 * 2e-10 * np.linalg.norm(want)
