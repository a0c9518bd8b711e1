"""A cooperative BiCGSTAB launch whose grid barrier gives up (csrc/bicg_coop.cuh).

BSC_BARRIER_STUCK=1 starts the barrier's count out of the arrivals' reach: every
block's first wait runs out (a few tenths of a second) and the launch ends with x as it
was.  The five kernels that go on from there (their products are timed, those
of the cooperative form are not) have to give their own run's iterations and
bits, and so does the launch that holds.  The tanks take the merged form, and the
forms for up to 77824, 155648 and 233472 rows.
"""
import numpy as np
import pytest

from beach_slope_confined_gb300 import Solver, scenario as sc, setup_tank

pytestmark = pytest.mark.gpu


SPMV = 16  # timing slot


def pressure(dx):
    spec = sc.TankSpec(dx=dx)
    scen = sc.build(spec)
    g = Solver(sc.make_params(spec, scen.bounds, solver="bicgstab", tol=1e-10, maxit=20000))
    setup_tank(g, scen)
    info = g.step(1)
    p = g.download_state()["p"]
    timed = g.timings().calls[SPMV]
    g.close()
    assert info.converged
    return info.iterations, p, timed


@pytest.mark.parametrize("dx", [0.02, 0.0075, 0.0038, 0.0025])
def test_the_kernels_go_on_from_x(dx, monkeypatch):
    monkeypatch.setenv("BSC_PROFILE_ITER", "1")  # the five kernels alone
    it, want, _ = pressure(dx)
    monkeypatch.setenv("BSC_PROFILE_ITER", "0")
    k, p, timed = pressure(dx)
    assert timed == 0 and k == it and np.array_equal(p, want)
    monkeypatch.setenv("BSC_BARRIER_STUCK", "1")
    k, p, timed = pressure(dx)
    assert timed > 0 and k == it and np.array_equal(p, want)
