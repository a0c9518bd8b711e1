"""The dense operator of the small multigrid levels against the single-CTA tail.

Both apply the same V-cycle, so the solves take the same iterations (one
apart at most: a residual may land on either side of the stop) and their
pressures agree to what the stops leave: twice the tolerance of 1e-10 times
the Jacobi-scaled matrix's condition number, about 600 at these spacings.
The tanks give grids whose first dense level is the only one, is level 1 with
odd sides, and lies under one or two levels of their own kernels.
"""
import numpy as np
import pytest

from beach_slope_confined_gb300 import Solver, scenario as sc, setup_tank

pytestmark = pytest.mark.gpu


def pressure(spec, prec):
    scen = sc.build(spec)
    P = sc.make_params(spec, scen.bounds, precision=prec, solver="fgmres", precond="mg", tol=1e-10, maxit=2000,
                       restart=40, inner_tol=1e-5, max_outer=60)
    g = Solver(P)
    setup_tank(g, scen)
    info = g.step(1)
    out = g.download_state()["p"]
    g.close()
    return info.iterations, out


@pytest.mark.parametrize("prec", ["fp64", "mixed"])
@pytest.mark.parametrize("dx,length", [(0.04, 0.8), (0.021, 1.7), (0.02, 4.0), (0.011, 4.0), (0.0063, 4.0)])
def test_dense_levels_equal_the_tail(dx, length, prec, monkeypatch):
    spec = sc.TankSpec(dx=dx, length=length, toe_x=0.5 * length)
    it, p = pressure(spec, prec)
    monkeypatch.setenv("BSC_MG_TAIL", "300")
    it_tail, p_tail = pressure(spec, prec)
    assert abs(it - it_tail) <= 1
    assert np.linalg.norm(p - p_tail) <= 600 * 2e-10 * np.linalg.norm(p_tail)
