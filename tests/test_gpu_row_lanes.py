"""The FGMRES passes with several lanes per row against BiCGSTAB's pressure.

Both solvers stop at 1e-10 of the right-hand side, so their pressures agree to
twice that times the Jacobi-scaled matrix's condition number, about 600 at
these spacings.  The tanks: a few hundred rows, rows that do not fill their
last warp, and both sides of the size up to which lanes share a row.
"""
import numpy as np
import pytest

from beach_slope_confined_gb300 import Solver, scenario as sc, setup_tank

pytestmark = pytest.mark.gpu


def pressure(spec, **kw):
    scen = sc.build(spec)
    g = Solver(sc.make_params(spec, scen.bounds, tol=1e-10, maxit=20000, **kw))
    setup_tank(g, scen)
    info = g.step(1)
    out = g.download_state()["p"]
    n = g.n
    g.close()
    assert info.converged
    return n, out


@pytest.mark.parametrize("kernel", [0, 1])
@pytest.mark.parametrize("dx,length", [(0.04, 0.8), (0.021, 1.7), (0.0083, 4.0), (0.0078, 4.0)])
def test_lanes_per_row(dx, length, kernel):
    spec = sc.TankSpec(dx=dx, length=length, toe_x=0.5 * length, kernel=kernel)
    n, want = pressure(spec, solver="bicgstab")
    assert (n <= 20000) == (dx > 0.008)
    mg = dict(solver="fgmres", precond="mg", restart=40, inner_tol=1e-5, max_outer=60)
    for prec in ("fp64", "mixed"):
        p = pressure(spec, precision=prec, **mg)[1]
        assert np.linalg.norm(p - want) <= 600 * 2e-10 * np.linalg.norm(want), prec
