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


@pytest.mark.parametrize("kernel", [0, 1])
@pytest.mark.parametrize("dx", [0.0068, 0.0064])
def test_lanes_per_particle_keep_the_bits(dx, kernel, monkeypatch):
    """The FP64 search by lanes and the one-thread FP64 phase over the
    warp-per-cell search's lists write the same lists and fields (a tank on
    each side of the 30000 particles up to which lanes share a particle)."""
    spec = sc.TankSpec(dx=dx, kernel=kernel, piston_ramp=0.0)
    scen = sc.build(spec)
    assert (scen.n <= 30000) == (dx > 0.0066)
    out = []
    for variant in ("thread", "warpcell"):
        monkeypatch.setenv("BSC_NEIGHBOUR", variant)
        g = Solver(sc.make_params(spec, scen.bounds, solver="fgmres", precond="mg", tol=1e-8, maxit=2000))
        setup_tank(g, scen)
        g.step(1)
        out.append((g.download_state(), g.get_neighbors()))
        g.close()
    (a, la), (b, lb) = out
    assert np.array_equal(la[0], lb[0]) and np.array_equal(la[1], lb[1])
    for f in ("x", "y", "vx", "vy", "p", "nut", "porosity", "L"):
        assert np.array_equal(a[f], b[f]), f
