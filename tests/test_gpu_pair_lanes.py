"""One and four lanes per particle in the pair kernels (csrc/lanes.cuh), at the
same sizes: the sums run in list order either way, so the lists and every field
are the same bits, on both paths and with both smoothing kernels.

The tanks do not fill their last warp or block (BSC_PAIR_LANES takes four lanes
above the sizes that the rule gives them to, and one below); some particles are
dead or buffer, and the porous layer and the free surface are in.
"""
import numpy as np
import pytest

from beach_slope_confined_gb300 import Solver, scenario as sc, setup_tank
from pairrun import sprinkle_flags

pytestmark = pytest.mark.gpu


def run(scen, P, lanes, monkeypatch):
    monkeypatch.setenv("BSC_PAIR_LANES", str(lanes))
    g = Solver(P)
    setup_tank(g, scen)
    info = g.step(2)
    out = g.download_state()
    lists = g.get_neighbors()
    g.close()
    return info.iterations, out, lists


@pytest.mark.parametrize("prec", ["fp64", "mixed"])
@pytest.mark.parametrize("dx,kernel", [(0.02, 1), (0.021, 0), (0.0064, 1)])
def test_lanes_keep_the_bits(dx, kernel, prec, monkeypatch):
    spec = sc.TankSpec(dx=dx, kernel=kernel, piston_ramp=0.0)
    scen = sprinkle_flags(sc.build(spec))
    P = sc.make_params(spec, scen.bounds, precision=prec, solver="fgmres", precond="mg", tol=1e-8, maxit=2000,
                       restart=40, inner_tol=1e-5, max_outer=60)
    (ia, a, la), (ib, b, lb) = (run(scen, P, lanes, monkeypatch) for lanes in (1, 4))
    assert ia == ib
    assert np.array_equal(la[0], lb[0]) and np.array_equal(la[1], lb[1])
    for f in a:
        assert np.array_equal(a[f], b[f]), f
