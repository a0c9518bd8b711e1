"""The WCSPH step's polynomial EOS (whole gamma) against its general one.

A gamma one ulp above a whole number takes pow(); its own effect on the EOS is
a part in 10^15, so the two runs differ by the rounding of pow(q, gamma) - 1
only (a few parts in 10^13 of the pressure at the start), amplified over the
run as the comparison with the oracle allows: 1e-9 of the largest elevation,
1e-8 of the largest gradient.  The tanks meet every lane layout of the step's
kernels: eight lanes a particle below 10000 particles, four below 20000, one
above.
"""
import numpy as np
import pytest

from beach_slope_confined_gb300 import Solver, scenario as sc, setup_tank

pytestmark = pytest.mark.gpu


def run(dx, gamma, steps=12):
    spec = sc.TankSpec(dx=dx, dt=5e-5, por_cells=(16, 4))
    scen = sc.build(spec)
    g = Solver(sc.make_params(spec, scen.bounds))
    setup_tank(g, scen)
    wp, grid = sc.wcsph_params(spec, scen)
    wp.gamma = gamma
    g.wcsph_setup(wp)
    eta = g.wcsph_forward(steps, 5)
    w = np.random.default_rng(2).standard_normal(eta.shape)
    grad = g.wcsph_adjoint(w)
    g.close()
    return eta, grad


@pytest.mark.parametrize("dx,gamma", [(0.02, 7.0), (0.0095, 7.0), (0.0075, 7.0), (0.02, 1.0), (0.02, 8.0)])
def test_whole_gamma_equals_the_general_eos(dx, gamma):
    e0, g0 = run(dx, gamma)
    e1, g1 = run(dx, float(np.nextafter(gamma, 9.0)))
    assert np.max(np.abs(e0 - e1)) <= 1e-9 * np.max(np.abs(e1))
    assert np.max(np.abs(g0 - g1)) <= 1e-8 * np.max(np.abs(g1))
