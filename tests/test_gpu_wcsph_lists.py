"""The neighbour lists that a WCSPH run leaves in its context.

A run's steps build their lists in the buffers that the adjoint reads; what the
context offers afterwards has to be the lists of the last search that ran, the
one at the start of the last step.  They are compared, exactly, with all pairs
of the positions that this search saw: the run is deterministic and the piston
at rest, so those are the positions after one step fewer.  The particles start
off their lattice, with velocities that change the lists from step to step.
"""
import numpy as np
import pytest

from beach_slope_confined_gb300 import BscError, Solver, scenario as sc, setup_tank

pytestmark = pytest.mark.gpu


def tank():
    spec = sc.TankSpec(dx=0.02, dt=2e-4, por_cells=(16, 4), piston_amp=(0.0,))
    scen = sc.build(spec)
    fl = scen.tid == sc.TID_FLUID
    u = sc.splitmix64_uniform(5, 4 * scen.n).reshape(4, -1) - 0.5
    scen.x = scen.x + np.where(fl, 0.3 * spec.dx * u[0], 0.0)
    scen.y = scen.y + np.where(fl, 0.3 * spec.dx * u[1], 0.0)
    scen.vx = np.where(fl, 2.0 * u[2], 0.0)
    scen.vy = np.where(fl, 2.0 * u[3], 0.0)
    P = sc.make_params(spec, scen.bounds, precision="fp64")
    g = Solver(P)
    setup_tank(g, scen)
    return g, P, spec, scen


def all_pairs(x, y, H):
    off, ids = [0], []
    for i in range(x.size):
        dx, dy = x[i] - x, y[i] - y
        near = np.sqrt(dx * dx + dy * dy) < H
        near[i] = False
        ids.append(np.nonzero(near)[0])
        off.append(off[-1] + ids[-1].size)
    return np.array(off), np.concatenate(ids)


@pytest.mark.parametrize("steps,every,adjoint", [(6, 8, False), (6, 4, False), (6, 8, True), (6, 4, True)])
def test_lists_are_those_of_the_last_search(steps, every, adjoint):
    g, P, spec, scen = tank()
    for stage in (g.cellshift, g.neighbour, g.effpor, g.eddyvis, g.int_vel):
        stage()
    g.ppesolve()
    first = g.get_neighbors()
    g.wcsph_setup(sc.wcsph_params(spec, scen)[0])
    # an adjoint of several segments ends on the recomputation of the first
    ran = every if adjoint and every < steps else steps
    g.wcsph_forward(ran - 1, every)
    before = g.download_state()
    eta = g.wcsph_forward(steps, every)
    if adjoint:
        g.wcsph_adjoint(np.ones_like(eta))
    off, ids = g.get_neighbors()
    want = all_pairs(before["x"], before["y"], 2 * P.h)
    assert not np.array_equal(first[1], want[1])  # the motion has changed them
    assert np.array_equal(off, want[0]) and np.array_equal(ids, want[1])
    g.int_vel()
    g.comp_vel()
    s = g.download_state()
    assert np.isfinite(s["vx"]).all() and np.isfinite(s["vy"]).all()
    with pytest.raises(BscError):  # the matrix assembled before the run lay on other lists
        g.export_csr()
    g.close()
