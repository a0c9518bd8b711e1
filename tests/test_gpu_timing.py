"""bsc_get_timings over runs longer than the ring of events behind it.

Thirty steps record well over 512 events; every stage has to be counted once
per call, its time taken whole, and the stages of a step add up to the step
(they share their boundary events; 1 us of rounding per span is allowed for).
"""
import pytest

from beach_slope_confined_gb300 import Solver, scenario as sc, setup_tank

pytestmark = pytest.mark.gpu

CELLSHIFT, NEIGHBOUR, STEP, K_NEIGHBOUR = 1, 3, 15, 25
STAGES = [0, 1, 3, 4, 5, 6, 7, 8, 9, 10, 11, 12, 13, 14]  # those that follow one another in a step


@pytest.mark.parametrize("chunks", [[30], [1] * 30, [7, 23]])
def test_every_stage_counted_and_stages_fill_the_step(chunks):
    spec = sc.TankSpec(dx=0.02)
    scen = sc.build(spec)
    P = sc.make_params(spec, scen.bounds, solver="fgmres", precond="mg", tol=1e-8, maxit=2000, restart=40)
    g = Solver(P)
    setup_tank(g, scen)
    g.step(1)
    g.reset_timings()
    for k in chunks:
        g.step(k)
    t = g.timings()
    assert t.calls[STEP] == 30 and t.calls[NEIGHBOUR] == t.calls[CELLSHIFT] == t.calls[K_NEIGHBOUR] == 60
    stages = sum(t.ms[s] for s in STAGES)
    assert 0.0 < t.ms[K_NEIGHBOUR] <= t.ms[NEIGHBOUR] + 0.06
    assert abs(stages - t.ms[STEP]) <= 0.001 * sum(t.calls[s] for s in STAGES)
