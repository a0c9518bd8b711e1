"""Drag terms that are not finite outside the porous layer: at n = 1 the Ergun
terms carry the factor 1 - n = 0, which is a zero next to finite values and a
NaN next to others, in effpor's coefficient and in the WCSPH step, as in the
oracle.
"""
import numpy as np
import pytest

import oracle
from beach_slope_confined_gb300 import Solver, scenario as sc, setup_tank
from pairrun import make_pair, small_spec

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", ["fp64", "mixed"])
@pytest.mark.parametrize("case", ["plain", "d50", "alpha", "beta", "oden", "v"])
def test_effpor_coefficient(case, prec):
    scen = sc.build(small_spec())
    P = sc.make_params(small_spec(), scen.bounds, precision=prec)
    if case == "d50":
        P.d50 = 0.0
    if case in ("alpha", "beta"):
        setattr(P, {"alpha": "darcy_alpha", "beta": "forch_beta"}[case], np.inf)
    ctxs = make_pair(scen, P, Solver)
    st = ctxs[1].download_state()
    some = np.nonzero(st["tid"] == sc.TID_FLUID)[0][[50, 60, 900]]
    if case == "oden":
        st["oden"][some] = 0.0
    if case == "v":
        st["vx"][some] = [1e200, np.inf, np.nan]
        st["vy"][:] = 0.5
    got = []
    for ctx in ctxs:
        ctx.upload_state(st)
        ctx.effpor()
        got.append(np.isnan(ctx.download_state()["resist"]))
    assert got[1].any() == (case != "plain")
    assert np.array_equal(*got)


@pytest.mark.parametrize("d50", [0.0, 5e-3])
def test_wcsph_step(d50):
    spec = sc.TankSpec(dx=0.02, dt=2e-4, por_cells=(16, 4), d50=d50)
    scen = sc.build(spec)
    P = sc.make_params(spec, scen.bounds, precision="fp64")
    got = []
    for ctx in (Solver(P), oracle.context(P)):
        setup_tank(ctx, scen, initial_effpor=False)
        ctx.wcsph_setup(sc.wcsph_params(spec, scen)[0])
        ctx.wcsph_forward(1, 1)
        got.append(np.isnan(ctx.download_state()["vx"]))
        ctx.close()
    assert got[1].any() == (d50 == 0.0)
    assert np.array_equal(*got)
