"""Coefficients that are not finite, or whose harmonic mean is 0/0, reach the
salinity flux of every pair, also of pairs of one concentration: the particles
whose concentration scalart and scalarupdate turn into a NaN are the oracle's.
"""
import numpy as np
import pytest

from beach_slope_confined_gb300 import Solver, scenario as sc
from pairrun import advance_to_lists, make_pair, small_spec

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("case", ["nan", "inf", "zero", "none"])
def test_nan_reaches_pairs_of_one_concentration(case):
    scen = sc.build(small_spec())
    P = sc.make_params(small_spec(), scen.bounds, salinity=True)
    if case == "zero":
        P.diffusivity = P.disp_long = P.disp_trans = 0.0
    ctxs = make_pair(scen, P, Solver)
    st = ctxs[1].download_state()
    fl = st["tid"] == sc.TID_FLUID
    st["con"] = np.where(fl, 0.5, 0.0)
    st["nut"] = np.zeros(fl.size)
    if case in ("nan", "inf"):
        st["nut"][np.nonzero(fl)[0][[100, 700]]] = getattr(np, case)
    got = []
    for ctx in ctxs:
        ctx.upload_state(st)
        advance_to_lists([ctx])
        ctx.effpor()
        ctx.scalart()
        ctx.scalarupdate(1.0)
        got.append(np.isnan(ctx.download_state()["con"]))
    assert got[1].any() == (case != "none")
    assert np.array_equal(*got)
