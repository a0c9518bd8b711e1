"""scalart's pair rules on the GPU (csrc/scalar.cu) against the oracle, over
concentration fields that take each of them: pairs of one concentration (no
flux, skipped), pairs on a jump, pairs that all differ.

Both sides run the same routines on the same uploaded state, so they differ by
the rounding of a pair's term (some 15 operations, 2e-15 of it) and of the sum
over a particle's neighbours, whose signed terms largely cancel on a smooth
field: 1e-11 of the largest flux allows a cancellation of 5000.
"""
import numpy as np
import pytest

from beach_slope_confined_gb300 import Solver, scenario as sc
from pairrun import advance_to_lists, make_pair, small_spec

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("field", ["one", "jump", "ramp"])
@pytest.mark.parametrize("nut", [0.0, 1e-4])
def test_flux_by_concentration_field(field, nut):
    scen = sc.build(small_spec())
    P = sc.make_params(small_spec(), scen.bounds, salinity=True)
    ctxs = make_pair(scen, P, Solver)
    st = ctxs[1].download_state()
    fl = st["tid"] == sc.TID_FLUID
    x = st["x"]
    con = {"one": np.full(x.size, 0.5), "jump": np.where(x < np.median(x[fl]), -0.5, 0.5), "ramp": np.sin(3 * x)}
    st["con"] = np.where(fl, con[field], 0.0)
    st["nut"] = np.where(fl, nut * np.cos(x) ** 2, 0.0)
    flux = []
    for ctx in ctxs:
        ctx.upload_state(st)
        advance_to_lists([ctx])
        ctx.effpor()
        ctx.scalart()
        before = ctx.download_state()["con"]
        ctx.scalarupdate(1.0)
        flux.append((ctx.download_state()["con"] - before)[fl])
    g, c = flux
    if field == "one":
        assert not g.any() and not c.any()
    else:
        assert np.abs(c).max() > 0
        assert np.abs(g - c).max() <= 1e-11 * np.abs(c).max() + 2e-16 * np.abs(st["con"]).max()
