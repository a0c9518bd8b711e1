"""Porosity sums where a particle's support holds more solids than the kernels'
column of 32 takes at a time (csrc/pairs.cu k_effpor, csrc/wcsph.cu k_wc_por).

Every solid of the tank is replaced by four or nine that share its mass, a
quarter of the spacing apart, so that a support in the slope holds some
hundred of them.  effpor is compared with the oracle (both sum some hundred
positive terms of FP64 rounding: 1e-13 allows for the order; the mixed path's
terms are FP32: 1e-6), four lanes with one (the same bits), and the WCSPH run
and its gradient with the oracle's at the bounds of their own comparison.
"""
import numpy as np
import pytest

import oracle
from beach_slope_confined_gb300 import Solver, scenario as sc, setup_tank
from pairrun import make_pair

pytestmark = pytest.mark.gpu


def tank(split, **kw):
    spec = sc.TankSpec(dx=0.02, por_cells=(16, 4), **kw)
    scen = sc.build(spec)
    off = (np.arange(split) - 0.5 * (split - 1)) * 0.25 * spec.dx
    ox, oy = (a.ravel() for a in np.meshgrid(off, off))
    scen.sx = (scen.sx[:, None] + ox).ravel()
    scen.sy = (scen.sy[:, None] + oy).ravel()
    scen.smass = np.repeat(scen.smass / split**2, split**2)
    scen.srho = np.repeat(scen.srho, split**2)
    return spec, scen


@pytest.mark.parametrize("prec,tol", [("fp64", 1e-13), ("mixed", 1e-6)])
@pytest.mark.parametrize("split", [2, 3])
def test_effpor(split, prec, tol, monkeypatch):
    spec, scen = tank(split)
    P = sc.make_params(spec, scen.bounds, precision=prec)
    out = []
    for lanes in ("4", "1"):
        monkeypatch.setenv("BSC_PAIR_LANES", lanes)
        g, c = make_pair(scen, P, Solver)
        g.effpor()
        c.effpor()
        out.append((g.download_state(), c.download_state()))
        g.close()
        c.close()
    (a, want), (b, _) = out
    fl = scen.tid == sc.TID_FLUID
    assert 0.1 < want["porosity"][fl].min() < 0.9
    assert np.abs(a["porosity"] - want["porosity"]).max() <= tol
    for f in ("porosity", "rho", "resist"):
        assert np.array_equal(a[f], b[f]), f


@pytest.mark.parametrize("split", [2, 3])
def test_wcsph(split):
    spec, scen = tank(split, dt=2e-4)
    P = sc.make_params(spec, scen.bounds, precision="fp64")
    out = []
    for ctx in (Solver(P), oracle.context(P)):
        setup_tank(ctx, scen)
        ctx.wcsph_setup(sc.wcsph_params(spec, scen)[0])
        eta = ctx.wcsph_forward(20, 8)
        w = np.random.default_rng(3).standard_normal(eta.shape)
        out.append((eta, ctx.wcsph_adjoint(w)))
        ctx.close()
    (eg, gg), (ec, gc) = out
    assert np.max(np.abs(eg - ec)) <= 1e-9 * np.max(np.abs(ec))
    assert np.max(np.abs(gg[:2] - gc[:2]) / np.abs(gc[:2])) <= 1e-8
    assert np.max(np.abs(gg[2:] - gc[2:])) <= 1e-8 * np.max(np.abs(gc[2:]))
