"""Advection-diffusion: the FP64 predictor's one operator per direction for the
gradient, the flux and its divergence against the oracle's predictor, which
forms them one after another; the cell kernel's own face fluxes (small grids)
against the face kernel's."""
import dataclasses

import numpy as np
import pytest

import aderdg
import pyoracle as po

from helpers import oracle_config

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N", [1, 2, 3, 4, 5])
@pytest.mark.parametrize("mode", [0, 1])
def test_predictor(gpu_lib, N, mode):
    cfg, ic, params, _ = aderdg.workloads.make("ad_sine", side=8, N=N)
    cfg = dataclasses.replace(cfg, imax=7, jmax=5, ad_flux_mode=mode, a=0.05, cx=1.3, cy=-0.7)
    uh, _ = aderdg.project_initial_condition(cfg, ic, params)
    uh = uh * (1 + 0.2 * np.random.default_rng(N).uniform(-1, 1, uh.size))
    o, g = po.Oracle(oracle_config(cfg)), aderdg.Solver(cfg)
    o.set(po.UH, uh)
    g.upload(uh)
    assert g.calc_time_step(0.0, 1.0) == o.calc_time_step(0.0, 1.0)
    o.predictor()
    g.space_time_predictor()
    for mine, ref in ((aderdg.A_QHI, po.QHI), (aderdg.A_FHI, po.FHI), (aderdg.A_QBND, po.QBND),
                      (aderdg.A_GRADQBND, po.GRADQBND)):
        a, b = g.get(mine), o.get(ref)
        # both sides round a few hundred terms, gradients at most (N + 1)^2 times the state over dx
        assert np.abs(a - b).max() <= 1e-12 * np.abs(b).max(), mine


@pytest.mark.parametrize("precision", [aderdg.FP64, aderdg.FP32_MIXED])
@pytest.mark.parametrize("N", [1, 2, 5])
@pytest.mark.parametrize("bc", [(3, 3, 3, 3), (1, 1, 1, 1), (2, 2, 2, 2), (1, 2, 3, 3)])
def test_faces_of_small_grids(gpu_lib, precision, N, bc):
    """A grid small enough for the cell kernel to form its face fluxes, alone and as
    one of two in a batch too large for that: state and face fluxes are the same
    bit for bit (one expression, evaluated in either kernel)."""
    cfg, ic, params, _ = aderdg.workloads.make("ad_sine", side=8, N=N, precision=precision)
    cfg = dataclasses.replace(cfg, imax=7, jmax=5, bc=bc, a=0.05, cx=1.3, cy=-0.7)
    big = dataclasses.replace(cfg, imax=500, jmax=300)
    s = aderdg.Solver(cfg)
    s.initial_condition(ic, params)
    t, _ = s.run(0.0, 1e30, 3)
    units = aderdg.Batch.units(cfg) + aderdg.Batch.units(big) + 64
    b = aderdg.Batch(cfg.system, N, precision, cfg.limiter, capacity_units=units, max_instances=2)
    small = b.admit_ic(cfg, ic, params, 1e30, 3)
    b.admit_ic(big, ic, params, 1e30, 3)
    b.launch(3)
    b.sync()
    assert b.query(small)["time"] == t
    assert np.array_equal(b.download(small), s.download()[0])
    if precision == aderdg.FP64:
        # the phase API's faces, on the face states of the last fused step
        f = [s.get(aderdg.A_FU), s.get(aderdg.A_GU)]
        s.calc_time_step(t, 1e30)
        s.riemann_problem()
        assert np.array_equal(f[0], s.get(aderdg.A_FU)) and np.array_equal(f[1], s.get(aderdg.A_GU))
