"""FP64 advection-diffusion predictor: one operator per direction for the
gradient, the flux and its divergence, against the oracle's predictor, which
forms them one after another."""
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
