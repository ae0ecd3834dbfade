"""The FP64 predictor's fixed-point linear algebra (N >= 3, Euler and
Baer-Nunziato; csrc/predictor_fix.cuh) against the oracle, on grids whose cell
count is no multiple of a CTA's cells, and at the edges of its range: states
scaled until every line takes the FP64 path, and lines holding NaN or infinity.

Tolerance: the oracle's FP64 sums have at most 6 terms and N+1 Picard
iterations, each rounding to 2^-53 of terms at most ~20 times the largest value
of a variable (the derivative matrices' row sums): 6 * 6 * 20 * 2^-53 = 8e-14,
taken as 1e-12 of the variable's largest magnitude.
"""
import dataclasses

import numpy as np
import pytest

import aderdg
import pyoracle as po

from helpers import oracle_config

pytestmark = pytest.mark.gpu
TOL = 1e-12
CASES = [(name, N, grid) for name in ("euler_vortex", "euler_rp2d", "bn_cylinder") for N in (3, 4, 5)
         for grid in ((7, 5), (1, 1))]
OUT = (("qhi", aderdg.A_QHI, po.QHI), ("fhi", aderdg.A_FHI, po.FHI), ("qbnd", aderdg.A_QBND, po.QBND),
       ("fbnd", aderdg.A_FBND, po.FBND))


def state(name, N, grid):
    cfg, ic, params, _ = aderdg.workloads.make(name, side=8, N=N)
    cfg = dataclasses.replace(cfg, imax=grid[0], jmax=grid[1])
    uh, _ = aderdg.project_initial_condition(cfg, ic, params)
    # no value repeated over a cell: 1% of noise, seeded
    return cfg, uh * (1.0 + 0.01 * np.random.default_rng(7).uniform(-1, 1, uh.size))


def predict(cfg, uh, dt):
    g = aderdg.Solver(cfg)
    g.upload(uh)
    g.set_time_step(0.0, dt)
    g.space_time_predictor()
    out = {k: g.get(w) for k, w, _ in OUT}
    g.close()
    return out


def near(a, b, V):
    a, b = a.reshape(-1, V), b.reshape(-1, V)
    return np.all(np.abs(a - b).max(0) <= TOL * np.abs(b).max(0) + 1e-300)


@pytest.mark.parametrize("name,N,grid", CASES)
def test_predictor_equals_oracle(gpu_lib, name, N, grid):
    cfg, uh = state(name, N, grid)
    o = po.Oracle(oracle_config(cfg))
    o.set(po.UH, uh)
    dt = o.calc_time_step(0.0, 1e30)
    o.predictor()
    got = predict(cfg, uh, dt)
    for k, _, w in OUT:
        assert near(got[k], o.get(w), cfg.nvar), k


@pytest.mark.parametrize("name,N", [("euler_vortex", 3), ("euler_rp2d", 5)])
@pytest.mark.parametrize("power", [-900, 905])
def test_scaled_states(gpu_lib, name, N, power):
    """The Euler fluxes scale with the state: beyond the fixed-point range the
    FP64 path gives the scaled result."""
    cfg, uh = state(name, N, (7, 5))
    o = po.Oracle(oracle_config(cfg))
    o.set(po.UH, uh)
    dt = o.calc_time_step(0.0, 1e30)
    one, scaled = predict(cfg, uh, dt), predict(cfg, np.ldexp(uh, power), dt)
    for k in one:
        assert near(np.ldexp(scaled[k], -power), one[k], cfg.nvar), k


@pytest.mark.parametrize("name,N", [("euler_vortex", 4), ("bn_cylinder", 3)])
@pytest.mark.parametrize("bad", [np.nan, np.inf])
def test_nonfinite_lines_stay_in_their_cell(gpu_lib, name, N, bad):
    cfg, uh = state(name, N, (7, 5))
    o = po.Oracle(oracle_config(cfg))
    o.set(po.UH, uh)
    dt = o.calc_time_step(0.0, 1e30)
    hit = uh.copy()
    per = cfg.nvar * cfg.P * cfg.P
    hit[17 * per + 3] = bad
    one, two = predict(cfg, uh, dt), predict(cfg, hit, dt)
    for k in one:
        a, b = one[k].reshape(cfg.cells, -1), two[k].reshape(cfg.cells, -1)
        assert not np.all(np.isfinite(b[17])), k
        keep = np.arange(cfg.cells) != 17
        assert np.array_equal(a[keep], b[keep]), k
