"""FP64 phase calls after fused steps and after one another, in the orders a
caller may take them: with the time step given (set_time_step) and without
limiter_prepare, the counts and arrays are those of the full sequence."""
import dataclasses

import numpy as np
import pytest

import aderdg

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _gpu(gpu_lib):
    return gpu_lib


def build(name, N, grid):
    cfg, ic, params, _ = aderdg.workloads.make(name, side=8, N=N)
    cfg = dataclasses.replace(cfg, imax=grid[0], jmax=grid[1])
    return cfg, aderdg.project_initial_condition(cfg, ic, params)


def phase_step(s, t, dt=None, prepare=True):
    """One step by phases; dt given: set_time_step in place of calc_time_step."""
    if dt is None:
        dt = s.calc_time_step(t, 1e30)
    else:
        s.set_time_step(t, dt)
    if prepare:
        s.limiter_prepare()
    s.space_time_predictor()
    s.volume_integral()
    s.riemann_problem()
    s.surface_integral()
    n = s.element_update()
    settled = s.info()["n_settled"]
    bounds = s.get(aderdg.A_LMIN), s.get(aderdg.A_LMAX)
    s.limiter()
    return t + dt, dt, n, settled, bounds


@pytest.mark.parametrize("name,N,grid", [("euler_rp2d", 3, (40, 33)), ("bn_cylinder", 2, (24, 31))])
def test_given_time_step_after_settled_cells(name, N, grid):
    """The cells a fused step settled are no part of the phase steps after it."""
    cfg, (uh, lh) = build(name, N, grid)
    a, b = aderdg.Solver(cfg), aderdg.Solver(cfg)
    a.upload(uh)
    a.init_limiter(lh)
    t = 0.0
    for _ in range(200):
        t, dt, _ = a.step(t, 1e30)
        if a.info()["n_settled"]:
            break
    assert a.info()["n_settled"] > 0
    b.upload(a.download()[0])
    b.upload_limiter(*a.download_limiter())
    for k in range(3):
        ra, rb = (phase_step(s, t, 0.5 * dt, prepare=False) for s in (a, b))
        assert ra[2:4] == rb[2:4] and ra[3] == 0, k
        for w in (aderdg.A_RECOMPUTE, aderdg.A_STATUS, aderdg.A_UH):
            assert np.array_equal(a.get(w), b.get(w)), (k, w)
        t = ra[0]


@pytest.mark.parametrize("name,N,grid", [("euler_rp2d", 3, (13, 10)), ("bn_cylinder", 2, (13, 14))])
def test_phase_steps_without_prepare(name, N, grid):
    """Consecutive phase steps form the same minima and maxima with and without
    limiter_prepare, recompute = 2 cells that stay unlimited among them."""
    cfg, (uh, lh) = build(name, N, grid)
    a, b = aderdg.Solver(cfg), aderdg.Solver(cfg)
    for s in (a, b):
        s.upload(uh)
        s.init_limiter(lh)
    t, kept = 0.0, 0
    for k in range(4):
        ra, rb = phase_step(a, t), phase_step(b, t, prepare=False)
        assert ra[:4] == rb[:4], k
        for x, y in zip(ra[4], rb[4]):
            assert np.array_equal(x, y), k
        for w in (aderdg.A_RECOMPUTE, aderdg.A_STATUS, aderdg.A_UH):
            assert np.array_equal(a.get(w), b.get(w)), (k, w)
        kept += int(((a.get(aderdg.A_RECOMPUTE) == 2) & (a.get(aderdg.A_STATUS) == 0)).sum())
        t = ra[0]
    assert kept > 0
