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


BOUNDS = (aderdg.A_LMIN, aderdg.A_LMAX)


@pytest.mark.parametrize("name,N,grid", [("euler_rp2d", 3, (13, 10)), ("bn_cylinder", 2, (13, 14))])
@pytest.mark.parametrize("then", ["no_step", "no_run", "no_host_step", "upload", "upload_no_step", "initial_condition",
                                  "init_limiter", "upload_limiter", "limiter_prepare"])
def test_bounds_of_the_last_step_on_request(name, N, grid, then):
    """lmin and lmax stay those of the last step taken, whatever comes between it
    and the request short of another step."""
    cfg, ic, params, _ = aderdg.workloads.make(name, side=8, N=N)
    cfg = dataclasses.replace(cfg, imax=grid[0], jmax=grid[1])
    uh, lh = aderdg.project_initial_condition(cfg, ic, params)
    a, b = aderdg.Solver(cfg), aderdg.Solver(cfg)
    for s in (a, b):
        s.upload(uh)
        s.init_limiter(lh)
        t = s.run(0.0, 1e30, 5)[0]
    want = [a.get(w) for w in BOUNDS]
    st, l = a.download_limiter()
    assert st.any()
    other = 1.5 * uh
    if then == "no_step":
        b.step(t, t)
    elif then == "no_run":
        b.run(t, t, 3)
    elif then == "no_host_step":
        b.step_host(b.download()[0], t, t)
    elif then == "upload":
        b.upload(other)
    elif then == "upload_no_step":
        b.upload(other)
        b.step(t, t)
    elif then == "initial_condition":
        b.initial_condition(ic, params)
    elif then == "init_limiter":
        b.upload(other)
        b.init_limiter(2.0 * lh)
    elif then == "upload_limiter":
        b.upload_limiter(np.zeros_like(st), 2.0 * l)
    else:
        b.calc_time_step(t, 1e30)
        b.limiter_prepare()
    for w, x in zip(BOUNDS, want):
        assert np.array_equal(b.get(w), x), w
    assert all(np.array_equal(a.get(w), x) for w, x in zip(BOUNDS, want))  # a second request: the same


@pytest.mark.parametrize("name,N,grid", [("euler_rp2d", 3, (13, 10)), ("bn_cylinder", 2, (13, 14))])
def test_bounds_are_those_of_the_phases(name, N, grid):
    """After several fused steps on one trajectory, lmin and lmax of the last equal
    those the phase API forms from its start state."""
    cfg, (uh, lh) = build(name, N, grid)
    a, b = aderdg.Solver(cfg), aderdg.Solver(cfg)
    a.upload(uh)
    a.init_limiter(lh)
    t = a.run(0.0, 1e30, 4)[0]
    b.upload(a.download()[0])
    b.upload_limiter(*a.download_limiter())
    a.step(t, 1e30)
    r = phase_step(b, t)
    for w, x in zip(BOUNDS, r[4]):
        assert np.array_equal(a.get(w), x), w
