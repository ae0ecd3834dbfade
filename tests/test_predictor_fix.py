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


def uniform(name, N, grid, velocity):
    cfg, ic, params, _ = aderdg.workloads.make(name, side=8, N=N)
    cfg = dataclasses.replace(cfg, imax=grid[0], jmax=grid[1])
    if cfg.nvar == 4:
        q = [0.7, 0.7 * velocity[0], 0.7 * velocity[1], 2.3]
    else:
        q = [0.6, 0.6 * velocity[0], 0.6 * velocity[1], 1.9, 0.23, 0.23 * velocity[1], 0.23 * velocity[0], 0.87, 0.61]
    return cfg, np.tile(q, (cfg.cells, cfg.P ** 2, 1))


@pytest.mark.parametrize("name", ["euler_vortex", "bn_cylinder"])
@pytest.mark.parametrize("N", [3, 4, 5])
@pytest.mark.parametrize("velocity", [(0.0, 0.0), (0.3, -0.7)])
def test_constant_states_are_exact(gpu_lib, name, N, velocity):
    """The derivative of a constant is 0: a uniform state is its own time average, and
    at rest its mass fluxes are 0, to the last bit."""
    cfg, u = uniform(name, N, (5, 3), velocity)
    got = predict(cfg, u.ravel(), 0.01)
    assert np.array_equal(got["qhi"].reshape(u.shape), u)
    f = got["fhi"].reshape(cfg.cells, cfg.P ** 2, 2, cfg.nvar)
    assert np.all(f == f[:1, :1])
    if velocity == (0.0, 0.0):
        assert not f[..., 0].any() and not f[..., 3].any()


@pytest.mark.parametrize("name", ["euler_vortex", "bn_cylinder"])
@pytest.mark.parametrize("N", [3, 4, 5])
def test_zero_lines_stay_zero(gpu_lib, name, N):
    """A state that varies along x only has no momentum along y, to the last bit."""
    cfg, u = uniform(name, N, (6, 4), (0.2, 0.0))
    V, P = cfg.nvar, cfg.P
    factor = 1.0 + 0.05 * np.random.default_rng(9).uniform(-1, 1, (cfg.imax, P))
    w = u.reshape(cfg.jmax, cfg.imax, P, P, V).copy()  # [j][i][y][x]
    w[..., [0, 1, 3] + ([4, 6, 7] if V == 9 else [])] *= factor[None, :, None, :, None]
    if V == 9:
        w[..., 5:7] = w[..., 6:4:-1]
    got = predict(cfg, w.ravel(), 0.01)["qhi"].reshape(-1, V)
    assert not got[:, 2].any()
    if V == 9:
        assert not got[:, 6].any()


# values of the states are 0.01 to 20: powers that leave every line within the
# fixed-point range (2^-823 .. 2^900), that split the lines and that leave it
@pytest.mark.parametrize("name,N", [("euler_vortex", 3), ("euler_rp2d", 4), ("euler_rp2d", 5)])
@pytest.mark.parametrize("power", [-850, -824, -820, -815, -664, -60, 60, 664, 890, 895, 899])
def test_scaled_states_within_the_range_and_at_its_edges(gpu_lib, name, N, power):
    test_scaled_states(gpu_lib, name, N, power)


@pytest.mark.parametrize("N", [3, 5])
@pytest.mark.parametrize("tiny", [1e-200, 1e-260, 1e-300])
def test_lines_of_both_kinds(gpu_lib, N, tiny):
    """A momentum below the fixed-point range beside lines within it."""
    cfg, uh = state("euler_vortex", N, (7, 5))
    u = uh.reshape(-1, 4).copy()
    u[:, 2] *= tiny
    o = po.Oracle(oracle_config(cfg))
    o.set(po.UH, u.ravel())
    dt = o.calc_time_step(0.0, 1e30)
    o.predictor()
    got = predict(cfg, u.ravel(), dt)
    for k, _, w in OUT:
        assert near(got[k], o.get(w), 4), k
