"""The FP64 fused step on states at the edge of the arithmetic (NaN, infinities,
products that underflow), against the phase API's operation order."""
import dataclasses

import numpy as np
import pytest

import aderdg

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _gpu(gpu_lib):
    return gpu_lib


def by_phases(s, time, tend):
    dt = s.calc_time_step(time, tend)
    s.limiter_prepare()
    s.space_time_predictor()
    s.volume_integral()
    s.riemann_problem()
    s.surface_integral()
    n = s.element_update()
    s.limiter()
    return time + dt, dt, n


def config(name, N, grid):
    cfg, ic, params, _ = aderdg.workloads.make(name, side=8, N=N)
    return dataclasses.replace(cfg, imax=grid[0], jmax=grid[1]), ic, params


def resolved(cfg, uh, cell, lh):
    """Lh and uh after a step (fused, then by phases) that re-solves `cell` from the
    subcell data lh: its polynomial's energy is negative."""
    V = cfg.nvar
    u = uh.reshape(cfg.cells, -1, V).copy()
    u[cell, :, 3] *= -0.5
    status = np.zeros(cfg.cells, dtype=np.int32)
    status[cell] = 1
    out = []
    for fused in (True, False):
        s = aderdg.Solver(cfg)
        s.upload(u.ravel())
        s.upload_limiter(status, lh.ravel())
        r = s.step(0.0, 1e30) if fused else by_phases(s, 0.0, 1e30)
        assert s.get(aderdg.A_STATUS)[cell] == 1
        out.append((r, s.get(aderdg.A_LH).reshape(cfg.cells, -1, V)[cell], s.get(aderdg.A_UH).reshape(cfg.cells, -1, V),
                    s.get(aderdg.A_RECOMPUTE), s.get(aderdg.A_STATUS)))
    return out


def uniform(system, N):
    cfg = aderdg.Config(system=system, N=N, imax=6, jmax=5, bc=(3, 3, 3, 3))
    q = [1.0, 0.5, 0.0, 2.5] if system == aderdg.SYS_EULER else [0.7, 0.35, 0.0, 2.0, 0.3, 0.1, 0.0, 0.9, 0.6]
    uh = np.tile(q, (cfg.cells, cfg.P ** 2, 1))
    return cfg, uh.ravel(), np.tile(q, (cfg.cells, cfg.S, cfg.S, 1))


SYSTEMS = [(aderdg.SYS_EULER, 2), (aderdg.SYS_EULER, 5), (aderdg.SYS_BN, 2), (aderdg.SYS_BN, 4)]


@pytest.mark.parametrize("system,N", SYSTEMS)
@pytest.mark.parametrize("size", [1e-170, 3e-163, 1e-155, 1e-300])
def test_slopes_whose_product_underflows(system, N, size):
    """A transverse momentum of growing tiny values: minmod is 0 where the slopes'
    product underflows.  Tolerance: the other variables are uniform, so that each
    value is a sum of a few tens of multiples of the momenta's largest."""
    cfg, uh, lh = uniform(system, N)
    cell = 14
    lh[cell, :, :, 2] = size * (1.0 + 0.3 * np.arange(cfg.S) ** 2)[None, :]
    (ra, a, _, *fa), (rb, b, _, *fb) = resolved(cfg, uh, cell, lh)
    assert ra == rb and all(np.array_equal(x, y) for x, y in zip(fa, fb))
    # away from the cell's sides, whose slopes meet the neighbours' zeros
    inner, want = (x.reshape(cfg.S, cfg.S, -1)[2:-2, 2:-2, 2] for x in (a, b))
    assert np.abs(want).max() > 0
    assert np.abs(inner - want).max() <= 1e-13 * np.abs(want).max() + 1e-322


def same_values(a, b):
    assert np.array_equal(np.isnan(a), np.isnan(b)) and np.array_equal(np.isinf(a), np.isinf(b))
    ok = np.isfinite(b)
    assert np.abs(a[ok] - b[ok]).max() <= 1e-12 * np.abs(b[ok]).max()


@pytest.mark.parametrize("system,N", SYSTEMS)
@pytest.mark.parametrize("at", [(0, 0), (2, 1)])
@pytest.mark.parametrize("v", [1, 3])
def test_nan_subcell(system, N, at, v):
    """One subcell holds a NaN among noisy ones: slopes beside it are those of the
    reference's minmod, and as many values become NaN."""
    cfg, uh, lh = uniform(system, N)
    cell = 14
    lh[cell] *= 1.0 + 0.01 * np.random.default_rng(3).uniform(-1, 1, lh[cell].shape)
    lh[cell, at[0], at[1], v] = np.nan
    (ra, a, ua, *fa), (rb, b, ub, *fb) = resolved(cfg, uh, cell, lh)
    assert ra == rb and all(np.array_equal(x, y) for x, y in zip(fa, fb))
    same_values(a, b)
    same_values(ua, ub)


@pytest.mark.parametrize("system,N", SYSTEMS)
@pytest.mark.parametrize("at", [(0, 0), (2, 1)])
@pytest.mark.parametrize("value", [np.inf, 1e308])
def test_infinite_density(system, N, at, value):
    """One subcell of infinite (or 1e308) density: its velocity is 0, as by division."""
    cfg, uh, lh = uniform(system, N)
    cell = 14
    lh[cell, at[0], at[1], 0] = value
    (ra, a, ua, *fa), (rb, b, ub, *fb) = resolved(cfg, uh, cell, lh)
    assert ra == rb and all(np.array_equal(x, y) for x, y in zip(fa, fb))
    assert np.array_equal(np.isfinite(a), np.isfinite(b)) and np.array_equal(np.isnan(a), np.isnan(b))
    assert np.array_equal(np.isfinite(ua), np.isfinite(ub))


@pytest.mark.parametrize("system,N", SYSTEMS)
@pytest.mark.parametrize("value,v", [(np.nan, 3), (np.nan, -1), (np.inf, 0), (1e150, 0), (1e-150, 0), (0.0, -1)])
def test_faces(system, N, value, v):
    """Face fluxes beside a cell of NaN, infinite, huge, tiny or zero values, against
    the reference's order on the same face states (fluxes of ordinary size: 64
    roundings of terms below 4, see test_fp64_fused_physics)."""
    cfg, uh, _ = uniform(system, N)
    u = uh.reshape(cfg.cells, -1, cfg.nvar).copy()
    u *= 1.0 + 0.01 * np.random.default_rng(5).uniform(-1, 1, u.shape)
    u[14, :, v] = value
    s = aderdg.Solver(dataclasses.replace(cfg, limiter=0))
    s.upload(uh)
    dt = s.calc_time_step(0.0, 1e30)
    s.set(aderdg.A_UH, u.ravel())
    t, _, _ = s.step(0.0, 0.1 * dt)
    which = [aderdg.A_FU, aderdg.A_GU] + ([aderdg.A_FP, aderdg.A_GP] if system == aderdg.SYS_BN else [])
    fused = [s.get(w) for w in which]
    s.set_time_step(t, dt)
    s.riemann_problem()
    for a, w in zip(fused, which):
        b = s.get(w)
        assert np.array_equal(np.isnan(a), np.isnan(b)) and np.array_equal(np.isinf(a), np.isinf(b)), w
        size = np.abs(b)
        ok = np.isfinite(b)
        assert np.all(np.abs(a - b)[ok] <= 64 * 2.0 ** -53 * 16.0 + 1e-10 * size[ok] * (size[ok] > 10.0)), w


@pytest.mark.parametrize("name,N,grid", [("euler_rp2d", 1, (15, 12)), ("euler_rp2d", 3, (12, 14)), ("euler_vortex", 4, (9, 10)),
                                         ("bn_cylinder", 2, (13, 12)), ("bn_cylinder", 3, (9, 11))])
@pytest.mark.parametrize("seed", range(6))
def test_nan_neighbour(name, N, grid, seed):
    """Cells of NaN energy (either sign) among noisy ones, all of magnitudes whose DMP
    is decided in FP64: the neighbourhoods' minima and maxima leave the NaN out."""
    cfg, ic, params = config(name, N, grid)
    uh, _ = aderdg.project_initial_condition(cfg, ic, params)
    rng = np.random.default_rng(seed)
    V = cfg.nvar
    u = uh.reshape(cfg.cells, -1, V) * (1.0 + 0.02 * 0.1 ** seed * rng.uniform(-1, 1, (cfg.cells, cfg.P ** 2, 1)))
    u[..., : 8 if V == 9 else 4] *= 1.0e6
    u[rng.choice(cfg.cells, 8, replace=False), :, 3] = -np.nan if seed % 2 else np.nan
    out = []
    for fused in (True, False):
        s = aderdg.Solver(cfg)
        s.upload(u.ravel())
        r = s.step(0.0, 1e30) if fused else by_phases(s, 0.0, 1e30)
        out.append((r, s.get(aderdg.A_RECOMPUTE), s.get(aderdg.A_STATUS), s.get(aderdg.A_LMIN), s.get(aderdg.A_LMAX)))
    (ra, *a), (rb, *b) = out
    assert ra == rb
    for x, y in zip(a, b):
        assert np.array_equal(x, y, equal_nan=True)
