"""The FP64 fused step's face fluxes and subcell re-solve (reciprocal-sharing
forms) against the phase API's (the reference's operation order)."""
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


def build(name, N, grid):
    cfg, ic, params, _ = aderdg.workloads.make(name, side=8, N=N)
    cfg = dataclasses.replace(cfg, imax=grid[0], jmax=grid[1])
    return cfg, aderdg.project_initial_condition(cfg, ic, params)


CASES = [("euler_vortex", 1, (5, 7)), ("euler_rp2d", 2, (16, 9)), ("euler_rp2d", 5, (8, 8)), ("bn_cylinder", 1, (9, 12)),
         ("bn_cylinder", 3, (12, 10)), ("bn_cylinder", 4, (8, 8))]


@pytest.mark.parametrize("name,N,grid", CASES)
def test_faces(name, N, grid):
    cfg, (uh, lh) = build(name, N, grid)
    s = aderdg.Solver(cfg)
    s.upload(uh)
    s.init_limiter(lh)
    t, _, _ = s.step(0.0, 1e30)
    which = [aderdg.A_FU, aderdg.A_GU] + ([aderdg.A_FP, aderdg.A_GP] if cfg.system == aderdg.SYS_BN else [])
    fused = [s.get(w) for w in which]
    s.calc_time_step(t, 1e30)
    s.riemann_problem()  # the reference's order, on the same face states
    q, f = np.abs(s.get(aderdg.A_QBND)).max(), np.abs(s.get(aderdg.A_FBND)).max()
    # at most 64 roundings of terms no larger than a flux or a speed (below 4
    # in these fields) times a state
    tol = 64 * 2.0 ** -53 * (f + 4.0 * q)
    for a, w in zip(fused, which):
        assert np.abs(a - s.get(w)).max() <= tol, w


@pytest.mark.parametrize("name,N,grid", [c for c in CASES if c[0] != "euler_vortex"])
def test_inadmissible_states(name, N, grid):
    """A cell with a negative pressure: its sound speeds are NaN and leave the
    velocities, in both orders; the re-solved state agrees, NaN for NaN."""
    cfg, (uh, lh) = build(name, N, grid)
    u = uh.reshape(cfg.cells, (N + 1) ** 2, cfg.nvar).copy()
    lh = lh.reshape(cfg.cells, -1, cfg.nvar).copy()
    u[cfg.cells // 2, :, 3] *= -0.5
    lh[cfg.cells // 2, :, 3] *= -0.5
    out = []
    for fused in (True, False):
        s = aderdg.Solver(cfg)
        s.upload(u.ravel())
        s.init_limiter(lh.ravel())
        t, dt, n = s.step(0.0, 1e30) if fused else by_phases(s, 0.0, 1e30)
        out.append((t, n, s.get(aderdg.A_UH), s.get(aderdg.A_STATUS)))
    (ta, na, a, sa), (tb, nb, b, sb) = out
    assert ta == tb and na == nb and na > 0 and np.array_equal(sa, sb)
    assert np.array_equal(np.isnan(a), np.isnan(b))
    ok = np.isfinite(b)
    # as the admissible states' comparison of both orders (sums of a step's few
    # hundred roundings)
    assert np.abs(a[ok] - b[ok]).max() <= 1e-12 * np.abs(b[ok]).max()


@pytest.mark.parametrize("name,N,grid", [("euler_rp2d", 3, (17, 12)), ("bn_cylinder", 2, (13, 14)), ("euler_rp2d", 5, (8, 8))])
def test_host_step(name, N, grid):
    """A host step and upload, upload_limiter and a step: the same time step, decisions
    and state, bit for bit.  (Both prime with certified bounds; against exact ones:
    test_fp64_restart.py.)"""
    cfg, (uh, lh) = build(name, N, grid)
    h, d = aderdg.Solver(cfg), aderdg.Solver(cfg)
    for s in (h, d):
        s.upload(uh)
        s.init_limiter(lh)
    u, t = uh.copy(), 0.0
    for _ in range(3):
        st, l = h.download_limiter()
        d.upload(u)
        d.upload_limiter(st, l)
        td, dtd, nd = d.step(t, 1e30)
        t, dt, n = h.step_host(u, t, 1e30)
        assert (t, dt, n) == (td, dtd, nd)
        assert np.array_equal(u, d.download()[0]) and np.array_equal(h.get(aderdg.A_STATUS), d.get(aderdg.A_STATUS))
        assert np.array_equal(h.get(aderdg.A_LMIN), d.get(aderdg.A_LMIN))


@pytest.mark.parametrize("fused_first", [False, True])
def test_phases_without_limiter_prepare(gpu_lib, fused_first):
    """The phase API forms exact minima and maxima itself where the caller leaves out
    limiter_prepare after an upload or a fused step."""
    cfg, (uh, lh) = build("euler_rp2d", 3, (13, 10))
    a, b = aderdg.Solver(cfg), aderdg.Solver(cfg)
    for s in (a, b):
        s.upload(uh)
        s.init_limiter(lh)
        t = s.step(0.0, 1e30)[0] if fused_first else 0.0
        s.calc_time_step(t, 1e30)
        if s is a:
            s.limiter_prepare()
        s.space_time_predictor()
        s.volume_integral()
        s.riemann_problem()
        s.surface_integral()
        s.element_update()
        s.limiter()
    for w in (aderdg.A_UH, aderdg.A_LMIN, aderdg.A_LMAX, aderdg.A_STATUS, aderdg.A_RECOMPUTE):
        assert np.array_equal(a.get(w), b.get(w)), w
