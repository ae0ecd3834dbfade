"""The FP64 mode's fused step decides the DMP from certified FP32 projections;
its time step, flags and neighbourhood min/max are those of the phase API, which
projects every cell in FP64, bit for bit, and its state to 1e-12: on states with
shocks, uniform regions and smooth flow, on magnitudes beyond the FP32 bound's
reach (x 1e4), and on states placed within 1e-9 of the DMP thresholds."""
import dataclasses

import numpy as np
import pytest

import aderdg

pytestmark = pytest.mark.gpu

CASES = [("euler_rp2d", 1, (13, 9)), ("euler_rp2d", 3, (17, 12)), ("euler_rp2d", 5, (9, 7)), ("euler_vortex", 4, (9, 11)),
         ("bn_cylinder", 2, (13, 14)), ("bn_cylinder", 3, (12, 9)), ("bn_cylinder", 5, (7, 6))]


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


def same(f, p, uh, lh, steps):
    for s in (f, p):
        s.upload(uh)
        s.init_limiter(lh)
    tf = tp = 0.0
    for k in range(steps):
        # the phase API's volume integral sums in another order than the fused
        # predictor: feed both the same state every step
        tf, dtf, nf = f.step(tf, 1e30)
        tp, dtp, np_ = by_phases(p, tp, 1e30)
        assert dtf == dtp and nf == np_, k
        assert np.array_equal(f.get(aderdg.A_RECOMPUTE), p.get(aderdg.A_RECOMPUTE)), k
        assert np.array_equal(f.get(aderdg.A_STATUS), p.get(aderdg.A_STATUS)), k
        for which in (aderdg.A_LMIN, aderdg.A_LMAX):
            assert np.array_equal(f.get(which), p.get(which)), (k, which)
        a, b = f.get(aderdg.A_UH), p.get(aderdg.A_UH)
        assert np.abs(a - b).max() <= 1e-12 * np.abs(b).max(), k
        st, l = p.download_limiter()
        for s in (f, p):
            s.set(aderdg.A_UH, b)
            s.upload_limiter(st, l)
        tf = tp


@pytest.mark.parametrize("name,N,grid", CASES)
@pytest.mark.parametrize("scale", [1.0, 1.0e4])
def test_fused_step_equals_phases(gpu_lib, name, N, grid, scale):
    cfg, ic, params, _ = aderdg.workloads.make(name, side=8, N=N)
    cfg = dataclasses.replace(cfg, imax=grid[0], jmax=grid[1])
    uh, lh = aderdg.project_initial_condition(cfg, ic, params)
    if scale != 1.0:
        # every conserved variable but the volume fraction
        for a in (uh, lh):
            a.reshape(-1, cfg.nvar)[:, : 8 if cfg.system == aderdg.SYS_BN else 4] *= scale
    f, p = aderdg.Solver(cfg), aderdg.Solver(cfg)
    same(f, p, uh, lh, 4)


@pytest.mark.parametrize("name,N", [("euler_vortex", 2), ("bn_cylinder", 2)])
def test_decisions_near_the_thresholds(gpu_lib, name, N):
    """A bump on one cell, grown in steps until the phase path's troubled count
    changes (the bump also widens the old bounds, so not every growth does),
    then bisected to 1e-9 of that threshold: both paths count alike throughout."""
    cfg, ic, params, _ = aderdg.workloads.make(name, side=9, N=N)
    if name == "bn_cylinder":
        params = (0.0, 0.0, 0.0) + tuple(params[3:])  # no inside: uniform
    uh, lh = aderdg.project_initial_condition(cfg, ic, params)
    f, p = aderdg.Solver(cfg), aderdg.Solver(cfg)
    per = cfg.nvar * cfg.P * cfg.P
    cell = (cfg.cells // 2) * per

    def marks(s, bump, fused):
        x = uh.copy()
        x[cell] += bump
        s.upload(x)
        return (s.step(0.0, 1e30) if fused else by_phases(s, 0.0, 1e30))[2]

    bumps = np.linspace(0.0, 0.5 * abs(uh[cell]), 41)
    counts = [marks(p, b, False) for b in bumps]
    assert [marks(f, b, True) for b in bumps] == counts
    change = np.flatnonzero(np.diff(counts))
    assert change.size
    lo, hi, base = bumps[change[0]], bumps[change[0] + 1], counts[change[0]]
    while hi - lo > 1e-9:
        mid = 0.5 * (lo + hi)
        n = marks(p, mid, False)
        assert marks(f, mid, True) == n, mid
        if n != base:
            hi = mid
        else:
            lo = mid
