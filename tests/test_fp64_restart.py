"""The FP64 mode's time steps do not depend on how a state was reached: a run
continued from its downloaded state, steps on a host array and the phase API's
calc_time_step give the time step of the uninterrupted run, bit for bit (the
fused step finds the cells that may hold the largest CFL denominator from FP32
bounds and evaluates those in the reference's order)."""
import dataclasses

import numpy as np
import pytest

import aderdg

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _gpu(gpu_lib):
    return gpu_lib


CASES = [("euler_vortex", 1, (9, 7)), ("euler_vortex", 4, (16, 13)), ("euler_rp2d", 2, (40, 33)), ("euler_rp2d", 3, (33, 21)),
         ("euler_rp2d", 5, (11, 9)), ("bn_cylinder", 1, (17, 12)), ("bn_cylinder", 2, (24, 31)), ("bn_cylinder", 3, (20, 17)),
         ("bn_cylinder", 5, (9, 8))]


def build(name, N, grid, limiter=1):
    cfg, ic, params, _ = aderdg.workloads.make(name, side=8, N=N)
    cfg = dataclasses.replace(cfg, imax=grid[0], jmax=grid[1], limiter=limiter)
    return cfg, aderdg.project_initial_condition(cfg, ic, params)


def start(cfg, uh, lh):
    s = aderdg.Solver(cfg)
    s.upload(uh)
    if cfg.limiter:
        s.init_limiter(lh)
    return s


def same_state(a, b):
    (ua, sa), (ub, sb) = a.download(), b.download()
    return np.array_equal(ua, ub) and np.array_equal(sa, sb)


@pytest.mark.parametrize("name,N,grid", CASES)
def test_continued_run(name, N, grid):
    cfg, (uh, lh) = build(name, N, grid)
    a, b, c = start(cfg, uh, lh), start(cfg, uh, lh), aderdg.Solver(cfg)
    t = a.run(0.0, 1e30, 12)[0]
    tb = b.run(0.0, 1e30, 7)[0]
    c.upload(b.download()[0])
    c.upload_limiter(*b.download_limiter())
    assert c.run(tb, 1e30, 5)[0] == t
    assert same_state(a, c)


@pytest.mark.parametrize("name,N,grid", CASES)
def test_host_steps(name, N, grid):
    cfg, (uh, lh) = build(name, N, grid)
    a, b = start(cfg, uh, lh), start(cfg, uh, lh)
    t = a.run(0.0, 1e30, 6)[0]
    u, tb = uh.copy(), 0.0
    for _ in range(6):
        tb, _, _ = b.step_host(u, tb, 1e30)
    assert tb == t and np.array_equal(u, a.download()[0])


@pytest.mark.parametrize("limiter", [1, 0])
@pytest.mark.parametrize("name,N,grid", CASES)
def test_calc_time_step_is_the_next_step(name, N, grid, limiter):
    cfg, (uh, lh) = build(name, N, grid, limiter)
    a, b = start(cfg, uh, lh), start(cfg, uh, lh)
    t = 0.0
    for k in range(5):
        want = b.calc_time_step(t, 1e30)
        ta, dt, _ = a.step(t, 1e30)
        assert dt == want, k
        b.upload(a.download()[0])
        t = ta


def random_states(cfg, rng):
    """Independent nodes: densities and pressures over eight decades, Mach numbers up
    to 1e3, a tenth of the cells uniform, one cell inadmissible."""
    n, P2, V = cfg.cells, cfg.P * cfg.P, cfg.nvar
    u = np.empty((n, P2, V))

    def phase(gamma, pi):
        r, p = 10.0 ** rng.uniform(-4, 4, (n, P2)), 10.0 ** rng.uniform(-4, 4, (n, P2))
        c = np.sqrt(gamma * (p + pi) / r)
        m, phi = c * 10.0 ** rng.uniform(-3, 3, (n, P2)), rng.uniform(0, 2 * np.pi, (n, P2))
        vx, vy = m * np.cos(phi), m * np.sin(phi)
        return r, r * vx, r * vy, (p + gamma * pi) / (gamma - 1) + 0.5 * r * m * m

    if cfg.system == aderdg.SYS_EULER:
        u[..., :4] = np.stack(phase(cfg.gamma, 0.0), -1)
    else:
        a = np.where(rng.uniform(size=(n, P2)) < 0.1, 10.0 ** rng.uniform(-6, -1, (n, P2)), rng.uniform(0.05, 0.95, (n, P2)))
        u[..., 8] = a
        u[..., :4] = np.stack(phase(cfg.gamma_s, cfg.pi_s), -1) * a[..., None]
        u[..., 4:8] = np.stack(phase(cfg.gamma_g, cfg.pi_g), -1) * (1 - a[..., None])
    flat = rng.uniform(size=n) < 0.1
    u[flat] = u[flat][:, :1]
    u[n // 3, :, 3] *= -0.5
    return u.ravel()


@pytest.mark.parametrize("name,N", [("euler_vortex", 2), ("euler_rp2d", 3), ("bn_cylinder", 2), ("bn_cylinder", 3)])
@pytest.mark.parametrize("seed", range(6))
@pytest.mark.parametrize("scale", [1.0, 1e-12, 1e25])
def test_random_states(name, N, seed, scale):
    """The time step after one very short step from random states is the reference
    order's, with the largest denominator in re-solved and other cells alike."""
    cfg, _ = build(name, N, (9, 7))
    uh = random_states(cfg, np.random.default_rng(seed))
    if scale != 1.0 and cfg.system == aderdg.SYS_EULER:
        uh = uh * scale
    a, b = aderdg.Solver(cfg), aderdg.Solver(cfg)
    for s in (a, b):
        s.upload(uh)
    short = 1e-9 * a.calc_time_step(0.0, 1e30)
    assert short > 0.0
    for s in (a, b):
        t, _, n = s.step(0.0, short)
    assert n > 0 and np.array_equal(a.download()[0], b.download()[0], equal_nan=True)
    want = b.calc_time_step(t, 1e30)
    if np.isfinite(want) and want < 1e19:  # no NaN among the denominators
        assert a.step(t, 1e30)[1] == want


def largest_along_x(system, N):
    """Cells so large that FP32's 1/dx, 1/dy are denormal numbers, the first 2e-4 too
    small, the second 2e-4 too large; a cell whose flow along x gives the largest CFL
    denominator and one whose flow along y gives 5e-5 less (by those FP32 values 1e-4
    more), among cells at rest."""
    unit = 2.0 ** -149
    dx, dy = 1.0 / (2000.4 * unit), 1.0 / (2000.6 * unit)
    x, y = float(np.float32(1 / dx)), float(np.float32(1 / dy))
    assert x == 2000 * unit and y == 2001 * unit
    cfg = aderdg.Config(system=system, N=N, imax=8, jmax=6, bc=(3, 3, 3, 3), xr=(8 * dx, 6 * dy), cfl=1e-8)
    c, U = 1e15, 3e15
    V = (((U + c) / dx + c / dy) * (1 - 5e-5) - c / dx) * dy - c
    assert (U + c) * x + c * y < (c * x + (V + c) * y) * (1 - 1e-4)
    u = np.zeros((cfg.cells, cfg.P ** 2, cfg.nvar))
    mom = np.zeros((cfg.cells, 2))
    mom[11], mom[29] = (U, 0.0), (0.0, V)
    phases = [(0, cfg.gamma, 1.0)] if system == aderdg.SYS_EULER else [(0, cfg.gamma_s, 0.6), (4, cfg.gamma_g, 0.4)]
    for o, g, a in phases:
        u[..., o] = a
        u[..., o + 1:o + 3] = a * mom[:, None]
        u[..., o + 3] = a * (c * c / g / (g - 1) + 0.5 * (mom ** 2).sum(1))[:, None]
    if system == aderdg.SYS_BN:
        u[..., 8] = 0.6
    return cfg, u.ravel()


@pytest.mark.parametrize("system", [aderdg.SYS_EULER, aderdg.SYS_BN])
@pytest.mark.parametrize("N", [2, 4])
def test_huge_cells(system, N):
    """The time step where 1/dx has few bits in FP32."""
    cfg, uh = largest_along_x(system, N)
    a, b = aderdg.Solver(cfg), aderdg.Solver(cfg)
    for s in (a, b):
        s.upload(uh)
    short = 1e-9 * a.calc_time_step(0.0, 1e30)
    for s in (a, b):
        t, _, _ = s.step(0.0, short)
    assert np.array_equal(a.download()[0], b.download()[0])
    b.upload(b.download()[0])
    want = b.calc_time_step(t, 1e30)
    assert 0.0 < want < 1e19  # below the scheme's largest time step
    assert a.step(t, 1e30)[1] == want


@pytest.mark.parametrize("name,N,grid", [("euler_rp2d", 2, (17, 12)), ("euler_vortex", 4, (9, 8)), ("bn_cylinder", 2, (13, 14)),
                                         ("bn_cylinder", 3, (10, 9))])
@pytest.mark.parametrize("noise", [2e-5, 1e-4, 1e-3])
def test_priming_bounds(name, N, grid, noise):
    """A host step primes with certified FP32 bounds on the minima and maxima; the same
    step from exact ones (limiter_prepare: FP64 projections in the reference's order)
    takes the same decisions and gives the same state bit for bit, on states with
    noise about the DMP's tolerance, where the bounds leave comparisons open."""
    cfg, (uh, lh) = build(name, N, grid)
    uh = uh * (1.0 + noise * np.random.default_rng(1).uniform(-1, 1, uh.size))
    h, d = start(cfg, uh, lh), start(cfg, uh, lh)
    u, t, marked = uh.copy(), 0.0, 0
    for _ in range(4):
        st, l = h.download_limiter()
        d.upload(u)
        d.upload_limiter(st, l)
        d.limiter_prepare()
        want = d.step(t, 1e30)
        got = h.step_host(u, t, 1e30)
        assert got == want
        assert np.array_equal(u, d.download()[0])
        for w in (aderdg.A_STATUS, aderdg.A_RECOMPUTE, aderdg.A_LMIN, aderdg.A_LMAX):
            assert np.array_equal(h.get(w), d.get(w)), w
        t, marked = got[0], marked + got[2]
    assert marked > 0 or noise < 1e-4
