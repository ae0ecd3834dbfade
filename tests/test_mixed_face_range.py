"""The FP32-mixed Baer-Nunziato face fluxes are the FP64 values rounded once to
FP32, up to the largest finite flux and down to denormal ones."""
import dataclasses

import numpy as np
import pytest

import aderdg

pytestmark = pytest.mark.gpu
FACES = (aderdg.A_FU, aderdg.A_FP, aderdg.A_GU, aderdg.A_GP)


def fluxes(cfg, q, f):
    """The face fluxes of the face states q and fluxes f."""
    s = aderdg.Solver(cfg)
    s.set(aderdg.A_QBND, q.astype(float).ravel())
    s.set(aderdg.A_FBND, f.astype(float).ravel())
    s.set_time_step(0.0, 1e-3)
    s.riemann_problem()
    out = [s.get(a).reshape(-1, 9)[:, :8] for a in FACES]
    s.close()
    return out


@pytest.mark.parametrize("power", [0, 100, 127, 128, -100, -126, -130, -140])
def test_scaled_faces(gpu_lib, power):
    """States and fluxes scaled by powers of two in all but the volume fraction (whose
    own flux is a velocity), the largest flux within a factor 2 of that power: the
    FP64 mode's fluxes of the same FP32 states, to half an ulp of FP32 and the FP64
    forms' own roundings."""
    cfg = aderdg.Config(system=aderdg.SYS_BN, N=2, imax=4, jmax=3, bc=(3, 3, 3, 3), limiter=0, gamma_s=1.4, gamma_g=1.67,
                        precision=aderdg.FP32_MIXED)
    fp64 = dataclasses.replace(cfg, precision=aderdg.FP64)
    rng = np.random.default_rng(11)
    q = np.array([0.6, 1.2, -0.3, 2.5, 0.3, 0.6, 0.3, 1.9, 0.6]) * (1 + 0.2 * rng.uniform(-1, 1, (cfg.cells, cfg.P, 4, 9)))
    f = 5.0 * (1 + 0.1 * rng.uniform(-1, 1, q.shape)) * (np.arange(9) < 8)
    top = max(np.abs(x).max() for x in fluxes(fp64, q, f))
    scale = 2.0 ** (power - np.ceil(np.log2(top)))  # the largest flux in (0.5, 1] 2^power
    w = np.where(np.arange(9) == 8, 1.0, scale)
    q, f = (q * w).astype(np.float32), (f * w).astype(np.float32)
    assert np.isfinite(q).all() and np.isfinite(f).all()
    for a, b in zip(fluxes(cfg, q, f), fluxes(fp64, q, f)):
        ulp = np.spacing(np.abs(b).astype(np.float32)).astype(float)
        assert np.all(np.abs(a - b) <= 0.5 * ulp * (1 + 1e-6) + 1e-13 * np.abs(b))


@pytest.mark.parametrize("precision", [aderdg.FP32_MIXED, aderdg.FP64])
@pytest.mark.parametrize("rho", [2e-30, 1e-20, 1e-10, 1e10, 1e20, 1e28])
def test_fastest_wave_of_extreme_densities(gpu_lib, precision, rho):
    """The largest of the faces' four speeds is found where the squares of the solid's
    momenta underflow in FP32 (or its sound speed's does): the gas's fluxes, which it
    multiplies, are those of the reference order's speeds."""
    cfg = aderdg.Config(system=aderdg.SYS_BN, N=2, imax=5, jmax=4, bc=(3, 3, 3, 3), limiter=0, gamma_s=1.4, gamma_g=1.67,
                        precision=precision)
    rng = np.random.default_rng(3)
    shape = (cfg.cells, cfg.P, 4)
    r, u, v, c = rho * rng.uniform(1, 1.2, shape), *(rng.uniform(-900, 900, (2,) + shape)), rng.uniform(200, 1200, shape)
    p = r * c * c / 1.4
    solid = [r, r * u, r * v, p / 0.4 + 0.5 * r * (u * u + v * v)]
    gas = np.array([0.3, 0.1, 0.05, 0.7]) * (1 + 0.2 * rng.uniform(-1, 1, shape + (4,)))
    q = np.concatenate([np.stack(solid, -1), gas, np.full(shape + (1,), 0.6)], -1).astype(np.float32)
    f = np.zeros_like(q)
    if precision == aderdg.FP64:
        # the fused step's faces, on the states its predictor leaves (uniform cells)
        s = aderdg.Solver(cfg)
        uh = np.repeat(q[:, :1, :1].reshape(cfg.cells, 1, 9), cfg.P ** 2, 1).astype(float)
        s.upload(uh.ravel())
        dt = s.calc_time_step(0.0, 1e30)
        t, _, _ = s.step(0.0, 1e-6 * dt)
        a = [s.get(w).reshape(-1, 9)[:, 4:8] for w in FACES]
        s.set_time_step(t, dt)
        s.riemann_problem()
        b = [s.get(w).reshape(-1, 9)[:, 4:8] for w in FACES]
    else:
        a = [x[:, 4:] for x in fluxes(cfg, q, f)]
        b = [x[:, 4:] for x in fluxes(dataclasses.replace(cfg, precision=aderdg.FP64), q, f)]
    for x, y in zip(a, b):
        assert np.all(np.abs(x - y) <= 2.0 ** -23 * np.abs(y) + 1e-12 * np.abs(y).max())
