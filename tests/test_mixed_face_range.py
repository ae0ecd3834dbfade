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
