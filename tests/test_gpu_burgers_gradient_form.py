"""WENO5-Z in FP32 forward runs with an adjoint: their states are the candidates' weighted mean rounded operation by
operation, because a gradient jumps where a rounding decides the sign of beta0 - beta2. Restated here in
exactly rounded FP32 operations, and compared bit for bit at the edges of the stage's tiles."""
import numpy as np
import pytest

from multigpu_advectiondiffusion_gb300 import _native as N
from multigpu_advectiondiffusion_gb300.solvers import BurgersConfig, burgers_run_fixed

pytestmark = pytest.mark.gpu

f32, ext = np.float32, np.longdouble


def fma(a, b, c):
    return (np.multiply(a, b, dtype=ext) + c).astype(f32)


def _side(a, b, c, d, e):
    eps, k = f32(4e-6), f32(13 / 3)
    t = [fma(f32(-2), b, a) + c, fma(f32(-2), c, b) + d, fma(f32(-2), d, c) + e]
    s = [fma(f32(3), c, fma(f32(-4), b, a)), b - d, fma(f32(3), c, fma(f32(-4), d, e))]
    w0, w1, w2 = (fma(k * x, x, fma(y, y, eps)) for x, y in zip(t, s))
    q = [fma(f32(0.25 if i == 0 else -0.25), s[i], fma(f32(1 / 12), t[i], c)) for i in range(3)]
    tau, p12 = np.abs(w0 - w2), w1 * w2
    P = w0 * p12
    a0, a1, a2 = fma(tau, p12, P), f32(6) * fma(tau, w0 * w2, P), f32(3) * fma(tau, w0 * w1, P)
    return fma(a2, q[2], fma(a1, q[1], a0 * q[0])) / ((a0 + a1) + a2)


def _stage(cfg, stage, un, u, dt):
    hu, ha = f32(0.25) * u, f32(0.5) * np.abs(u)
    fp, fm = u * (hu + ha), u * (hu - ha)
    L = None
    for ax, h in ((1, cfg.dy), (2, cfg.dx), (0, cfg.dz)):
        at = lambda f, j: np.roll(f, -j, axis=ax)  # noqa: E731
        F = _side(*(at(fp, j) for j in (-2, -1, 0, 1, 2))) + _side(*(at(fm, j) for j in (3, 2, 1, 0, -1)))
        d = at(F, -1) - F
        L = d * f32(1 / h) if L is None else fma(d, f32(1 / h), L)
    v = f32(dt) * L
    if stage == 1:
        return un + v
    return f32(0.75) * un + f32(0.25) * (u + v) if stage == 2 else fma(f32(2), u + v, un) / f32(3)


@pytest.mark.parametrize("size", [(31, 15, 9), (33, 17, 8), (32, 16, 7), (36, 18, 11), (64, 33, 6), (6, 6, 6), (66, 7, 13)])
@pytest.mark.parametrize("div", [N.ADV_DIV_F32, N.ADV_DIV_F64])
def test_forward_states(cuda, size, div):
    import torch
    nx, ny, nz = size
    cfg = BurgersConfig(nx, ny, nz, 2.0 / nx, 2.0 / ny, 2.0 / nz, N.ADV_WENO5_Z, N.ADV_LF_LOCAL, N.ADV_BC_PERIODIC)
    cfg.div = div
    rng = np.random.default_rng(5)
    x, y, z = (np.arange(n) / n for n in size)
    u = 0.2 + 0.6 * np.sin(6.28 * x)[None, None, :] * np.cos(6.28 * y)[None, :, None] - 0.3 * np.sin(6.28 * z)[:, None, None]
    u = (u + 0.05 * rng.standard_normal(u.shape)).astype(f32)
    got = burgers_run_fixed(cfg, torch.from_numpy(u).to(cuda), 1e-3, 2).cpu().numpy()
    for _ in range(2):
        a = _stage(cfg, 1, u, u, 1e-3)
        b = _stage(cfg, 2, u, a, 1e-3)
        u = _stage(cfg, 3, u, b, 1e-3)
    np.testing.assert_array_equal(got, u)
