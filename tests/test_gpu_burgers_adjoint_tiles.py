"""The Burgers adjoint step at the edges of its 32 x 16 tiles and on the smallest periodic grids (halos
that wrap more than once), odd rows included, against the oracle's scatter-form adjoint with the
tolerances of the same comparison at other sizes."""
import numpy as np
import pytest

from multigpu_advectiondiffusion_gb300 import _native as N
from multigpu_advectiondiffusion_gb300.solvers import BurgersConfig, burgers_adjoint_step

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(6, 6, 6), (8, 7, 9), (31, 17, 7), (33, 15, 6), (32, 32, 8), (66, 18, 13)])
@pytest.mark.parametrize("weno", [N.ADV_WENO5_Z, N.ADV_WENO5_JS])
def test_adjoint_step_at_tile_edges(cuda, oracle, shape, weno):
    import torch
    nx, ny, nz = shape
    cfg = BurgersConfig(nx, ny, nz, 2.0 / nx, 2.0 / ny, 2.0 / nz, weno, N.ADV_LF_LOCAL, N.ADV_BC_PERIODIC, N.ADV_DIV_FAST)
    x, y, z = (np.arange(n) / n for n in shape)
    u0 = (0.3 + 0.5 * np.sin(6.28 * x)[None, None, :] * np.cos(6.28 * y)[None, :, None] - 0.3 * np.sin(6.28 * z)[:, None, None]).ravel()
    dt = 0.2 * cfg.dx
    un, u1, u2 = oracle.burgers_forward_states(cfg, u0, dt, 1)[0][0]
    lam = np.random.default_rng(nx).standard_normal(u0.size)
    want = oracle.burgers_step_adjoint(cfg, un, u1, u2, dt, lam)
    for dtype, tol in ((np.float64, 1e-12), (np.float32, 5e-5)):
        d = [torch.from_numpy(a.astype(dtype)).to(cuda) for a in (un, u1, u2, lam)]
        burgers_adjoint_step(cfg, d[0], d[1], d[2], dt, d[3])
        got = d[3].double().cpu().numpy()
        assert np.linalg.norm(got - want) < tol * np.linalg.norm(want), dtype
