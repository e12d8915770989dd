"""The heat-with-k(x) step and adjoint step at the edges of their thread tiles (rows of whole vectors and
not, one to a few planes, grids smaller than a tile), against the oracle bit for bit."""
import numpy as np
import pytest

from multigpu_advectiondiffusion_gb300.solvers import HeatKConfig, heatk_adjoint_step, heatk_step

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(4, 3, 3), (3, 2, 1), (1, 1, 4), (64, 16, 2), (68, 17, 5), (63, 15, 3), (33, 34, 9),
                                   (30, 31, 40), (66, 33, 4)])
@pytest.mark.parametrize("zb", [True, False])
@pytest.mark.parametrize("dtype", [np.float32, np.float64])
def test_steps_at_tile_edges(cuda, oracle, shape, zb, dtype):
    import torch
    nx, ny, nz = shape
    cfg = HeatKConfig(nx, ny, nz, 0.11, 0.07, 0.05, zb)
    rng = np.random.default_rng(nx + nz)
    k, u, lam, g = (rng.uniform(0.2, 1.0, cfg.numel).astype(dtype) for _ in range(4))
    kt, ut, lt, gt = (torch.from_numpy(v.copy()).to(cuda) for v in (k, u, lam, g))
    out = torch.full_like(ut, float("nan"))
    heatk_step(cfg, kt, ut, out)
    np.testing.assert_array_equal(out.cpu().numpy(), oracle.heatk_step(shape, zb, (0.11, 0.07, 0.05), k, u))
    out.fill_(float("nan"))
    heatk_adjoint_step(cfg, kt, ut, lt, out, gt)
    want_g = g.copy()
    want_lam = oracle.heatk_adjoint(shape, zb, (0.11, 0.07, 0.05), k, u, lam, want_g)
    np.testing.assert_array_equal(out.cpu().numpy(), want_lam)
    np.testing.assert_array_equal(gt.cpu().numpy(), want_g)
