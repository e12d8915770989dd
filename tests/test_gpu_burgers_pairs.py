"""The fused Burgers stage at the edges of its tiles and pairs: two columns per thread, row pairs in
the x-faces, one warp for the faces left over, rows TMA can and cannot describe (even rows with
element copies among them), a 2D member in a batch of 3D ones."""
import numpy as np
import pytest

from multigpu_advectiondiffusion_gb300 import _native as N
from multigpu_advectiondiffusion_gb300.solvers import BurgersConfig, Ensemble, burgers_run, burgers_stage

pytestmark = pytest.mark.gpu

# tile edges 32 x 16 +- 1, one plane past the pipeline's depth, thin and minimal grids
SIZES = [(31, 15, 9), (33, 17, 8), (32, 16, 7), (34, 18, 11), (64, 33, 6), (6, 6, 6), (66, 7, 13), (130, 9, 3)]


def _cfg(size, bc, weno, lf):
    nx, ny, nz = size
    c = BurgersConfig(nx, ny, nz, 2.0 / nx, 2.0 / ny, 2.0 / nz, weno, lf, bc)
    if bc == N.ADV_BC_FROZEN:
        c.C = 1e-2
    return c


def _field(cfg, seed):
    rng = np.random.default_rng(seed)
    x, y, z = (np.arange(n) / n for n in (cfg.nx, cfg.ny, cfg.nz))
    u = 0.2 + 0.6 * np.sin(6.28 * x)[None, None, :] * np.cos(6.28 * y)[None, :, None] - 0.3 * np.sin(6.28 * z)[:, None, None]
    return (u + 0.05 * rng.standard_normal(u.shape)).ravel()


@pytest.mark.parametrize("size", SIZES)
@pytest.mark.parametrize("bc,weno,lf", [(N.ADV_BC_PERIODIC, N.ADV_WENO5_Z, N.ADV_LF_GLOBAL),
                                        (N.ADV_BC_FROZEN, N.ADV_WENO5_JS, N.ADV_LF_LOCAL)])
def test_stage_at_tile_edges(cuda, oracle, size, bc, weno, lf):
    """FP64 bit for bit; FP32 within 4e-7 max|u| of the FP32 oracle and the FP64 fast form within
    1e-14 max|u| of the FP64 one (the tolerances of the same comparisons at other sizes)."""
    import torch
    if bc == N.ADV_BC_PERIODIC and min(size) < 6:
        pytest.skip("periodic grids need 6 cells per axis")
    cfg = _cfg(size, bc, weno, lf)
    uin, un = _field(cfg, 1), _field(cfg, 2)
    alpha = float(np.abs(uin).max())
    for dtype, div, tol in [(np.float64, N.ADV_DIV_F32, 0.0), (np.float64, N.ADV_DIV_FAST, 1e-14),
                            (np.float32, N.ADV_DIV_F32, 4e-7), (np.float32, N.ADV_DIV_FAST, 4e-7)]:
        cfg.div = div
        a, b = (torch.from_numpy(v.astype(dtype)).to(cuda) for v in (uin, un))
        out = torch.full_like(a, float("nan"))
        burgers_stage(cfg, 2, a, b, out, 1e-3, alpha)
        want = oracle.burgers_stage(cfg, 2, uin.astype(dtype), un.astype(dtype), 1e-3)
        assert np.abs(out.cpu().numpy().astype(float) - want.astype(float)).max() <= tol * alpha


def test_batch_with_a_2d_member_equals_single_runs(cuda):
    import torch
    cfgs = [BurgersConfig.reference_2d(2.0, 2.0, 40, 36), BurgersConfig.reference(2.0, 2.0, 2.0, 24, 20, 16, C=0.0)]
    cfgs[1].weno = cfgs[0].weno
    us = [torch.from_numpy(_field(c, 3 + i).astype(np.float32)).to(cuda) for i, c in enumerate(cfgs)]
    alone = [u.clone() for u in us]
    for c, u in zip(cfgs, alone):
        burgers_run(c, u, 1e9, 0.2, N.ADV_DT_FIXED, max_steps=5)
    ens = Ensemble(burgers=[(c, u, 1e9, 0.2, N.ADV_DT_FIXED, 5) for c, u in zip(cfgs, us)])
    ens.run(0)
    for u, w in zip(us, alone):
        assert torch.equal(u, w)
    ens.close()
