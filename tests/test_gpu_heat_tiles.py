"""The heat stage's one-node-per-thread tiles (FP64: 16 x 16; FP32 rows TMA cannot describe: 32 wide) at
their edges, all stages, and subnormal / zero / huge states through stage 3's division, against the oracle
bit for bit."""
import numpy as np
import pytest

from multigpu_advectiondiffusion_gb300 import _native as N
from multigpu_advectiondiffusion_gb300.solvers import HeatConfig, heat_stage

pytestmark = pytest.mark.gpu


def _check(cuda, oracle, cfg, stage, uin, un):
    import torch
    a, b = (torch.from_numpy(v).to(cuda) for v in (uin, un))
    if stage == 1:
        b = a
    out = torch.full_like(a, float("nan"))
    heat_stage(cfg, stage, a, b, out)
    np.testing.assert_array_equal(out.cpu().numpy().view(np.uint8),
                                  oracle.heat_stage(cfg, stage, uin, uin if stage == 1 else un).view(np.uint8))


@pytest.mark.parametrize("size", [(15, 17, 5), (16, 16, 6), (17, 33, 7), (31, 65, 5), (33, 31, 9), (66, 15, 6), (97, 34, 1),
                                  (45, 130, 1)])
@pytest.mark.parametrize("order", [2, 4])
@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("stage", [1, 2, 3])
def test_tiles_at_their_edges(cuda, oracle, size, order, dtype, stage):
    nx, ny, nz = size
    cfg = HeatConfig(2 if nz == 1 else 3, nx, ny, nz, order, order // 2, order == 2, 0.031, 0.017, 0.023 if nz > 1 else 0.0,
                     0.6)
    rng = np.random.default_rng(nx + stage)
    _check(cuda, oracle, cfg, stage, *(rng.standard_normal(cfg.numel).astype(dtype) for _ in range(2)))


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("scale", [0.0, -0.0, 1e-320, 1e-300, 1e-43, 1e-37, 1e30, 1e37, 1e300])
@pytest.mark.parametrize("stage", [2, 3])
def test_extreme_states(cuda, oracle, dtype, scale, stage):
    """Scales the type cannot hold are left out; the states stay below overflow of the stencil's sums."""
    if dtype == np.float32 and not (scale == 0.0 or 1e-44 < scale < 2e37):
        pytest.skip("outside FP32")
    for nx in (32, 33):  # both load paths
        cfg = HeatConfig(3, nx, 12, 8, 2, 1, True, 0.03, 0.02, 0.01, 0.5)
        rng = np.random.default_rng(3)
        with np.errstate(under="ignore"):
            u, v = ((scale * rng.uniform(-1, 1, cfg.numel)).astype(dtype) for _ in range(2))
        if scale == 0.0:
            u[:], v[:] = scale, scale
        _check(cuda, oracle, cfg, stage, u, v)
