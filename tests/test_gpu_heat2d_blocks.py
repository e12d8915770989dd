"""2D FP32 runs in register blocks (heat2d_multi_kernel) at the edges of their tiles: 48- and 32-node
tiles of forward Euler, 52 and 40 of SSP-RK3, odd rows (scalar access), grids smaller than a block,
every remainder of the step count, against the oracle's step-by-step loop bit for bit."""
import numpy as np
import pytest

from multigpu_advectiondiffusion_gb300 import _native as N
from multigpu_advectiondiffusion_gb300.solvers import HeatConfig, heat_run

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("size", [(47, 49), (48, 96), (52, 53), (80, 41), (105, 31), (7, 7), (130, 200)])
@pytest.mark.parametrize("order,frozen,zero", [(2, 1, True), (4, 3, False), (4, 2, True)])
@pytest.mark.parametrize("time,nsteps", [(N.ADV_EULER, 2), (N.ADV_EULER, 19), (N.ADV_SSPRK3, 1), (N.ADV_SSPRK3, 2),
                                         (N.ADV_SSPRK3, 9)])
def test_blocks_equal_the_oracle(cuda, oracle, size, order, frozen, zero, time, nsteps):
    import torch
    nx, ny = size
    cfg = HeatConfig(2, nx, ny, 1, order, frozen, zero, 0.031, 0.023, 0.0, 0.7, time)
    u0 = np.random.default_rng(nx + nsteps).standard_normal(nx * ny).astype(np.float32)
    u = torch.from_numpy(u0).to(cuda)
    heat_run(cfg, u, nsteps)
    np.testing.assert_array_equal(u.cpu().numpy(), oracle.heat_run(cfg, u0, nsteps, time))
