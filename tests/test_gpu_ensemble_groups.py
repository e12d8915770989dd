"""Burgers members of an ensemble with CTAs of their own (up to 64) and in one flat range (more), uneven
sizes: every member ends bit for bit where a run of its own does, and stops at its own step."""
import numpy as np
import pytest

from multigpu_advectiondiffusion_gb300 import _native as N
from multigpu_advectiondiffusion_gb300.solvers import BurgersConfig, Ensemble, burgers_run

pytestmark = pytest.mark.gpu


def _member(i, unaligned):
    sizes = [(96, 80, 70), (8, 8, 8), (36, 17, 40), (64, 33, 6), (16, 96, 11), (32, 16, 130)]
    if unaligned:
        sizes[1] = (37, 29, 9)
    nx, ny, nz = sizes[i % len(sizes)]
    return BurgersConfig(nx, ny, nz, 2.0 / nx, 2.0 / ny, 2.0 / nz, N.ADV_WENO5_Z, N.ADV_LF_GLOBAL, N.ADV_BC_PERIODIC)


@pytest.mark.parametrize("n,dtype,unaligned", [(1, np.float32, False), (3, np.float64, False), (6, np.float32, True),
                                               (64, np.float32, False), (65, np.float32, False), (67, np.float64, True)])
def test_members_end_where_their_own_runs_do(cuda, n, dtype, unaligned):
    import torch
    rng = np.random.default_rng(n)
    cfgs = [_member(i, unaligned) for i in range(n)]
    us = [torch.from_numpy((0.5 + 0.4 * rng.uniform(-1, 1, c.numel)).astype(dtype)).to(cuda) for c in cfgs]
    steps = [1 + i % 4 for i in range(n)]
    alone = [u.clone() for u in us]
    want = [burgers_run(c, u, 1e9, 0.2, N.ADV_DT_MAXU, max_steps=k) for c, u, k in zip(cfgs, alone, steps)]
    with torch.cuda.device(cuda):
        ens = Ensemble(burgers=[(c, u, 1e9, 0.2, N.ADV_DT_MAXU, k) for c, u, k in zip(cfgs, us, steps)])
    ens.run(0)
    for i in range(n):
        assert ens.burgers_result(i) == want[i]
        assert torch.equal(us[i], alone[i]), i
    ens.close()
