"""The fused FP32 WENO7 stage at the edges of its 32 x 16 tiles, on grids thinner than its stencil, in 2D
and 3D: right-hand side and runs (launched directly, and through the graph) against FP64, with the bounds
of the same comparisons at other sizes; both kinds of run give the same bits."""
import numpy as np
import pytest

from multigpu_advectiondiffusion_gb300.solvers import Weno7Config, weno7_rhs, weno7_run

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(32, 16, 9), (31, 17, 8), (33, 15, 10), (3, 2, 2), (66, 34, 5), (64, 33, 1), (35, 2, 1)])
def test_fused_stage_at_tile_edges(cuda, shape):
    import torch
    nx, ny, nz = shape
    cfg = Weno7Config(nx, ny, nz, *(2.0 / max(n - 1, 1) for n in shape))
    rng = np.random.default_rng(nx)
    u0 = rng.uniform(-0.6, 0.9, cfg.numel)
    got = {}
    for dtype in (np.float64, np.float32):
        u = torch.from_numpy(u0.astype(np.float32).astype(dtype)).to(cuda)
        L = torch.full_like(u, float("nan"))
        weno7_rhs(cfg, u, L)
        got[dtype] = L.double().cpu().numpy()
    ref = got[np.float64]
    assert np.linalg.norm(got[np.float32] - ref) <= 5e-6 * np.linalg.norm(ref)
    # four steps: at most eight are launched directly, an open step limit takes the graph
    a = torch.from_numpy(u0.astype(np.float32)).to(cuda)
    b = a.clone()
    t, steps = weno7_run(cfg, a, 1e9, 0.1, max_steps=4)
    assert steps == 4
    assert weno7_run(cfg, b, t, 0.1) == (t, 4) and torch.equal(a, b)
