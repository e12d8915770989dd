"""The fused FP32 WENO7 stage at the edges of its 32 x 16 tiles, on grids thinner than its stencil, in 2D
and 3D: right-hand side and runs (launched directly, and through the graph) against FP64, with the bounds
of the same comparisons at other sizes; both kinds of run give the same bits."""
import numpy as np
import pytest

from multigpu_advectiondiffusion_gb300.solvers import Weno7Config, weno7_rhs, weno7_run, weno7_workspace

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


@pytest.mark.parametrize("dtype,shape,steps", [(np.float32, (40, 36, 20), 8), (np.float32, (40, 36, 1), 8),
                                               (np.float64, (40, 36, 1), 2), (np.float64, (24, 20, 17), 8)])
def test_steps_past_the_end_do_no_work(cuda, native, dtype, shape, steps):
    """A run that reaches tEnd after one of the steps it may take: the same state and step count as a run limited to that
    step, nothing more written to its work arrays (faces or stages), no launch more counted."""
    import torch
    cfg = Weno7Config(*shape, *(2.0 / max(n - 1, 1) for n in shape))
    u0 = np.random.default_rng(3).uniform(-0.6, 0.9, cfg.numel).astype(dtype)
    t, _ = weno7_run(cfg, torch.from_numpy(u0).to(cuda), 1e9, 0.1, max_steps=1)
    got = []
    for limit in (1, steps):
        u = torch.from_numpy(u0).to(cuda)
        ws = weno7_workspace(cfg, u)
        ws.zero_()
        before = native.adv_kernel_launch_count()
        assert weno7_run(cfg, u, t, 0.1, max_steps=limit, workspace=ws) == (t, 1)
        launched = native.adv_kernel_launch_count() - before
        fields = 4 * ((u.numel() * u.element_size() + 255) // 256 * 256)
        got.append((u, ws.view(torch.uint8)[:fields], launched))
    assert torch.equal(got[0][0], got[1][0])
    assert torch.equal(got[0][1], got[1][1])
    if dtype == np.float32:  # (the larger FP64 run is a graph)
        assert got[0][2] == got[1][2]
