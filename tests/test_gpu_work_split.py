"""How a stage's (tile, plane) pairs are shared among CTAs never shows in its result: every pair once, at
sizes that take each form of the split (tile by tile, one range, the longer shares first or spread)."""
import numpy as np
import pytest

from multigpu_advectiondiffusion_gb300 import _native as N
from multigpu_advectiondiffusion_gb300.solvers import BurgersConfig, HeatConfig, burgers_stage, heat_run, heat_stage

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("size", [(224, 232, 240), (233, 233, 233), (256, 256, 193)])
def test_heat_stage_on_both_sides_of_the_l2(cuda, oracle, size):
    import torch
    cfg = HeatConfig(3, *size, 2, 1, True, 0.03, 0.02, 0.01, 0.5)
    u = np.random.default_rng(5).standard_normal(cfg.numel).astype(np.float32)
    a = torch.from_numpy(u).to(cuda)
    out = torch.full_like(a, float("nan"))
    heat_stage(cfg, 1, a, a, out)
    np.testing.assert_array_equal(out.cpu().numpy().view(np.uint8), oracle.heat_stage(cfg, 1, u, u).view(np.uint8))


@pytest.mark.parametrize("size", [(128, 300, 340), (320, 199, 201), (256, 192, 270)])
@pytest.mark.parametrize("frozen,zero", [(1, True), (2, False)])
def test_euler_steps_of_a_state_beyond_the_l2(cuda, oracle, size, frozen, zero):
    """Every second step walks its shares downwards in z (tiles of both widths, ragged rows)."""
    import torch
    cfg = HeatConfig(3, *size, 2, frozen, zero, 0.03, 0.02, 0.01, 0.5, N.ADV_EULER)
    u = np.random.default_rng(7).standard_normal(cfg.numel).astype(np.float32)
    a = torch.from_numpy(u).to(cuda)
    heat_run(cfg, a, 3)
    for _ in range(3):
        u = oracle.heat_stage(cfg, 1, u, u)
    np.testing.assert_array_equal(a.cpu().numpy().view(np.uint8), u.view(np.uint8))


@pytest.mark.parametrize("size", [(96, 96, 96), (128, 112, 101), (250, 200, 1), (40, 33, 64), (97, 65, 300)])
@pytest.mark.parametrize("dtype", [np.float32, np.float64])
def test_burgers_stage_of_a_rolled_state_is_the_rolled_stage(cuda, size, dtype):
    """On a periodic grid a shift along z moves every share's edges to other planes; each node's operations
    stay the same, so the states and the maximum agree bit for bit."""
    import torch
    nx, ny, nz = size
    if nz == 1:
        cfg = BurgersConfig.reference_2d(2.0, 2.0, nx, ny)
        shifts = (0,)
    else:
        cfg = BurgersConfig(nx, ny, nz, 2.0 / nx, 2.0 / ny, 2.0 / nz, N.ADV_WENO5_Z, N.ADV_LF_GLOBAL, N.ADV_BC_PERIODIC)
        shifts = (0, 1, nz // 3)
    u = np.random.default_rng(6).uniform(-1, 1, (nz, ny, nx)).astype(dtype)
    bits, real = (torch.int64, torch.float64) if dtype == np.float64 else (torch.int32, torch.float32)
    key = torch.zeros(1, dtype=bits, device=cuda)
    want = None
    for k in shifts:
        a = torch.from_numpy(np.ascontiguousarray(np.roll(u, k, 0)).ravel()).to(cuda)
        out = torch.full_like(a, float("nan"))
        key.zero_()
        burgers_stage(cfg, 1, a, a, out, 1e-3, 1.0, maxabs_key=key)
        got = np.roll(out.cpu().numpy().reshape(nz, ny, nx), -k, 0)
        assert np.isfinite(got).all()
        top = key.view(real).item()
        if nz > 1:
            assert top == np.abs(got).max()
        want = got if want is None else want
        np.testing.assert_array_equal(got, want)


@pytest.mark.parametrize("size", [(250, 200, 1), (1000, 90, 1), (33, 17, 1)])
@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("periodic", [True, False])
def test_burgers_2d_stage_and_maximum(cuda, oracle, size, dtype, periodic):
    """One plane: FP64 equals the oracle bit for bit, FP32 the FP32 oracle within 4e-7 of the maximum (two units of a state's
    rounding and four faces' at dt = h/20), and the key is the maximum of what was written."""
    import torch
    nx, ny, nz = size
    cfg = BurgersConfig(nx, ny, nz, 0.01, 0.01, 0.01, N.ADV_WENO5_Z, N.ADV_LF_GLOBAL, N.ADV_BC_PERIODIC) if periodic else \
        BurgersConfig.reference_2d(0.01 * (nx - 1), 0.01 * (ny - 1), nx, ny)
    rng = np.random.default_rng(8)
    u, un = (rng.uniform(-1, 1, cfg.numel).astype(dtype) for _ in range(2))
    bits, real = (torch.int64, torch.float64) if dtype == np.float64 else (torch.int32, torch.float32)
    key = torch.zeros(1, dtype=bits, device=cuda)
    a, b = (torch.from_numpy(v).to(cuda) for v in (u, un))
    out = torch.full_like(a, float("nan"))
    burgers_stage(cfg, 3, a, b, out, 5e-4, float(np.abs(u).max()), maxabs_key=key)
    got, want = out.cpu().numpy(), oracle.burgers_stage(cfg, 3, u, un, 5e-4)
    if dtype == np.float64:
        np.testing.assert_array_equal(got, want)
    else:
        assert np.abs(got - want).max() <= 4e-7 * np.abs(want).max()
    assert key.view(real).item() == np.abs(got).max()
