"""FP64 Burgers stages over constant, zero, subnormal and tiny states and over tiles with columns and rows past
the domain or in the frozen layers, bit for bit against the oracle: the divisions' numerators reach zero
there, and whole warps have no face to reconstruct."""
import numpy as np
import pytest

from multigpu_advectiondiffusion_gb300 import _native as N
from multigpu_advectiondiffusion_gb300.solvers import BurgersConfig, burgers_stage

pytestmark = pytest.mark.gpu

SIZES = [(36, 20, 9), (33, 35, 8), (97, 98, 7), (35, 16, 10), (34, 19, 9), (32, 51, 7), (40, 50, 1)]


@pytest.mark.parametrize("size", SIZES)
@pytest.mark.parametrize("state", ["zero", "constant", "half", "tiny", "subnormal", "steps"])
@pytest.mark.parametrize("bc,weno,C", [(N.ADV_BC_PERIODIC, N.ADV_WENO5_Z, 0.0), (N.ADV_BC_FROZEN, N.ADV_WENO5_Z, 1e-2),
                                       (N.ADV_BC_FROZEN, N.ADV_WENO5_JS, 0.0)])
def test_stage_over_zero_numerators(cuda, oracle, size, state, bc, weno, C):
    import torch
    nx, ny, nz = size
    if nz == 1:
        if bc == N.ADV_BC_PERIODIC:
            pytest.skip("2D grids are frozen")
        cfg = BurgersConfig.reference_2d(2.0, 2.0, nx, ny)
    else:
        cfg = BurgersConfig(nx, ny, nz, 2.0 / nx, 2.0 / ny, 2.0 / nz, weno, N.ADV_LF_LOCAL, bc)
        cfg.C = C
    rng = np.random.default_rng(4)
    u = rng.uniform(-1, 1, (nz, ny, nx))
    if state == "zero":
        u[:] = 0.0
        u[:, :, : nx // 3] = -0.0
    elif state == "constant":
        u[:] = 0.7
    elif state == "half":
        u[:, :, nx // 2:] = 0.0
        u[:, ny // 2:, :] = -0.25
    elif state == "tiny":
        u *= 1e-60
    elif state == "subnormal":
        u *= 1e-310
    else:
        u = np.round(2 * u) / 2
    u = np.ascontiguousarray(u).ravel()
    un = rng.permutation(u)
    for stage in (1, 3):
        base = u if stage == 1 else un
        a, b = (torch.from_numpy(v).to(cuda) for v in (u, base))
        out = torch.full_like(a, float("nan"))
        burgers_stage(cfg, stage, a, b, out, 1e-3, float(np.abs(u).max()))
        np.testing.assert_array_equal(out.cpu().numpy().view(np.uint8),
                                      oracle.burgers_stage(cfg, stage, u, base, 1e-3).view(np.uint8))


@pytest.mark.parametrize("size", [(36, 20, 9), (35, 16, 10), (40, 50, 1)])
@pytest.mark.parametrize("scale", [1e38, 1e39, 1e60])
def test_js_weights_that_all_underflow(cuda, oracle, size, scale):
    """From |u| of about 1e39 on, every (eps + beta)^2 overflows, the weights are 0 and a side is 0/0: NaN, as in
    the scheme as written (constant lines, whose indicators vanish, stay finite)."""
    import torch
    nx, ny, nz = size
    cfg = BurgersConfig.reference_2d(2.0, 2.0, nx, ny) if nz == 1 else BurgersConfig(
        nx, ny, nz, 2.0 / nx, 2.0 / ny, 2.0 / nz, N.ADV_WENO5_JS, N.ADV_LF_LOCAL, N.ADV_BC_PERIODIC)
    cfg.weno, cfg.C = N.ADV_WENO5_JS, 0.0
    u = scale * np.random.default_rng(4).uniform(-1, 1, (nz, ny, nx))
    u[:, : ny // 2] = 0.25 * scale
    u = u.ravel()
    want = oracle.burgers_stage(cfg, 1, u, u, 1e-3 / scale)
    assert np.isnan(want).any() == (scale > 1e38) and np.isfinite(want).any()
    a = torch.from_numpy(u).to(cuda)
    out = torch.zeros_like(a)
    burgers_stage(cfg, 1, a, a, out, 1e-3 / scale, scale)
    np.testing.assert_array_equal(out.cpu().numpy(), want)


@pytest.mark.parametrize("size", [(36, 20, 9), (35, 16, 10), (33, 35, 8)])
@pytest.mark.parametrize("scale", [1e77, 2e77, 1e78, 1e100])
def test_z_indicators_that_are_all_infinite(cuda, oracle, size, scale):
    """tau = |beta0 - beta2| of two infinite indicators is NaN, and so is the side: NaN wherever the scheme as
    written gives one. (3D: on a 2D grid the oracle also reconstructs the equal z-faces, whose rounding overflows
    at this scale; the stage leaves them out.)"""
    import torch
    nx, ny, nz = size
    cfg = BurgersConfig(nx, ny, nz, 2.0 / nx, 2.0 / ny, 2.0 / nz, N.ADV_WENO5_Z, N.ADV_LF_LOCAL, N.ADV_BC_PERIODIC)
    u = scale * np.random.default_rng(4).uniform(-1, 1, (nz, ny, nx))
    u[:, : ny // 2] = 0.25 * scale
    u = u.ravel()
    want = oracle.burgers_stage(cfg, 1, u, u, 1e-3 / scale)
    assert np.isnan(want).any()
    a = torch.from_numpy(u).to(cuda)
    out = torch.zeros_like(a)
    burgers_stage(cfg, 1, a, a, out, 1e-3 / scale, scale)
    assert np.isnan(out.cpu().numpy())[np.isnan(want)].all()


@pytest.mark.parametrize("size", [(36, 20, 9), (35, 16, 10), (33, 35, 8)])
@pytest.mark.parametrize("scale", [6.5e76, 8e76, 1.1e77])
def test_indicators_whose_first_difference_squared_overflows(cuda, oracle, size, scale):
    """C^2 beyond the largest number where C^2/4 is not: finite indicators, finite results."""
    import torch
    nx, ny, nz = size
    cfg = BurgersConfig(nx, ny, nz, 2.0 / nx, 2.0 / ny, 2.0 / nz, N.ADV_WENO5_Z, N.ADV_LF_LOCAL, N.ADV_BC_PERIODIC)
    u = scale * np.random.default_rng(4).uniform(-1, 1, nx * ny * nz)
    want = oracle.burgers_stage(cfg, 1, u, u, 1e-3 / scale)
    assert np.isfinite(want).any()
    a = torch.from_numpy(u).to(cuda)
    out = torch.zeros_like(a)
    burgers_stage(cfg, 1, a, a, out, 1e-3 / scale, scale)
    np.testing.assert_array_equal(out.cpu().numpy(), want)


@pytest.mark.parametrize("dtype,scale", [(np.float64, 7e76), (np.float32, 2.6e9)])
def test_sweep_where_the_first_difference_squared_overflows(cuda, native, oracle, dtype, scale):
    import torch
    u = (scale * np.random.default_rng(4).uniform(-1, 1, (9, 9, 40))).astype(dtype)
    want = oracle.burgers_sweep_all(0, True, u, 0.1, np.zeros_like(u))
    a = torch.from_numpy(u.ravel()).to(cuda)
    L = torch.zeros_like(a)
    assert native.adv_ref_burgers_sweep_all(N.ADV_F64 if dtype == np.float64 else N.ADV_F32, 0, N.ADV_WENO5_Z, 40, 40, 9,
                                            9, 0.1, a.data_ptr(), L.data_ptr(), None) == N.ADV_OK
    np.testing.assert_array_equal(L.cpu().numpy().reshape(u.shape), want)
