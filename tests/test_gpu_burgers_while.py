"""A Burgers run of any number of steps equals the same steps taken one run at a time, whatever the number
of steps in the loop's body, and a run that ends on its time ends there."""
import numpy as np
import pytest

from multigpu_advectiondiffusion_gb300 import _native as N
from multigpu_advectiondiffusion_gb300.solvers import BurgersConfig, burgers_run

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("steps", [1, 2, 3, 4, 5, 7, 8, 9])
def test_steps_of_one_run_equal_single_steps(cuda, oracle, steps):
    import torch
    cfg = BurgersConfig.periodic(20, weno="z")
    u0 = torch.from_numpy(oracle.ic_burgers_fourier(20, 20, 20, 2.0, 3)).to(cuda)
    one, many = u0.clone(), u0.clone()
    t_one = 0.0
    for _ in range(steps):
        t, n = burgers_run(cfg, one, 1e9, 0.4, N.ADV_DT_MAXU, max_steps=1)
        assert n == 1
        t_one += t
    t, n = burgers_run(cfg, many, 1e9, 0.4, N.ADV_DT_MAXU, max_steps=steps)
    assert n == steps and t == t_one
    assert torch.equal(one, many)
    # the end time inside the run: the steps up to it, the last one trimmed, nothing after it
    part = u0.clone()
    t_end, n_end = burgers_run(cfg, part, t_one * 0.6, 0.4, N.ADV_DT_MAXU, max_steps=1000)
    want, t_w, n_w = oracle.burgers_run(cfg, u0.cpu().numpy(), t_one * 0.6, 0.4, 1)
    assert t_end == t_w and n_end == n_w
    np.testing.assert_array_equal(part.cpu().numpy(), want)
