"""Segment batches at the sizes and lengths from which they run in two phases (2^18 quadrotor or 2^19
6-state segments of more than ten steps): the same rows, verdicts and step counts as slices of 2^17,
which one kernel runs in one pass."""
import numpy as np
import pytest

import kpax
import kpax_envs as E
from test_gpu_kernels import bits

pytestmark = pytest.mark.gpu

SIZES = [("di", 1 << 19, 10), ("di", 1 << 19, 11), ("dubins", (1 << 19) - 1, 20), ("dubins", 1 << 19, 11),
         ("dubins", (1 << 19) + 33, 20), ("quad", (1 << 18) - 1, 25), ("quad", 1 << 18, 11), ("quad", (1 << 18) + 31, 25)]


@pytest.mark.parametrize("name,n,length", SIZES)
@pytest.mark.parametrize("obstacles", [1, 2000])
def test_two_phases_equal_one_pass(cuda, name, n, length, obstacles):
    import torch

    cfg = kpax.preset({"di": kpax.PRESET_DI, "dubins": kpax.PRESET_DUBINS, "quad": kpax.PRESET_QUAD}[name])
    cfg.max_propagation_duration = length
    d_obs = torch.from_numpy(E.random_boxes(obstacles, 7).astype(np.float32)).cuda()
    env = kpax.Env(cfg, d_obs.data_ptr(), obstacles)
    par = torch.from_numpy(E.sample_states(cfg.model, n, 5, cfg.v_min, cfg.v_max)).cuda()
    draws = torch.from_numpy(np.ascontiguousarray(E.uniform_draws(n, 6)[:, :5])).cuda()

    def run(step):
        rows = torch.zeros((n, cfg.sample_dim), device="cuda")
        valid, steps = torch.zeros(n, dtype=torch.uint8, device="cuda"), torch.zeros(n, dtype=torch.int32, device="cuda")
        for lo in range(0, n, step):
            m = min(n, lo + step) - lo
            kpax.propagate_batch(cfg, env, par[lo:].data_ptr(), draws[lo:].data_ptr(), 0, m, rows[lo:].data_ptr(),
                                 valid[lo:].data_ptr(), steps[lo:].data_ptr())
        torch.cuda.synchronize()
        return rows.cpu().numpy(), valid.cpu().numpy(), steps.cpu().numpy()

    a, b = run(n), run(1 << 17)
    assert np.array_equal(bits(a[0]), bits(b[0]))
    assert np.array_equal(a[1], b[1]) and np.array_equal(a[2], b[2])
    assert 0 < a[1].mean() < 1
