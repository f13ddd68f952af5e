"""An allocation that fails is reported by its own call and by no later one."""
import numpy as np
import pytest

import kpax
import kpax_envs as E

pytestmark = pytest.mark.gpu


def test_calls_after_a_failed_allocation(cuda):
    import torch

    obs, s, g = E.di_scene()
    d = torch.from_numpy(np.ascontiguousarray(obs, np.float32)).cuda()
    cfg = kpax.preset(kpax.PRESET_DI)
    cfg.max_tree_size, cfg.expansions_per_iter, cfg.max_iter = 1 << 13, 1 << 10, 4
    env = kpax.Env(cfg, d.data_ptr(), len(obs))
    lo = torch.rand((1000, 3), device="cuda") * 100
    out = [torch.zeros(1000, dtype=torch.uint8, device="cuda") for _ in range(2)]
    planner = kpax.KPAX(cfg)
    sizes = [planner.plan(s, g, d.data_ptr(), len(obs)).tree_size]
    kpax.collide_batch(env, lo.data_ptr(), lo.data_ptr(), 1000, out[0].data_ptr())
    huge = cfg.copy()
    huge.max_tree_size = 1 << 24
    for later in (lambda: kpax.collide_batch(env, lo.data_ptr(), lo.data_ptr(), 1000, out[1].data_ptr()),
                  lambda: sizes.append(planner.plan(s, g, d.data_ptr(), len(obs)).tree_size)):
        with pytest.raises(kpax.KpaxError) as e:
            kpax.Batch([huge] * 400)  # half a terabyte
        assert e.value.status == kpax.ENOMEM
        later()
    torch.cuda.synchronize()
    assert torch.equal(out[0], out[1]) and min(sizes) > 1
