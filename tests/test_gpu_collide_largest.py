"""The largest swept-box batch that the entry's 32-bit count allows, whose last stride passes 2^32."""
import pytest

import kpax
import kpax_envs as E

pytestmark = pytest.mark.gpu


def test_the_largest_batch_ends_and_finds_every_hit(cuda):
    import torch

    n = (1 << 32) - 1
    if torch.cuda.mem_get_info()[0] < 80 << 30:
        pytest.skip("needs 80 GB of device memory")
    cfg = kpax.preset(kpax.PRESET_QUAD)
    obs = E.quad_scene(n_total=1000)[0]
    d_obs = torch.from_numpy(obs).cuda()
    env = kpax.Env(cfg, d_obs.data_ptr(), len(obs))
    assert env.stats()[1] >= 4096  # large enough for the kernel with the grid in shared memory
    boxes = torch.full((n, 3), -7.0, device="cuda")  # points outside the workspace: free
    inside = torch.from_numpy((obs[0, :3] + obs[0, 3:]) / 2).cuda()
    hits = [0, 1 << 31, (1 << 32) - 303105, (1 << 32) - 303104, n - 1]
    for i in hits:
        boxes[i] = inside
    free = torch.full((n,), 7, dtype=torch.uint8, device="cuda")
    kpax.collide_batch(env, boxes.data_ptr(), boxes.data_ptr(), n, free.data_ptr())
    torch.cuda.synchronize()
    assert int(free.amax()) == 1
    assert n - int(torch.count_nonzero(free)) == len(hits)
    assert all(int(free[i]) == 0 for i in hits)
    env.close()
    del boxes, free
    torch.cuda.empty_cache()
