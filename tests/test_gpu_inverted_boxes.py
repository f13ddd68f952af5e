"""Obstacles whose lower corner lies above the upper one in some dimensions: they cover no cells, whichever
kernels build the grid (up to 256 obstacles one, above three), and the other obstacles are found as without
them."""
import itertools

import numpy as np
import pytest

import kpax
import kpax_envs as E

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("total", [255, 256, 257, 300])
@pytest.mark.parametrize("axes", [a for r in (1, 2, 3) for a in itertools.combinations(range(3), r)])
def test_inverted_boxes_cover_no_cells(cuda, total, axes):
    import torch

    cfg = kpax.preset(kpax.PRESET_QUAD)
    good = E.random_boxes(20, seed=7, side=(5.0, 15.0))
    rng = np.random.default_rng(total)
    bad = np.empty((total - 20, 6), np.float32)
    for i in range(len(bad)):  # five to six cells apart, and out to the workspace's corners
        lo = rng.uniform(0, 70, 3) if i % 8 else np.zeros(3)
        hi = lo + 28.0 if i % 8 else np.full(3, 100.0)
        for a in axes:
            lo[a], hi[a] = hi[a], lo[a]
        bad[i] = np.concatenate([lo, hi])
    obs = np.concatenate([bad[:100], good, bad[100:]])
    d_obs, d_good = torch.from_numpy(obs).cuda(), torch.from_numpy(good).cuda()
    env, want = kpax.Env(cfg, d_obs.data_ptr(), len(obs)), kpax.Env(cfg, d_good.data_ptr(), len(good))
    assert env.stats() == want.stats()
    m = 20000
    lo = rng.uniform(-5, 105, (m, 3)).astype(np.float32)
    hi = (lo + rng.uniform(0, 3, (m, 3))).astype(np.float32)
    d_lo, d_hi = torch.from_numpy(lo).cuda(), torch.from_numpy(hi).cuda()
    out = torch.full((m,), 7, dtype=torch.uint8, device="cuda")
    kpax.collide_batch(env, d_lo.data_ptr(), d_hi.data_ptr(), m, out.data_ptr())
    torch.cuda.synchronize()
    hit = ((hi[:, None] > good[None, :, :3]) & (good[None, :, 3:] > lo[:, None])).all(2).any(1)
    assert np.array_equal(out.cpu().numpy(), (~hit).astype(np.uint8))
