"""Grids of few obstacles over many cells, on either side of the number of (cell, obstacle) pairs up to which one
kernel builds them: the same entries and verdicts as from the three kernels that build grids of more than 256
obstacles (the same obstacles and inverted boxes, which cover no cells), and the same segments from the
allocation-free entry."""
import numpy as np
import pytest

import kpax
import kpax_envs as E

pytestmark = pytest.mark.gpu


# (obstacles, of them boxes over 8820 of the 9261 cells); up to 40, 80 and 256 obstacles the limits differ
@pytest.mark.parametrize("n,full", [(1, 1), (40, 1), (40, 29), (41, 3), (41, 4), (80, 3), (80, 4), (81, 1), (81, 2), (256, 1), (256, 2)])
def test_grids_of_large_boxes(cuda, n, full):
    import torch

    cfg = kpax.preset(kpax.PRESET_DI)
    obs = E.random_boxes(n, seed=n + full, side=(0.5, 4.0))
    at = np.random.default_rng(n).choice(n, full, replace=False)
    # over every cell but the topmost, and off the side that the queries are on, so that few of them hit
    obs[at] = np.array([-1.0, -1.0, -1.0, 101.0, 101.0, 95.5], np.float32)
    pad = np.tile(np.array([80.0, 80.0, 20.0, 20.0, 20.0, 80.0], np.float32), (300 - n, 1))
    padded = np.concatenate([obs, pad])
    d = [torch.from_numpy(np.ascontiguousarray(o)).cuda() for o in (obs, padded)]
    envs = [kpax.Env(cfg, x.data_ptr(), len(x)) for x in d]
    assert envs[0].stats() == envs[1].stats()
    assert envs[0].stats()[1] >= 8820 * full
    m = 20000
    rng = np.random.default_rng(full)
    lo = rng.uniform([0, 0, 90], [100, 100, 102], (m, 3)).astype(np.float32)
    hi = (lo + rng.uniform(0, 3, (m, 3))).astype(np.float32)
    d_lo, d_hi = torch.from_numpy(lo).cuda(), torch.from_numpy(hi).cuda()
    hit = ((hi[:, None] > obs[None, :, :3]) & (obs[None, :, 3:] > lo[:, None])).all(2).any(1)
    for e in envs:
        out = torch.full((m,), 7, dtype=torch.uint8, device="cuda")
        kpax.collide_batch(e, d_lo.data_ptr(), d_hi.data_ptr(), m, out.data_ptr())
        torch.cuda.synchronize()
        assert np.array_equal(out.cpu().numpy(), (~hit).astype(np.uint8))
    par = E.sample_states(cfg.model, 1021, 3, cfg.v_min, cfg.v_max)
    par[:, 2] = 96.0 + par[:, 2] / 50.0
    d_par = torch.from_numpy(par).cuda()
    rows = []
    for x in d:
        r = torch.zeros((1021, cfg.sample_dim), device="cuda")
        v = torch.zeros(1021, dtype=torch.uint8, device="cuda")
        kpax.propagate_batch_noalloc(cfg, x.data_ptr(), len(x), d_par.data_ptr(), None, 3, 1021, r.data_ptr(), v.data_ptr())
        torch.cuda.synchronize()
        rows.append((r, v))
    assert torch.equal(rows[0][0], rows[1][0]) and torch.equal(rows[0][1], rows[1][1])
    assert 0 < int(rows[0][1].sum()) < 1021
