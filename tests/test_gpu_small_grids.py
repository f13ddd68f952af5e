"""Obstacle grids built by one kernel (up to 256 obstacles on up to 12000 cells) against the same obstacles
padded with copies of the first past 256, which three kernels build: the same verdicts and the
entries that the copies add, with boxes inside a cell, across a few and over the whole grid, whose
entries outgrow the first entry list; and the allocation-free entry at its limit of entries."""
import numpy as np
import pytest

import kpax
import kpax_envs as E

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 7, 128, 255, 256])
@pytest.mark.parametrize("cell", [5.0, 4.6, 4.4, 30.0])
@pytest.mark.parametrize("side", [(0.01, 0.1), (5.0, 15.0), (90.0, 250.0)])
def test_one_kernel_grid_equals_three_kernels(cuda, n, cell, side):
    import torch

    cfg = kpax.preset(kpax.PRESET_QUAD)
    cfg.hash_cell_size = cell
    obs = E.random_boxes(n, seed=n, side=side)
    pad = 300 - n
    envs = []
    for o in (obs, np.concatenate([obs, np.repeat(obs[:1], pad, axis=0)]), obs[:1]):
        d = torch.from_numpy(np.ascontiguousarray(o, np.float32)).cuda()
        envs.append(kpax.Env(cfg, d.data_ptr(), len(o)))
    cells, ents = zip(*(e.stats() for e in envs))
    assert cells[0] == cells[1] and ents[1] == ents[0] + pad * ents[2]
    m = 20000
    rng = np.random.default_rng(n)
    lo = rng.uniform(-5, 105, (m, 3)).astype(np.float32)
    hi = (lo + rng.uniform(0, 3, (m, 3))).astype(np.float32)
    d_lo, d_hi = torch.from_numpy(lo).cuda(), torch.from_numpy(hi).cuda()
    out = [torch.full((m,), 7, dtype=torch.uint8, device="cuda") for _ in range(2)]
    for e, o in zip(envs, out):
        kpax.collide_batch(e, d_lo.data_ptr(), d_hi.data_ptr(), m, o.data_ptr())
    torch.cuda.synchronize()
    hit = ((hi[:, None] > obs[None, :, :3]) & (obs[None, :, 3:] > lo[:, None])).all(2).any(1)
    for o in out:
        assert np.array_equal(o.cpu().numpy(), (~hit).astype(np.uint8))


def test_allocation_free_entry_counts_before_it_fills(cuda):
    import torch

    cfg = kpax.preset(kpax.PRESET_DI)
    n = 257
    par = torch.from_numpy(E.sample_states(cfg.model, n, 3, cfg.v_min, cfg.v_max)).cuda()
    rows = torch.full((n, cfg.sample_dim), 5.0, device="cuda")
    valid = torch.full((n,), 7, dtype=torch.uint8, device="cuda")

    def run(k):
        obs = torch.tensor([[-1.0, -1, -1, 101, 101, 101]], device="cuda").repeat(k, 1)
        kpax.propagate_batch_noalloc(cfg, obs.data_ptr(), k, par.data_ptr(), None, 0, n, rows.data_ptr(), valid.data_ptr())
        torch.cuda.synchronize()

    with pytest.raises(kpax.KpaxError) as e:
        run(256)  # every cell holds all 256
    assert e.value.status == kpax.ECAPACITY
    assert (valid == 7).all() and (rows == 5.0).all()
    run(20)
    assert (valid == 0).all() and not (rows == 5.0).all()
