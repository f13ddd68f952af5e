"""The allocation-free entry, which runs every batch in one pass, against the entry whose batches of this size run
in phases: two of them in groups of steps, three with a query per step."""
import numpy as np
import pytest

import kpax
import kpax_envs as E

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("preset,n,cell", [(kpax.PRESET_QUAD, (1 << 18) + 3, 5.0), (kpax.PRESET_QUAD, (1 << 18) + 3, 2.1),
                                           (kpax.PRESET_QUAD_REF, (1 << 18) + 1, 5.0), (kpax.PRESET_DUBINS, (1 << 19) + 5, 5.0)])
def test_phased_batches(cuda, preset, n, cell):
    import torch

    cfg = kpax.preset(preset)
    cfg.hash_cell_size = cell
    obs = E.dubins_scene()[0] if preset == kpax.PRESET_DUBINS else E.quad_scene(n_total=300)[0]
    d = torch.from_numpy(np.ascontiguousarray(obs, np.float32)).cuda()
    par = torch.from_numpy(E.sample_states(cfg.model, n, 3, max(cfg.v_min, -5.0), min(cfg.v_max, 5.0))).cuda()
    env = kpax.Env(cfg, d.data_ptr(), len(obs))
    out = []
    for alloc in (True, False):
        rows = torch.zeros((n, cfg.sample_dim), device="cuda")
        valid = torch.zeros(n, dtype=torch.uint8, device="cuda")
        steps = torch.zeros(n, dtype=torch.int32, device="cuda")
        args = (par.data_ptr(), None, 4, n, rows.data_ptr(), valid.data_ptr(), steps.data_ptr())
        if alloc:
            kpax.propagate_batch(cfg, env, *args)
        else:
            kpax.propagate_batch_noalloc(cfg, d.data_ptr(), len(obs), *args)
        torch.cuda.synchronize()
        out.append((rows, valid, steps))
    for a, b in zip(*out):
        assert torch.equal(a, b)
    assert 0 < int(out[0][1].sum()) < n
