"""Objects that live side by side: a batch plans the same whether or not another batch of another size
was created after it."""
import pytest

import kpax
import kpax_envs as E

pytestmark = pytest.mark.gpu

FIELDS = ("found", "goal_idx", "path_len", "tree_size", "iters", "tree_full", "expansions", "valid_expansions", "path_cost")
PRESETS = {kpax.MODEL_DOUBLE_INTEGRATOR: kpax.PRESET_DI, kpax.MODEL_DUBINS_AIRPLANE: kpax.PRESET_DUBINS,
           kpax.MODEL_QUADROTOR: kpax.PRESET_QUAD}


class _Queries:
    def __init__(self, n, block):
        import torch

        self.q = E.batch_queries(n, seed=n, obs_range=(10, 300), tree_range=(1 << 12, 1 << 14))
        self.obs = [torch.from_numpy(q["obstacles"]).cuda() for q in self.q]
        self.cfgs = []
        for q in self.q:
            c = kpax.preset(PRESETS[q["model"]])
            c.max_tree_size, c.expansions_per_iter, c.max_iter, c.block_size = q["tree"], 1 << 11, 10, block
            self.cfgs.append(c)

    def plan(self, batch):
        res, _ = batch.plan([q["start"] for q in self.q], [q["goal"] for q in self.q], [o.data_ptr() for o in self.obs],
                            [q["n_obs"] for q in self.q])
        return [{f: r[f] for f in FIELDS} for r in res]


@pytest.mark.parametrize("block", [0, 256, 512])
def test_a_batch_plans_the_same_after_another_one_was_created(cuda, block):
    large, small = _Queries(48, block), _Queries(3, block)
    want = []
    for s in (large, small):
        b = kpax.Batch(s.cfgs)
        want.append(s.plan(b))
        b.close()
    assert any(r["tree_size"] > 1 for r in want[0])
    a = kpax.Batch(large.cfgs)
    b = kpax.Batch(small.cfgs)  # smaller: needs less shared memory of the same kernels
    assert large.plan(a) == want[0]
    assert small.plan(b) == want[1]
    a.close()
    b.close()
