"""Objects that live side by side: a batch plans the same whether or not another batch of another size
was created after it, and swept-box queries of environments of different sizes run from several threads
at once."""
import threading

import numpy as np
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


def test_swept_box_queries_of_two_grids_from_two_threads(cuda):
    import torch

    cfg = kpax.preset(kpax.PRESET_QUAD)
    n, calls = 1 << 21, 3000  # from 2^21 boxes on the grid is held in shared memory, of the size that it needs
    rng = np.random.default_rng(3)
    lo = rng.uniform(0, 100, (n, 3)).astype(np.float32)
    d_lo, d_hi = torch.from_numpy(lo).cuda(), torch.from_numpy(lo + np.float32(0.2)).cuda()
    work = []
    for obstacles in (500, 3000):
        obs = torch.from_numpy(E.random_boxes(obstacles, seed=obstacles, side=(5.0, 8.0))).cuda()
        env = kpax.Env(cfg, obs.data_ptr(), obstacles)
        out = [torch.zeros(n, dtype=torch.uint8, device="cuda") for _ in range(2)]
        kpax.collide_batch(env, d_lo.data_ptr(), d_hi.data_ptr(), n, out[0].data_ptr())
        work.append((env, out, torch.cuda.Stream()))
    torch.cuda.synchronize()
    errors = []

    def loop(env, out, stream):
        try:
            for _ in range(calls):
                kpax.collide_batch(env, d_lo.data_ptr(), d_hi.data_ptr(), n, out[1].data_ptr(), stream.cuda_stream)
        except kpax.KpaxError as e:
            errors.append(str(e))

    threads = [threading.Thread(target=loop, args=w) for w in work]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    torch.cuda.synchronize()
    assert not errors, errors
    for _, out, _ in work:
        assert torch.equal(out[0], out[1])
