"""A plan call that is refused leaves its planner or batch as it was: a null obstacle buffer is reported before
any query's grid is rebuilt, so the proposal can be set and the next plan is the one of a fresh batch."""
import numpy as np
import pytest

import kpax
import kpax_envs as E
import kpax_learn as L

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("missing", [0, 1, 2])
def test_batch_after_a_refused_plan(cuda, missing):
    import torch

    net = L.load_network(L.DEFAULT_WEIGHTS)
    few, s, g = E.quad_scene(n_total=40)
    many = E.quad_scene(n_total=2000)[0]  # its entries do not fit the lists of the few
    cfg = kpax.preset(kpax.PRESET_QUAD)
    cfg.max_tree_size, cfg.expansions_per_iter, cfg.max_iter = 1 << 14, 1 << 11, 6
    d_few, d_many = torch.from_numpy(few).cuda(), torch.from_numpy(many).cuda()

    def plan(batch, d, n, null=None):
        ptrs = [0 if q == null else d.data_ptr() for q in range(3)]
        res, _ = batch.plan([s] * 3, [g] * 3, ptrs, [n] * 3)
        return [(r["tree_size"], r["iters"], r["valid_expansions"], r["path_cost"]) for r in res]

    want = []
    fresh = kpax.Batch([cfg] * 3)
    want.append(plan(fresh, d_few, len(few)))
    fresh.set_proposal(net, 0.3)
    want.append(plan(fresh, d_few, len(few)))
    fresh.close()
    batch = kpax.Batch([cfg] * 3)
    assert plan(batch, d_few, len(few)) == want[0]
    with pytest.raises(kpax.KpaxError) as e:
        plan(batch, d_many, len(many), missing)
    assert e.value.status == kpax.EINVAL
    batch.set_proposal(net, 0.3)
    assert plan(batch, d_few, len(few)) == want[1]
    batch.close()


def test_planner_after_a_refused_plan(cuda):
    import torch

    obs, s, g = E.quad_scene(n_total=300)
    cfg = kpax.preset(kpax.PRESET_QUAD)
    cfg.max_tree_size, cfg.expansions_per_iter, cfg.max_iter = 1 << 14, 1 << 11, 6
    d = torch.from_numpy(obs).cuda()
    sizes = []
    for refused in (False, True):
        pl = kpax.KPAX(cfg)
        pl.begin(s, g, d.data_ptr(), len(obs))
        pl.iterate(2)
        if refused:
            with pytest.raises(kpax.KpaxError):
                pl.begin(s, g, 0, len(obs))
        pl.iterate(2)
        sizes.append((pl.finish().tree_size, np.asarray(pl.export_tree()[1]).tobytes()))
        pl.close()
    assert sizes[0] == sizes[1]
