"""A collision query per step (steps that may go far against a grid cell) against a query per group of steps:
the grid's cell size chooses between them and changes no verdict, so rows, verdicts, step counts and plans are
the same on both sides of the line, in every kernel that integrates segments."""
import numpy as np
import pytest

import kpax
import kpax_envs as E

pytestmark = pytest.mark.gpu


def _config(model):
    """A preset whose five steps go up to 2.5 m (quadrotor: 3 m), with cells that group them or not."""
    cfg = kpax.preset({1: kpax.PRESET_DI, 2: kpax.PRESET_DUBINS, 3: kpax.PRESET_QUAD}[model])
    if model == 1:
        cfg.v_min, cfg.v_max = -5.0, 5.0
        for d in range(3):
            cfg.ctrl_min[d], cfg.ctrl_max[d] = -4.0, 4.0
    if model == 2:
        cfg.step_size = 0.25
    out = []
    for cell in (5.0, 1.9):
        c = cfg.copy()
        c.hash_cell_size = cell
        out.append(c)
    return out


def _scene(model):
    if model == 1:
        return E.di_scene()
    return E.dubins_scene() if model == 2 else E.quad_scene(n_total=400)


@pytest.mark.parametrize("model", [1, 2, 3])
@pytest.mark.parametrize("n", [1, 257, 5003, (1 << 18) - 1, (1 << 18) + 1, (1 << 19) + 3])
@pytest.mark.parametrize("given", [False, True])
def test_segments(cuda, model, n, given):
    import torch

    obs = torch.from_numpy(np.ascontiguousarray(_scene(model)[0], np.float32)).cuda()
    cfgs = _config(model)
    par = torch.from_numpy(E.sample_states(model, n, 3, cfgs[0].v_min, cfgs[0].v_max)).cuda()
    draws = torch.from_numpy(E.uniform_draws(n, 5)).cuda() if given else None
    out = []
    for cfg in cfgs:
        env = kpax.Env(cfg, obs.data_ptr(), len(obs))
        rows = torch.full((n, cfg.sample_dim), 7.0, device="cuda")
        valid = torch.full((n,), 7, dtype=torch.uint8, device="cuda")
        steps = torch.full((n,), -7, dtype=torch.int32, device="cuda")
        kpax.propagate_batch(cfg, env, par.data_ptr(), draws.data_ptr() if given else None, 9, n, rows.data_ptr(),
                             valid.data_ptr(), steps.data_ptr())
        torch.cuda.synchronize()
        out.append((rows, valid, steps))
        env.close()
    for a, b in zip(*out):
        assert torch.equal(a, b)
    assert n == 1 or 0 < int(out[0][1].sum()) < n


@pytest.mark.parametrize("model", [1, 2, 3])
@pytest.mark.parametrize("block,kernels", [(0, 0), (128, 0), (256, 0), (512, 0), (0, 1), (256, 1)])
def test_plans(cuda, model, block, kernels):
    import torch

    obs, s, g = _scene(model)
    d = torch.from_numpy(np.ascontiguousarray(obs, np.float32)).cuda()
    out = []
    for cfg in _config(model):
        cfg.max_tree_size, cfg.expansions_per_iter, cfg.max_iter = 1 << 16, 1 << 13, 12
        cfg.block_size, cfg.iteration_kernels = block, kernels
        pl = kpax.KPAX(cfg)
        r = pl.plan(s, g, d.data_ptr(), len(obs))
        rows, parents, costs = pl.export_tree()
        out.append((r.found, r.iters, r.expansions, r.valid_expansions, rows.tobytes(), parents.tobytes(), costs.tobytes()))
        pl.close()
    assert out[0] == out[1]


def test_learned_plan(cuda):
    import torch

    import kpax_learn as L

    obs, s, g = _scene(3)
    d = torch.from_numpy(np.ascontiguousarray(obs, np.float32)).cuda()
    net = L.load_network(L.DEFAULT_WEIGHTS)
    out = []
    for cfg in _config(3):
        cfg.max_tree_size, cfg.expansions_per_iter, cfg.max_iter = 1 << 16, 1 << 13, 10
        pl = kpax.KPAX(cfg)
        pl.set_proposal(net, 0.3)
        r = pl.plan(s, g, d.data_ptr(), len(obs))
        out.append((r.iters, r.valid_expansions, pl.export_tree()[0].tobytes()))
        pl.close()
    assert out[0] == out[1]


@pytest.mark.parametrize("block", [0, 256, 512])
@pytest.mark.parametrize("mode", ["", "0", "2"])
def test_batches_of_both_kinds(cuda, block, mode, monkeypatch):
    import torch

    if mode:
        monkeypatch.setenv("KPAX_BATCH_EXPAND", mode)
    cfgs, scenes = [], []
    for model in (3, 1, 2, 3, 1, 2):  # of the second three queries only the quadrotor's asks for a query per step
        cfg = _config(model)[1 if len(cfgs) == 3 else 0]
        cfg.max_tree_size, cfg.expansions_per_iter, cfg.max_iter, cfg.block_size = 1 << 15, 1 << 12, 8, block
        cfg.seed = 40 + len(cfgs)
        cfgs.append(cfg)
        scenes.append(_scene(model))
    obs = [torch.from_numpy(np.ascontiguousarray(o, np.float32)).cuda() for o, _, _ in scenes]
    batch = kpax.Batch(cfgs)
    res, _ = batch.plan([s for _, s, _ in scenes], [g for _, _, g in scenes], [o.data_ptr() for o in obs], [len(o) for o in obs])
    batch.close()
    fields = ("found", "tree_size", "iters", "expansions", "valid_expansions", "path_cost")
    for q, cfg in enumerate(cfgs):
        pl = kpax.KPAX(cfg)
        r = pl.plan(scenes[q][1], scenes[q][2], obs[q].data_ptr(), len(obs[q]))
        assert {f: res[q][f] for f in fields} == {f: getattr(r, f) for f in fields}, q
        pl.close()


@pytest.mark.parametrize("model", [1, 2, 3])
def test_warp_planner(cuda, model):
    import torch

    obs, s, g = _scene(model)
    d = torch.from_numpy(np.ascontiguousarray(obs, np.float32)).cuda()
    out = []
    for cfg in _config(model):
        rk = kpax.ReKinoLite(cfg, num_warps=64, samples_per_thread=16, max_iterations=20, timeout_ms=60000.0)
        r, path = rk.plan(s, g, d.data_ptr(), len(obs))
        out.append((r.expansions, r.valid_expansions) if not r.found else (r.goal_idx, r.iters, path.tobytes()))
        rk.close()
    assert out[0] == out[1]
