"""The fused iterations at budgets around the widths their expansion takes (tiles only as wide as spreads
the children over 148 CTAs, one to fourteen warps; one child; one tile per CTA exactly; one child more,
which takes tiles by look-back), and with one to many iterations per launch: the per-stage kernels'
plan, bit for bit."""
import pytest

import kpax
import kpax_envs as E
from test_gpu_fused import run, same

pytestmark = pytest.mark.gpu
CTAS = 148


@pytest.mark.parametrize("budget", [1, 31, CTAS - 1, CTAS * 32, CTAS * 32 + 1, CTAS * 288 + 5, CTAS * 448, CTAS * 448 + 1])
def test_budgets_around_the_tile_widths(cuda, budget):
    import torch

    cfg = kpax.preset(kpax.PRESET_DUBINS)
    cfg.expansions_per_iter, cfg.max_tree_size, cfg.max_iter = budget, 1 << 17, 12
    cfg.children_per_entry, cfg.root_repeat = 1024, 254  # the root fills the budget at once
    obs, s, g = E.dubins_scene()
    same(run(torch, cfg, obs, s, g, 0), run(torch, cfg, obs, s, g, 1))


@pytest.mark.parametrize("unroll", [1, 2, 7, 64])
def test_iterations_per_launch_leave_the_plan_unchanged(cuda, unroll):
    import torch

    cfg = kpax.preset(kpax.PRESET_DI)
    cfg.max_tree_size, cfg.expansions_per_iter, cfg.max_iter = 1 << 15, 1 << 12, 15
    cfg.v_min, cfg.v_max, cfg.unroll_iters = -5.0, 5.0, unroll
    obs, s, g = E.di_scene()
    fused, staged = run(torch, cfg, obs, s, g, 0), run(torch, cfg, obs, s, g, 1)
    same(fused, staged)
    assert fused["res"][4] == 15
