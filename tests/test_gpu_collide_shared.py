"""Large swept-box batches (2^21 boxes and more, the grid in shared memory) against the same boxes in
batches below that size: the same verdicts for boxes inside one cell, across many, inverted, outside the
workspace, with NaNs and infinities, from misaligned arrays, with no obstacle and with enough obstacles
for one CTA per SM and for none."""
import numpy as np
import pytest

import kpax
import kpax_envs as E

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_obs,extra,shift", [(0, 0, 0), (1, 1, 1), (300, 3, 0), (1000, 31, 3), (2000, 2, 0), (6000, 1, 0)])
def test_shared_grid_gives_the_global_verdicts(cuda, n_obs, extra, shift):
    import torch

    cfg = kpax.preset(kpax.PRESET_QUAD)
    obs = E.random_boxes(n_obs, seed=n_obs) if n_obs else np.zeros((0, 6), np.float32)
    d_obs = torch.from_numpy(np.concatenate([obs, np.zeros((1, 6), np.float32)])).cuda()
    env = kpax.Env(cfg, d_obs.data_ptr(), n_obs)
    n = (1 << 21) + extra
    rng = np.random.default_rng(n_obs)
    lo = rng.uniform(-5, 105, (n, 3)).astype(np.float32)
    hi = (lo + rng.uniform(0, 0.2, (n, 3))).astype(np.float32)
    hi[: n // 50] = lo[: n // 50] + rng.uniform(0, 30, (n // 50, 3)).astype(np.float32)
    hi[n // 50: n // 40] = lo[n // 50: n // 40] - 1.0
    odd = np.array([np.nan, np.inf, -np.inf, 1e30, -1e30, 0.0, 100.0, 50.0], np.float32)
    lo[n // 40: n // 30], hi[n // 40: n // 30] = rng.choice(odd, (2, n // 30 - n // 40, 3))

    def dev(a):
        buf = torch.zeros(3 * n + 4, device="cuda")
        buf[shift: shift + 3 * n] = torch.from_numpy(a.ravel()).cuda()
        return buf

    b_lo, b_hi = dev(lo), dev(hi)
    out = torch.full((n + 8,), 7, dtype=torch.uint8, device="cuda")
    want = torch.full((n + 8,), 7, dtype=torch.uint8, device="cuda")
    p_lo, p_hi = b_lo.data_ptr() + 4 * shift, b_hi.data_ptr() + 4 * shift
    kpax.collide_batch(env, p_lo, p_hi, n, out.data_ptr() + shift)
    for i in range(0, n, 1 << 20):
        kpax.collide_batch(env, p_lo + 12 * i, p_hi + 12 * i, min(1 << 20, n - i), want.data_ptr() + shift + i)
    torch.cuda.synchronize()
    assert torch.equal(out, want)
    assert (out[shift: shift + n] <= 1).all() and (out[shift + n:] == 7).all()
