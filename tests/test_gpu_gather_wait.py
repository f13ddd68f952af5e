"""The bounded wait of the fused iteration's gathers: every thread of a CTA gives up alike when the other CTA's
word never carries the tag, whether no word was written or one of an earlier or later iteration (tags compare in
30 bits), and the sums are right when it does; plans run as before afterwards."""
import ctypes

import numpy as np
import pytest

import kpax
import kpax_envs as E


def _hook():
    fn = kpax.load().kpax_test_gather_timeout
    u32 = ctypes.c_uint32
    fn.restype, fn.argtypes = ctypes.c_int32, [u32, u32, u32, ctypes.POINTER(u32), ctypes.c_void_p]
    return fn


def _gather(spin_limit, tag, peer):
    """Status and (threads that gave up, sum of the values, sum below) of one CTA's gather over two."""
    out = (ctypes.c_uint32 * 3)()
    return _hook()(spin_limit, tag, peer, out, None), list(out)


def test_arguments_are_checked_without_a_gpu():
    fn, out = _hook(), (ctypes.c_uint32 * 3)()
    assert fn(0, 1, 0, out, None) == kpax.EINVAL
    assert fn(16, 0, 0, out, None) == kpax.EINVAL
    assert fn((1 << 22) + 1, 1, 0, out, None) == kpax.EINVAL
    assert fn(16, 1, 0, None, None) == kpax.EINVAL


@pytest.mark.gpu
@pytest.mark.parametrize("tag,peer", [(1, 0), (7, 6), (7, 8), ((1 << 30) - 1, (1 << 30) - 2), (1 << 30, (1 << 30) - 1)])
def test_a_missing_or_stale_word_ends_the_wait(cuda, tag, peer):
    status, (gave_up, _, _) = _gather(1 << 10, tag, peer)
    assert status == kpax.ETIMEOUT and gave_up == 64


@pytest.mark.gpu
@pytest.mark.parametrize("tag", [1, 7, (1 << 30) - 1, (1 << 30) + 5])
def test_the_tagged_word_is_summed(cuda, tag):
    assert _gather(1 << 10, tag, tag) == (kpax.OK, [0, 12, 0])


@pytest.mark.gpu
def test_plans_run_after_a_wait_that_ended(cuda):
    import torch

    obs, s, g = E.di_scene()
    d = torch.from_numpy(np.ascontiguousarray(obs, np.float32)).cuda()
    cfg = kpax.preset(kpax.PRESET_DI)
    cfg.max_tree_size, cfg.expansions_per_iter, cfg.max_iter = 1 << 14, 1 << 11, 6
    out = []
    for _ in range(2):
        pl = kpax.KPAX(cfg)
        r = pl.plan(s, g, d.data_ptr(), len(obs))
        out.append((r.tree_size, r.valid_expansions))
        pl.close()
        assert _gather(1 << 10, 3, 2)[0] == kpax.ETIMEOUT
    assert out[0] == out[1]
