"""Segments whose length is not a multiple of the steps that share one collision query (three or five,
kpax_device.cuh: run_steps): the rows, verdicts and step counts of the oracle, which queries every
step, at lengths around the groups' ends, with obstacles dense enough that many segments end
inside a group."""
import numpy as np
import pytest

import kpax
import kpax_envs as E
import oracle as O
from test_gpu_kernels import PRESETS, bits, compare_segments, gpu_propagate

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name", list(PRESETS))
@pytest.mark.parametrize("length", [1, 2, 3, 4, 5, 6, 7, 11, 16])
def test_segment_lengths_around_the_groups(cuda, name, length):
    import torch

    cfg = kpax.preset(PRESETS[name])
    cfg.max_propagation_duration = length
    obs = E.random_boxes(600, seed=length)
    n = 3001
    par = E.sample_states(cfg.model, n, 50 + length, cfg.v_min, cfg.v_max)
    rows, valid, steps, _ = gpu_propagate(torch, cfg, obs, par, None, stream_id=length)
    orow, oval, ostep, margin, _, _ = O.propagate(cfg, obs, par, None, stream=length)
    if cfg.model == kpax.MODEL_DOUBLE_INTEGRATOR:
        assert np.array_equal(bits(rows), bits(orow)) and np.array_equal(valid, oval) and np.array_equal(steps, ostep)
    else:
        compare_segments(cfg, rows, valid, orow, oval, margin, name)
        assert np.array_equal(steps[margin >= 1e-4], ostep[margin >= 1e-4])
    assert 0 < oval.sum() < n
