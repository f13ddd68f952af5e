"""Loss and gradient at batch sizes around the kernels' row blocks (16 and 32 rows per CTA, the switch
between them at 16 rows per SM, 64-row splits of the weight gradients), and gathered rows: within the
bounds of test_gpu_learn.py's gradient test of the float64 oracle.  The parameters are a training
run's first ones, whose mixture has sigmas of about 1.8: where a sigma is far below 1 the loss
amplifies the outputs' rounding by its inverse, and FP32 gradients of any kernel miss a fixed bound."""
import numpy as np
import pytest

import kpax
import kpax_learn as L
import mlp_oracle as M

pytestmark = pytest.mark.gpu


def data(n, seed):
    rng = np.random.default_rng(seed)
    x = np.zeros((n, M.IN_PAD), np.float32)
    x[:, : M.IN] = rng.normal(0, 1, (n, M.IN))
    return x, rng.normal(0, 2, (n, M.DIM)).astype(np.float32)


@pytest.mark.parametrize("n", [1, 15, 17, 33, 63, 64, 129, 1025, 16 * 148, 16 * 148 + 1, 3001])
def test_gradient_around_the_row_blocks(cuda, n):
    import torch

    w = L.init_params(n)
    x, y = data(n, n)
    net = kpax.MLP(max_batch=n)
    net.set_params(w)
    d_x, d_y, d_g = torch.from_numpy(x).cuda(), torch.from_numpy(y).cuda(), torch.zeros(M.NUM_PARAMS, device="cuda")
    loss = net.loss_grad(d_x.data_ptr(), d_y.data_ptr(), n, d_g.data_ptr())
    l_ref, g_ref = M.loss_grad(w.astype(np.float64), x, y, (1, 1, 1, 1, 1))
    assert abs(loss - l_ref) <= 1e-5 * max(1.0, abs(l_ref))
    for name, a, b in zip(("W1", "b1", "W2", "b2", "W3", "b3"), M.unpack(d_g.cpu().numpy()), M.unpack(g_ref)):
        assert np.max(np.abs(a - b)) <= 1e-4 * max(np.max(np.abs(b)), 1e-12), name


def test_a_step_gathers_its_rows_and_keeps_the_transposed_weights(cuda):
    """A training step on rows idx, then the gradient at the new weights, equal the oracle's."""
    import torch

    w = L.init_params(3)
    x, y = data(500, 4)
    idx = np.random.default_rng(5).integers(0, 500, 200).astype(np.int32)
    net = kpax.MLP(max_batch=500)
    net.set_params(w)
    d_x, d_y, d_i = torch.from_numpy(x).cuda(), torch.from_numpy(y).cuda(), torch.from_numpy(idx).cuda()
    loss = net.train_step(d_x.data_ptr(), d_y.data_ptr(), d_i.data_ptr(), 200, 1e-3, want_loss=True)
    l_ref, g_ref = M.loss_grad(w.astype(np.float64), x[idx], y[idx], (1, 1, 1, 1, 1))
    assert abs(loss - l_ref) <= 1e-5 * max(1.0, abs(l_ref))
    m, _, _ = net.adam_state()
    assert np.max(np.abs(m - 0.1 * g_ref)) <= 1e-5 * np.max(np.abs(g_ref))
    w1 = net.get_params()
    d_g = torch.zeros(M.NUM_PARAMS, device="cuda")
    net.loss_grad(d_x.data_ptr(), d_y.data_ptr(), 500, d_g.data_ptr())
    _, g1 = M.loss_grad(w1.astype(np.float64), x, y, (1, 1, 1, 1, 1))
    for name, a, b in zip(("W1", "b1", "W2", "b2", "W3", "b3"), M.unpack(d_g.cpu().numpy()), M.unpack(g1)):
        assert np.max(np.abs(a - b)) <= 1e-4 * max(np.max(np.abs(b)), 1e-12), name
