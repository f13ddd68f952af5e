"""The FP32 forward pass with its outputs over its inputs (rows of 64 features in, of 96 outputs out) gives what
separate buffers give, at one block of rows and several."""
import pytest

import kpax
import kpax_learn as L

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 16, 17, 1000, 2369, 4096])
@pytest.mark.parametrize("shift", [0, 32, 64])
def test_outputs_over_inputs(cuda, n, shift):
    import torch

    net = kpax.MLP(max_batch=n)
    net.set_params(L.init_params(3))
    x = torch.randn((n, kpax.MLP_FEATURES), generator=torch.Generator(device="cuda").manual_seed(n), device="cuda")
    want = torch.zeros((n, kpax.MLP_OUTPUTS), device="cuda")
    net.forward(x.data_ptr(), n, want.data_ptr())
    buf = torch.zeros(n * kpax.MLP_OUTPUTS + 2 * shift, device="cuda")
    src = buf[shift:shift + n * kpax.MLP_FEATURES]
    for at in (0, shift, 2 * shift):  # outputs that start before, at and after the inputs
        src.copy_(x.view(-1))
        net.forward(src.data_ptr(), n, buf[at:].data_ptr())
        assert torch.equal(buf[at:at + want.numel()].view_as(want), want), at
