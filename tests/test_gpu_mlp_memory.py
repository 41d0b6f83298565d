"""The small-batch training buffers stay within their bound: a wide network's
handle holds what its parameters, moments and activations take and at most 256
MB more, and batches beyond the rows that fit there take the tiled kernels,
with the same gradient."""
import numpy as np
import pytest

from gabe_b200 import emulator as em

pytestmark = pytest.mark.gpu

MB = 1 << 20


def test_wide_network_footprint_and_gradient():
    import torch

    n_in, W, depth, n_out, R = 4, 2048, 8, 64, 4096
    x = torch.randn((R, n_in), device="cuda", generator=torch.Generator(device="cuda").manual_seed(1))
    t = torch.randn((R, n_out), device="cuda", generator=torch.Generator(device="cuda").manual_seed(2))
    with em.MLP(n_in=n_in, depth=1, max_rows=16) as warm:  # context and module loading
        warm.loss_grad(x[:16], torch.zeros((16, 192), device="cuda"))
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    with em.MLP(n_in=n_in, width=W, depth=depth, n_out=n_out, max_rows=R) as net:
        used = free - torch.cuda.mem_get_info()[0]
        P = net.num_params
        need = 4 * P * 4                                   # parameters, gradients, moments
        need += R * (n_in + 3 * n_out + 2 * W) * 4         # batch, outputs and their gradient, two deltas
        need += 2 * depth * R * W * 2                      # kept activations (BF16)
        need += 16 * W * W * 4 + (P - n_in * W) * 2        # split-K partials, BF16 weights
        assert need - 64 * MB <= used <= need + (256 + 48) * MB, (used / MB, need / MB)  # allocations are of whole 2 MB
        n = 2000  # small batch; its rows twice do not fit the buffers
        _, one = net.loss_grad(x[:n], t[:n])
        _, two = net.loss_grad(torch.cat([x[:n], x[:n]]), torch.cat([t[:n], t[:n]]))
    assert np.linalg.norm(one) > 0
    assert np.linalg.norm(one - two) / np.linalg.norm(one) <= 2e-5
