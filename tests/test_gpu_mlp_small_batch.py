"""The small-batch backward (data gradients, one launch of weight gradients,
one of reduction and update) against the tiled kernels that larger batches
take: a last row without finite targets adds nothing to the gradient, so 4096
rows (small) and those rows plus one such row (large) have the same one."""
import numpy as np
import pytest

from gabe_b200 import emulator as em

pytestmark = pytest.mark.gpu

SMALL = 4096  # rows up to which a batch takes the small-batch kernels


@pytest.mark.parametrize("shape,fp32_act", [((4, 256, 4, 192), False), ((4, 256, 4, 192), True), ((5, 64, 2, 6), False),
                                            ((3, 320, 1, 130), True)])
def test_small_batch_gradient_matches_the_tiled_kernels(shape, fp32_act):
    import torch

    n_in, width, depth, n_out = shape
    g = torch.Generator(device="cuda")
    g.manual_seed(6)
    x = torch.randn((SMALL + 1, n_in), generator=g, device="cuda")
    t = torch.randn((SMALL + 1, n_out), generator=g, device="cuda")
    t[SMALL] = float("nan")
    with em.MLP(n_in=n_in, width=width, depth=depth, n_out=n_out, seed=2, max_rows=SMALL + 1, fp32_act=fp32_act) as net:
        l0, g0 = net.loss_grad(x[:SMALL], t[:SMALL])
        l1, g1 = net.loss_grad(x, t)
    assert l0 == pytest.approx(l1, rel=1e-12)
    # FP32 sums over 4096 rows in two orders: a few eps sqrt(4096) of the norm
    assert np.linalg.norm(g0 - g1) / np.linalg.norm(g1) <= 2e-5
    assert np.linalg.norm(g1) > 0


@pytest.mark.parametrize("rows", [1, 15, 17, 33, 512, 1000])
def test_gradient_of_odd_row_counts_is_the_mean_of_its_rows(rows):
    import torch

    g = torch.Generator(device="cuda")
    g.manual_seed(rows)
    x = torch.randn((rows, 4), generator=g, device="cuda")
    t = torch.randn((rows, 192), generator=g, device="cuda")
    with em.MLP(n_in=4, seed=3, max_rows=2 * rows, fp32_act=True) as net:
        _, one = net.loss_grad(x, t)
        _, two = net.loss_grad(torch.cat([x, x]), torch.cat([t, t]))
    assert np.linalg.norm(one - two) / np.linalg.norm(one) <= 2e-5
