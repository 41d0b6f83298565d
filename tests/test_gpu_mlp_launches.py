"""gabe_mlp_launches_per_train_step follows the batch that was trained last."""
import pytest

from gabe_b200 import emulator as em

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("fp32_act", [False, True])
def test_launches_per_train_step_follow_the_batch(fp32_act):
    import torch

    n = 5000  # above the rows of a small batch
    x, t = torch.randn((n, 3), device="cuda"), torch.randn((n, 192), device="cuda")
    perm = torch.arange(n, dtype=torch.int32, device="cuda")
    with em.MLP(max_rows=n, fp32_act=fp32_act) as net:
        forward, layers = net.launches_per_forward, 5
        small = 2 + forward + (layers - 1) + 2  # gather, forward, loss, data gradients, weight gradients, update
        # weight gradients and reductions by layer, update, BF16 weights
        large = 2 + forward + (layers - 1) + 2 * layers + 1 + (not fp32_act)
        assert net.launches_per_train_step == small
        for batch, want in ((n, large), (512, small), (4097, large), (4096, small)):
            net.reset_batches()
            net.train_batches(x, t, perm, batch, 1)
            assert net.launches_per_train_step == want, batch
        net.sync()
