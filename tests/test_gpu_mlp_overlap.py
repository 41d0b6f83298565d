"""A forward whose output buffer overlaps its inputs gives what separate
buffers give."""
import pytest

from gabe_b200 import emulator as em

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 129, 40000])
@pytest.mark.parametrize("at", [0, 3, 4])
def test_forward_into_the_inputs_buffer(n, at):
    import torch

    g = torch.Generator(device="cuda").manual_seed(n)
    with em.MLP(n_in=8, width=256, depth=2, n_out=32, max_rows=1 << 16, seed=3) as net:
        x = torch.randn((n, 8), generator=g, device="cuda")
        want = net.forward(x)
        # the inputs over the first or the last quarter of the output, or right behind it (no overlap)
        flat = torch.empty(n * 32 + n * 8, device="cuda")
        y = flat[: n * 32].view(n, 32)
        lo = at * n * 8
        xin = flat[lo : lo + n * 8].view(n, 8)
        xin.copy_(x)
        got = net.forward(xin, out=y)
        net.sync()
        assert torch.equal(got, want)
