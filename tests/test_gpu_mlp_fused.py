"""The one-launch emulator forward against the layer-by-layer kernels, at row
counts around a tile of 128 rows and around the switch from one to two tiles
per group, and at the shapes it takes.  An output pointer 8 bytes off a 16-byte
boundary has no tensor map, so the same call then runs layer by layer."""
import numpy as np
import pytest

from gabe_b200 import emulator as em

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(4, 256, 4, 192), (8, 64, 1, 64), (3, 128, 3, 96), (1, 256, 2, 32)])
def test_fused_forward_matches_layer_by_layer(shape):
    import torch

    n_in, width, depth, n_out = shape
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    g = torch.Generator(device="cuda")
    g.manual_seed(1)
    with em.MLP(n_in=n_in, width=width, depth=depth, n_out=n_out, seed=2, max_rows=1 << 17) as net:
        assert net.launches_per_forward == 1
        p = net.get_params()
        net.set_params(p + 0.05 * np.random.default_rng(3).standard_normal(p.size).astype(np.float32))
        for n in (1, 31, 33, 127, 128, 129, 128 * sms, 128 * sms + 1, 256 * sms + 130):
            x = torch.randn((n, n_in), generator=g, device="cuda")
            y = net.forward(x)
            flat = torch.full((n * n_out + 2,), float("nan"), device="cuda")  # 8-byte aligned
            z = net.forward(x, flat[2:].view(n, n_out))
            net.sync()
            assert torch.isfinite(y).all()
            # same activations; the output layer's FP32 sums may be ordered differently
            assert float((y - z).norm() / z.norm()) <= 1e-5, n
            assert float((y - z).abs().max()) <= 1e-4 * float(z.abs().max()), n
