"""The one-launch forward against the layer-by-layer tcgen05 kernels bit for
bit, the layer-by-layer kernels at a width that only they take, and a training
step with an odd output count.

A network of eight inputs takes the one-launch forward; the same network with
a ninth input of zeros does not, and its first layer runs on another kernel.
The inputs, first-layer weights and biases are small integers that make every
z an integer of 40 to 136: its SiLU rounds to z in BF16 on either kernel, so
both networks' later layers see the same activations and run the same products
in the same order on tcgen05."""
import numpy as np
import pytest

from gabe_b200 import emulator as em

pytestmark = pytest.mark.gpu


def _pair_params(W, depth, n_out, seed):
    """Flat parameters for n_in = 8, and the same with a ninth row of W0."""
    rng = np.random.default_rng(seed)
    W0 = rng.integers(0, 4, (8, W)).astype(np.float32)
    rest = [np.full(W, 40.0, np.float32)]
    for l in range(1, depth + 1):
        N = n_out if l == depth else W
        rest.append((rng.standard_normal((W, N)) * 0.05).astype(np.float32).ravel())
        rest.append((rng.standard_normal(N) * 0.1).astype(np.float32))
    ninth = rng.standard_normal(W).astype(np.float32)
    return np.concatenate([W0.ravel(), *rest]), np.concatenate([W0.ravel(), ninth, *rest])


@pytest.mark.parametrize("W,depth,n_out", [(256, 4, 192), (64, 1, 64), (128, 3, 96), (256, 2, 32)])
def test_one_launch_forward_equals_the_layered_kernels(W, depth, n_out):
    import torch

    sms = torch.cuda.get_device_properties(0).multi_processor_count
    p8, p9 = _pair_params(W, depth, n_out, 3)
    kw = dict(width=W, depth=depth, n_out=n_out, max_rows=1 << 16)
    with em.MLP(n_in=8, **kw) as a, em.MLP(n_in=9, **kw) as b:
        assert a.launches_per_forward == 1 and b.launches_per_forward == depth + 1
        assert all(b.forward_form(l) == "tcgen05" for l in range(1, depth + 1))
        a.set_params(p8)
        b.set_params(p9)
        g = torch.Generator(device="cuda").manual_seed(5)
        for n in (1, 31, 33, 127, 128, 129, 128 * sms, 128 * sms + 1, 256 * sms + 130):
            x8 = torch.randint(0, 5, (n, 8), generator=g, device="cuda").float()
            x9 = torch.cat([x8, torch.zeros((n, 1), device="cuda")], 1)
            ya, yb = a.forward(x8), b.forward(x9)
            a.sync(), b.sync()
            assert torch.isfinite(ya).all() and torch.equal(ya, yb), n
            # the activations and pre-activations kept for training: the same gradients
            t = torch.randn((n, n_out), generator=g, device="cuda")
            (la, ga), (lb, gb) = a.loss_grad(x8, t), b.loss_grad(x9, t)
            assert la == lb
            np.testing.assert_array_equal(ga[:8 * W], gb[:8 * W], err_msg=str(n))
            np.testing.assert_array_equal(ga[8 * W:], gb[9 * W:], err_msg=str(n))
            assert np.linalg.norm(ga[8 * W + W:]) > 0


@pytest.mark.parametrize("n_in,W,depth,n_out", [(3, 192, 3, 192), (12, 256, 2, 64)])
def test_layered_tcgen05_kernels_match_mma_sync(n_in, W, depth, n_out):
    import torch

    kw = dict(n_in=n_in, width=W, depth=depth, n_out=n_out, seed=4, max_rows=1 << 15)
    with em.MLP(**kw) as a, em.MLP(mma_sync=True, **kw) as b:
        assert a.launches_per_forward == depth + 1
        assert all(a.forward_form(l) == "tcgen05" for l in range(1, depth + 1))
        p = a.get_params()
        p += 0.05 * np.random.default_rng(6).standard_normal(p.size).astype(np.float32)
        a.set_params(p)
        b.set_params(p)
        for n in (1, 127, 128, 130, 20000):
            x = torch.randn((n, n_in), generator=torch.Generator(device="cuda").manual_seed(n), device="cuda")
            ya, yb = a.forward(x), b.forward(x)
            a.sync(), b.sync()
            # the two SiLUs differ by FP32 roundings, which flips the BF16 rounding (2^-9) of few activations
            assert float((ya - yb).norm() / yb.norm()) <= 2e-3, n


@pytest.mark.parametrize("n_out", [1, 7, 33])
@pytest.mark.parametrize("fp32_act", [True, False])
def test_training_step_with_an_odd_output_count(n_out, fp32_act):
    import torch

    from oracle import mlp_oracle as mo

    rows = 300
    x, t = torch.randn((rows, 5), device="cuda"), torch.randn((rows, n_out), device="cuda")
    perm = torch.arange(rows, dtype=torch.int32, device="cuda")
    kw = dict(n_in=5, width=64, depth=2, n_out=n_out, max_rows=512, fp32_act=fp32_act)
    with em.MLP(lr=3e-3, weight_decay=0.01, seed=8, **kw) as net, em.MLP(**kw) as fresh:
        p = net.get_params()
        _, g = net.loss_grad(x, t)
        net.train_batches(x, t, perm, rows, 1)
        net.sync()
        p1 = net.get_params()
        z = np.zeros_like(p)
        want, _, _ = mo.adamw_step(p, g, z, z.copy(), 1, lr=3e-3, wd=0.01)
        np.testing.assert_allclose(p1, want, rtol=1e-6, atol=1e-7)
        # the step's BF16 weights are those of its parameters
        fresh.set_params(p1)
        y0, y1 = net.forward(x), fresh.forward(x)
        net.sync(), fresh.sync()
        assert torch.equal(y0, y1)
