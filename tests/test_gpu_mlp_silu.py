"""The forward's SiLU, z / (1 + 2^(-z log2 e)) on the approximate exponential
and reciprocal, against FP64, tails included.

A network of one input, unit first-layer weights and an identity output layer
returns its hidden activations exactly: with FP32 activations the scalar form
as computed, with BF16 activations the packed form rounded to BF16.

Bound, from the operations: the exponent t = -z log2 e carries two roundings
(of log2 e and of the product), 1.5 |t| 2^-24 ln 2 of the exponential at most;
ex2.approx 2^-22, rcp.approx 2^-23 and the roundings of the sum and the product
2^-24 each, 2^-21 together; results below the smallest normal number times |z|
may be flushed."""
import numpy as np
import pytest

from gabe_b200 import emulator as em

pytestmark = pytest.mark.gpu


def _arguments():
    rng = np.random.default_rng(2)
    tails = [np.linspace(-104, -80, 20001), np.linspace(80, 104, 2001), np.linspace(-30, 30, 60001)]
    wide = [s * 2.0 ** rng.uniform(-100, 99, 20000) for s in (-1.0, 1.0)]
    z = np.concatenate([*tails, *wide, [0.0, -0.0, 1.0, -1.0]]).astype(np.float32)
    return z[np.abs(z) < 1e30]


def _hidden(z, fp32_act):
    import torch

    W = 64
    with em.MLP(n_in=1, width=W, depth=1, n_out=W, max_rows=1 << 17, fp32_act=fp32_act) as net:
        assert net.launches_per_forward == (2 if fp32_act else 1)
        p = np.zeros(net.num_params, np.float32)
        p[:W] = 1.0                                          # W0: every unit's z is the input
        p[2 * W:2 * W + W * W] = np.eye(W, dtype=np.float32).ravel()  # after b0: W1
        net.set_params(p)
        y = net.forward(torch.tensor(z[:, None], device="cuda"))
        net.sync()
        assert bool((y == y[:, :1]).all())
        return y[:, 0].cpu()


def test_silu_scalar_and_packed_forms():
    import torch

    z = _arguments()
    scalar = _hidden(z, True)
    z64 = z.astype(np.float64)
    with np.errstate(over="ignore"):
        exact = z64 / (1.0 + np.exp(-z64))
    bound = (1.5 * np.abs(z64) * 2.0 ** -24 + 2.0 ** -21) * np.abs(exact) + np.abs(z64) * 2.0 ** -126 + 2.0 ** -149
    err = np.abs(scalar.numpy().astype(np.float64) - exact)
    assert np.all(err <= bound), z[np.argmax(err / bound)]
    # the packed form rounds each half as the scalar one: the same values after the BF16 store
    packed = _hidden(z, False)
    assert torch.equal(packed, scalar.to(torch.bfloat16).float())
