"""The FP64 sweeps' division by launch constants on the device: steps without
expansion (their fields depend on no energy sum) of states with signed zeros,
small and large values and, once a run has blown up, infinite Laplacians, against the oracle's
divisions bit for bit."""
import numpy as np
import pytest

import gabe_b200 as gb
from oracle import pyoracle as po

pytestmark = pytest.mark.gpu

N = 8


def _steps(model, field, dfield, n):
    cfg = po.Config(N=N, model=model, expansion=0)
    c0, c1, *_ = po.model_constants(model)
    st = po.init_state(cfg)
    st.field[0], st.dfield[0] = field, dfield
    a0 = st.sc.a[0] = st.sc.a[1] = 1.7
    with gb.Lattice(N, L=cfg.L, dt=cfg.dt, model=model, model_c=(c0, c1), expansion=0) as lat:
        lat.upload_state(field, dfield, a0=a0, adot0=st.sc.adot[0])
        lat.step(n)
        f, d = lat.download_state(False)[:2]
    po.step(st, n)
    return (f, d), (st.field[0], st.dfield[0])


def _same_bits(got, want):
    nan = np.isnan(want)
    np.testing.assert_array_equal(np.isnan(got), nan)
    np.testing.assert_array_equal(got[~nan].view(np.int64), want[~nan].view(np.int64))


@pytest.mark.parametrize("model", [po.MODEL_QUADRATIC, po.MODEL_LPHI4])
@pytest.mark.parametrize("case", ["ordinary", "zeros", "small", "large", "blown up"])
def test_steps_equal_the_oracle_bit_for_bit(case, model):
    rng = np.random.default_rng(11)
    f, d = rng.standard_normal((2, 2, N, N, N))
    steps = 1
    if case == "zeros":
        f, d = f * 0.0, d * 0.0  # zeros of both signs
    elif case == "small":
        f, d = f * 1e-250, d * 1e-250
    elif case == "large":
        f, d = f * 1e60, d * 1e60
    elif case == "blown up":  # one site overflows in the second step, its neighbours' Laplacians are infinite in the third
        f[:, 3, 4, 5] = 1e70
        steps = 3
    got, want = _steps(model, f, d, steps)
    for g, w in zip(got, want):
        _same_bits(g, w)
    if case == "blown up":
        assert np.isinf(want[0]).sum() > 2
