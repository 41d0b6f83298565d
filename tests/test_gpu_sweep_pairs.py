"""The FP32 sweeps on packed pairs of sites against the FP64 sweeps: one step
at every tile shape, with marches of 1, 2, 3 and 5 planes and a remainder, both
potentials, with and without the GW sources.

Tolerance, from the operations: a value stored in FP32 and a chain of at most
sixteen roundings of terms no larger than |d| + dt |lap| + dt |V'|, with
|lap| <= 12 |f| / dx^2 for the seven-point sum and |V'| <= V2 |f| for the
potential's largest second derivative V2 over the fluctuations."""
import numpy as np
import pytest

import gabe_b200 as gb
from gabe_b200.autotune import shapes_for
from gabe_b200.ic import random_state

pytestmark = pytest.mark.gpu

EPS = 2.0 ** -24
DT, L = 5e-3, 20.0


def one_step(N, model, gws, precision, state, shape=-1, ci=0):
    f, d, a, ad = state
    with gb.Lattice(N, L=L, dt=DT, gws=gws, precision=precision, model=model, tile_shape=shape, tile_ci=ci) as lat:
        lat.upload_state(f, d, a0=a, adot0=ad)
        lat.step(1)
        out = lat.download_state(False)
        return out[0], out[1], lat.calc_energy()


@pytest.mark.parametrize("model", [gb.MODEL_QUADRATIC, gb.MODEL_LPHI4])
@pytest.mark.parametrize("gws", [False, True])
def test_one_step_of_every_shape(model, gws):
    for shape, (tk, tj) in shapes_for(gb.FP32).items():
        N = max(32, tk, tj)
        f, d, a, ad = random_state(N, L=L, seed=5 + shape, model=model)
        state = (f.numpy(), d.numpy(), a, ad)
        f64, d64, e64 = one_step(N, model, gws, gb.FP64, state)
        fl = np.abs(state[0] - state[0].mean(axis=(1, 2, 3), keepdims=True)).max()
        dl = np.abs(state[1] - state[1].mean(axis=(1, 2, 3), keepdims=True)).max()
        p2 = np.abs(state[0][0]).max() ** 2
        lam, g = (1.0 / 0.342 ** 2, 100.0 / 0.342 ** 2) if model == gb.MODEL_LPHI4 else (1.0 / p2, 2e-6)
        force = 12.0 / (L / N) ** 2 + 3.0 * lam * p2 + g * p2
        tol_d = 16 * EPS * (dl + DT * force * fl)
        tol_f = 16 * EPS * (fl + DT * dl) + DT * tol_d
        for ci in (1, 2, 3, 5):
            f32, d32, e32 = one_step(N, model, gws, gb.FP32, state, shape, ci)
            assert np.abs(f32 - f64).max() <= tol_f, (shape, ci)
            assert np.abs(d32 - d64).max() <= tol_d, (shape, ci)
            # sums of squares and products of such values: twice their relative error, and N^3 FP32
            # values summed in runs of at most sixteen
            for k in ("kin", "pot", "rho"):
                assert abs(e32[k] - e64[k]) <= 64 * EPS * abs(e64["rho"]), (shape, ci, k)
