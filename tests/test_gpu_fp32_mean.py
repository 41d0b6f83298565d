"""FP32 storage keeps the mean of the force: over 300 steps of 256^3 the
energies and the scale factor follow the FP64 run to what unbiased roundings
leave in the mean field.

Tolerance, from the operations: a step rounds the momentum fluctuation at most
eight times by up to 2^-24 of |d| + dt F |f|, F = 12 / dx^2 the largest
coefficient of the force, and the field by as much of |f|; unbiased and
independent from site to site and step to step they leave the means
e_d = 8 2^-24 (rms d + dt F rms f) sqrt(steps / N^3) and
e_f = 8 2^-24 rms f sqrt(steps / N^3) + T e_d.  The potential is V' / V e_f
(lambda phi^4: 4 e_f / phi) off, the kinetic energy 2 e_d / phi', their sum and
with it a and a' by no more than the larger of the two.  A force whose small
terms are lost in the rounding of the Laplacian is off by 5e-12 here."""
import numpy as np
import pytest

import gabe_b200 as gb
from gabe_b200.ic import random_state

pytestmark = pytest.mark.gpu


def test_energies_follow_the_fp64_run():
    N, steps, dt, L = 256, 300, 1.0 / 256, 20.0
    f, d, a, ad = random_state(N, L=L, seed=1, model=gb.MODEL_LPHI4, device="cuda")
    f, d = f.cpu().numpy(), d.cpu().numpy()
    rms = lambda x: np.sqrt(np.mean((x - x.mean(axis=(1, 2, 3), keepdims=True)) ** 2, axis=(1, 2, 3))).max()
    out, end = {}, None
    for precision in (gb.FP64, gb.FP32):
        with gb.Lattice(N, L=L, dt=dt, precision=precision, model=gb.MODEL_LPHI4) as lat:
            lat.upload_state(f, d, a0=a, adot0=ad)
            lat.step(steps)
            out[precision] = lat.calc_energy() | {"a": lat.scalars()["a"][0], "adot": lat.scalars()["adot"][0]}
            if precision == gb.FP64:
                f1, d1 = lat.download_state(False)[:2]
                end = f1[0].mean(), d1[0].mean()
                rf, rd = max(rms(f), rms(f1)), max(rms(d), rms(d1))
    n = np.sqrt(steps / N ** 3)
    e_d = 8 * 2.0 ** -24 * (rd + dt * 12 / (L / N) ** 2 * rf) * n
    e_f = 8 * 2.0 ** -24 * rf * n + steps * dt * e_d
    tol = {"pot": 4 * e_f / abs(end[0]), "kin": 2 * e_d / abs(end[1])}
    for k in ("rho", "a", "adot"):
        tol[k] = max(tol["pot"], tol["kin"])
    for k, t in tol.items():
        assert abs(out[gb.FP32][k] / out[gb.FP64][k] - 1) <= t, (k, out[gb.FP32][k] / out[gb.FP64][k] - 1, t)
