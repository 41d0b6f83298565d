"""Ensembles with several batches of one size through the plane transform (48
MB of sources each: one lattice of 96^3 or 128^3, four of 64^3, 34 of 32^3),
with remainders, sizes interleaved and every coupling another: each lattice's
amplitudes are those of a single lattice with cuFFT's form, and replayed graphs
equal direct launches bit for bit."""
import numpy as np
import pytest

import gabe_b200 as gb

pytestmark = pytest.mark.gpu

SIZES = [96, 64, 128, 64, 96, 64, 32, 64, 128, 64, 96] + [32] * 36
COUPLINGS = [1.0 + 7.0 * q for q in range(len(SIZES))]


def _run(flags):
    n = len(SIZES)
    with gb.Ensemble(SIZES, COUPLINGS, [1.0] * n, range(1, n + 1), dt=2e-3, flags=flags) as ens:
        ens.init()
        adot = ens.scalars()[:, 2]
        start = [ens.download(q)[:2] for q in range(n)]
        ens.step(4)
        assert ens.graph_active == (0 if flags else 1)
        return adot, start, [ens.download(q) for q in range(n)], ens.launches_per_step


def test_every_lattice_of_every_batch():
    adot, start, got, launches = _run(0)
    batches = 3 + 2 + 2 + 2  # 96: 3 x 1; 64: 4 + 1; 128: 2 x 1; 32: 34 + 3
    assert launches == 2 + 2 * batches
    for q, n in enumerate(SIZES):
        f, d = start[q]
        with gb.Lattice(n, gws=True, precision=gb.FP32, dt=2e-3, flags=gb.FLAG_CUFFT_3D,
                        model_c=gb.lphi4_constants(COUPLINGS[q])) as lat:
            lat.upload_state(f, d, a0=1.0, adot0=adot[q])
            lat.step(4)
            want = lat.download_state()
        for x in (2, 3):
            assert np.linalg.norm(want[x]) > 0
            # the single lattice takes its means from the fluctuating state: 1e-5 of the fluctuation, as its fields
            assert np.linalg.norm(got[q][x] - want[x]) <= 3e-5 * np.linalg.norm(want[x]), (q, n, x)
    for q, direct in enumerate(_run(gb.FLAG_NO_GRAPH)[2]):
        for x in range(4):
            np.testing.assert_array_equal(got[q][x], direct[x], err_msg=str((q, x)))
