"""The plane transform (fftp.cuh) against cuFFT's 3-D plan with the separate
k-space pass, at every size it takes, and its amplitude order in restart
files and ensembles."""
import numpy as np
import pytest

import gabe_b200 as gb
from gabe_b200.ic import random_state

pytestmark = pytest.mark.gpu

FFT_TOL = 1e-5  # relative norm, FP32 transforms
SIZES = [16, 32, 48, 80, 96, 112, 128, 144, 160]


def _rel(a, b):
    return float(np.linalg.norm(a - b) / np.linalg.norm(b))


def _lattice(N, flags, dt=2e-3):
    f, d, a0, ad0 = random_state(N, seed=N)
    lat = gb.Lattice(N, gws=True, precision=gb.FP32, flags=flags, dt=dt)
    lat.upload_state(f.numpy(), d.numpy(), a0=a0, adot0=ad0)
    return lat


@pytest.mark.parametrize("N", SIZES)
def test_plane_transform_matches_cufft_3d(N):
    out = {}
    for name, flags in (("plane", 0), ("cufft", gb.FLAG_CUFFT_3D)):
        with _lattice(N, flags) as lat:
            assert lat.launches_per_step == (5 if name == "plane" else 3)
            lat.step(3)
            out[name] = (*lat.download_state(), lat.spec_out())
    (f0, d0, h0, l0, s0), (f1, d1, h1, l1, s1) = out["plane"], out["cufft"]
    np.testing.assert_array_equal(f0, f1)  # the fields do not depend on the GW chain
    np.testing.assert_array_equal(d0, d1)
    assert np.linalg.norm(l1) > 0
    assert _rel(h0, h1) <= FFT_TOL and _rel(l0, l1) <= FFT_TOL
    # every Fourier mode, not only the loud ones: the error of a mode scales with the array's rms
    assert np.abs(l0 - l1).max() <= 1e-4 * np.abs(l1).max()
    np.testing.assert_allclose(s0[1:, 5:7], s1[1:, 5:7], rtol=1e-4, atol=1e-9 * s1[:, 5].max())


@pytest.mark.parametrize("N", [48, 128])
def test_restart_file_of_another_amplitude_order(N, tmp_path):
    """A file written by cuFFT's form restarts a plane-transform handle, and
    the other way round: the amplitudes are reordered, not lost."""
    path = str(tmp_path / "state.bin")
    for src, dst in ((gb.FLAG_CUFFT_3D, 0), (0, gb.FLAG_CUFFT_3D)):
        with _lattice(N, src) as lat:
            lat.step(3)
            lat.save(path)
            want = lat.download_state()
        with gb.Lattice(N, gws=True, precision=gb.FP32, flags=dst, dt=2e-3) as lat:
            assert lat.load(path)
            got = lat.download_state()
        for a, b in zip(got, want):
            np.testing.assert_array_equal(a, b)


def test_ensemble_sizes_with_and_without_the_plane_transform():
    """Every lattice of a mixed ensemble (176 has no plane transform) carries
    the amplitudes of a single lattice holding its state."""
    N = [16, 48, 176, 32, 48, 96, 144, 48]
    g = [1.0, 50.0, 100.0, 300.0, 5.0, 100.0, 20.0, 400.0]
    with gb.Ensemble(N, g, [1.0] * len(N), range(1, len(N) + 1), dt=2e-3) as ens:
        ens.init()
        start = [ens.download(q) for q in range(len(N))]
        adot = ens.scalars()[:, 2]
        ens.step(4)
        for q, n in enumerate(N):
            f, d, _, _ = start[q]
            with gb.Lattice(n, gws=True, precision=gb.FP32, dt=2e-3, flags=gb.FLAG_CUFFT_3D,
                            model_c=gb.lphi4_constants(g[q])) as lat:
                lat.upload_state(f, d, a0=1.0, adot0=adot[q])
                lat.step(4)
                want = lat.download_state()
            got = ens.download(q)
            for x in (2, 3):
                assert np.linalg.norm(want[x]) > 0
                # the single lattice takes its means from the fluctuating state: 1e-5 of the fluctuation, as its fields
                assert _rel(got[x], want[x]) <= 3e-5, (q, n, x)
