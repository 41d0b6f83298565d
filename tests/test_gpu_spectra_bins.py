"""The binning kernel against numpy: counts exactly, power sums to the rounding
of the transform, at sizes whose lines end inside a warp's 32 points, with the
amplitudes in both storage orders and both readings of the kz = 0 plane."""
import numpy as np
import pytest

import gabe_b200 as gb
from gabe_b200.ic import random_state

pytestmark = pytest.mark.gpu

CASES = [(4, gb.FP64, 0), (20, gb.FP64, 0), (48, gb.FP64, 0), (16, gb.FP32, 0), (48, gb.FP32, 0),
         (64, gb.FP32, gb.FLAG_TRANSPOSED_FFT), (128, gb.FP32, 0)]


@pytest.mark.parametrize("quirk", [True, False])
@pytest.mark.parametrize("N,precision,flags", CASES)
def test_bins_match_numpy(N, precision, flags, quirk):
    f0, d0, a0, ad0 = random_state(N, seed=N)
    with gb.Lattice(N, gws=True, precision=precision, flags=flags, dt=1e-3, gw_spec_quirk=quirk) as lat:
        lat.upload_state(f0.numpy(), d0.numpy(), a0=a0, adot0=ad0)
        lat.step(3)
        sums, counts = lat.spectra_raw()
        f, _, _, ell = lat.download_state()
    nb, nz = gb.numbins(N), N // 2 + 1
    i = np.fft.fftfreq(N, 1.0 / N)
    n2 = i[:, None, None] ** 2 + i[None, :, None] ** 2 + np.arange(nz)[None, None, :] ** 2
    b = np.sqrt(np.rint(n2)).astype(int).ravel()
    w = np.full(nz, 2.0)
    w[0] = w[-1] = 1.0
    w = np.broadcast_to(w, n2.shape).ravel()
    np.testing.assert_array_equal(counts, np.bincount(b, w, nb))
    eps = 2.0 ** -24 if precision == gb.FP32 else 2.0 ** -53
    for x in range(2):
        p = np.abs(np.fft.rfftn(f[x])).ravel() ** 2
        ref = np.bincount(b, w * p, nb)
        # each coefficient carries a few eps of the field's 2-norm (FP32 storage transforms the fluctuations)
        e = 10 * eps * np.linalg.norm(f[x] - (f[x].mean() if precision == gb.FP32 else 0))
        e += 10 * 2.0 ** -53 * np.linalg.norm(f[x])
        tol = 2 * np.sqrt(ref * counts) * e + counts * e * e
        assert np.all(np.abs(sums[x] - ref) <= tol + 1e-14 * ref), (x, np.max(np.abs(sums[x] - ref) / (tol + 1e-300)))
    m = np.array([1, 2, 2, 1, 2, 1.0])
    p = sum(m[c] * (ell[2 * c] ** 2 + ell[2 * c + 1] ** 2) for c in range(6))
    if quirk:
        p[..., 0] = p[..., -1]
    ref = np.bincount(b, w * p.ravel(), nb)
    assert ref.max() > 0
    # the 12 components are formed from the amplitudes in FP64: only the sums' rounding differs
    np.testing.assert_allclose(sums[2], ref, rtol=1e-11, atol=1e-25 * ref.max())
