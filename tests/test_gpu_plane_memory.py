"""The plane transform works in place: with GABE_FLAG_NO_OVERLAP a handle that
takes it has one source buffer and no more device memory than cuFFT's in-line
form, with the same results."""
import numpy as np
import pytest

import gabe_b200 as gb
from gabe_b200.ic import random_state

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N", [16, 32, 48, 96, 128])
def test_source_buffers(N):
    f, d, a0, ad0 = random_state(N, seed=N)
    forms = {"plane": 0, "plane, no overlap": gb.FLAG_NO_OVERLAP, "cufft": gb.FLAG_CUFFT_3D,
             "cufft, no overlap": gb.FLAG_CUFFT_3D | gb.FLAG_NO_OVERLAP}
    size, out = {}, {}
    for name, flags in forms.items():
        with gb.Lattice(N, gws=True, precision=gb.FP32, flags=flags, dt=2e-3) as lat:
            assert lat.launches_per_step == (5 if name.startswith("plane") else 3)
            size[name] = lat.device_bytes
            lat.upload_state(f.numpy(), d.numpy(), a0=a0, adot0=ad0)
            lat.step(5)
            out[name] = lat.download_state()
    buffer = 10 * N * N * (N + 2) * 4
    assert size["cufft"] - size["cufft, no overlap"] == buffer
    assert size["plane, no overlap"] <= size["cufft, no overlap"]
    # below 128^3 the GW chain overlaps the sweeps, as cuFFT's does
    assert size["plane"] - size["plane, no overlap"] == (buffer if N < 128 else 0)
    for x, y in zip(out["plane"], out["plane, no overlap"]):
        np.testing.assert_array_equal(x, y)
