"""Every tile of the committed cache is one that the tuner itself times, so
running it again cannot put a tile in its place that was never compared with
it; tiles that time alike are timed again in turn before one is chosen."""
import json
import os
import re

import numpy as np
import pytest

from gabe_b200 import FP32, FP64, autotune


def _lattice_entries():
    path = os.path.join(os.path.dirname(autotune.__file__), "tiles.json")
    with open(path) as fh:
        return sorted((k, e) for k, e in json.load(fh).items() if "|ens32|" not in k)


@pytest.mark.parametrize("key,entry", _lattice_entries())
def test_cached_tile_is_a_candidate(key, entry):
    N = int(re.search(r"N=(\d+)", key).group(1))
    assert (entry["shape"], entry["ci"]) in autotune.candidates(N, FP32 if "|fp32|" in key else FP64)


def test_close_tiles_are_decided_by_their_median(tmp_path, monkeypatch):
    """A stand-in lattice whose timings drift: (0, 16) is 2 % slower than (1, 8)
    but was timed first, at a higher clock; (3, 32) ties with (1, 8), whose
    place in the table decides; the rest are far off."""
    timed = []

    class Lattice:
        def __init__(self, N, *, gws, precision, tile_shape, tile_ci):
            self.tile = (tile_shape, tile_ci)

        def __enter__(self):
            return self

        def __exit__(self, *exc):
            pass

        def upload_state(self, *a, **kw):
            pass

        def profile_steps(self, n):
            if n > 1:
                timed.append(self.tile)
            base = {(0, 16): 1.02, (1, 8): 1.0, (3, 32): 0.995}.get(self.tile, 2.0)
            first = self.tile == (0, 16) and timed.count((0, 16)) <= 1
            return {"stage1": 0.6 * base * (0.95 if first else 1.0), "stage2": 0.4 * base * (0.95 if first else 1.0)}

    monkeypatch.setattr(autotune, "Lattice", Lattice)
    monkeypatch.setattr(autotune, "CACHE", str(tmp_path / "tiles.json"))
    best = autotune.tune(64, FP32, True, steps=3, verbose=False)["best"]
    assert (best["shape"], best["ci"]) == (1, 8)
    assert best["sweeps_ms"] == pytest.approx(1.0)
    assert timed.count((1, 8)) == 1 + autotune.FINAL_ROUNDS
    with open(tmp_path / "tiles.json") as fh:
        (entry,) = json.load(fh).values()
    assert entry["shape"] == 1 and entry["ci"] == 8 and np.isclose(entry["sweeps_ms"], 1.0)
