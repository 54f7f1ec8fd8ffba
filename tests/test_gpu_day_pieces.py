"""The day loop over a beam wide enough to run in pieces: its footprints are found
when the runner is made, so no chunk waits for the GPU."""

import numpy as np
import pytest

from tod_generation_mapbased_beam_b200 import driver, kernels
from tod_generation_mapbased_beam_b200 import workloads as W


@pytest.mark.gpu
@pytest.mark.parametrize("comps", [[0, 1, 2], [2, 0, 1]])  # rows in place; through a buffer
def test_footprints_are_found_once(comps, monkeypatch):
    nside, S = 32, 16384 + 900
    rng = np.random.default_rng(1)
    r, a = np.radians(rng.uniform(5.0, 9.0, S)), rng.uniform(0, 2 * np.pi, S)
    vec = np.stack([np.sin(r) * np.cos(a), np.sin(r) * np.sin(a), np.cos(r)], -1).astype(np.float32)
    data = {"wide": dict(vec_orig=vec, beam_vals=np.full(S, 1.0 / S, np.float32), comp_indices=comps,
                         mp_stacked=np.ascontiguousarray(W.white_sky(nside, 2)[comps]), ra=np.zeros((1, 1)),
                         dec=np.full((1, 1), np.pi / 2))}
    scan = W.spin_scan(100, 1.0)
    whole = driver.DayRunner(data, nside).run(*scan)
    runner = driver.DayRunner(data, nside, chunk=32)

    def found_again(*args):
        raise AssertionError("piece_footprints called for a chunk")

    monkeypatch.setattr(kernels, "piece_footprints", found_again)
    assert np.array_equal(runner.run(*scan), whole) and np.abs(whole).max() > 0
