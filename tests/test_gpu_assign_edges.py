"""The assignment on both sides of its rule for lanes per pixel (16384 pixels) and of
a tile of centroids (2048): the first best centroid, for either form the same."""

import numpy as np
import pytest


@pytest.mark.gpu
@pytest.mark.parametrize("K", [1, 7, 2047, 2049])
@pytest.mark.parametrize("S", [16383, 16384, 16385])
def test_assignment(S, K):
    from tod_generation_mapbased_beam_b200.beam_cluster import _GpuKMeans

    rng = np.random.default_rng(S + K)
    v, c = rng.integers(-3, 4, (S, 3)).astype(float), rng.integers(-3, 4, (K, 3)).astype(float)
    km = _GpuKMeans(v, np.ones(S), K)
    km.assign(c)  # small whole numbers: exact products and many equal ones
    sim = v @ c.T
    assert np.array_equal(km.labels.cpu().numpy(), sim.argmax(axis=1))
    assert np.array_equal(km.best.cpu().numpy(), sim.max(axis=1))
