"""The k-means kernels about the sizes where their paths change: one-CTA seeding
(to 12288 pixels) and the two-launch form, one or eight lanes a pixel in the
assignment (65536 pixels), cluster sums from the labels (S K to 2^23) and from the
sorted pixels.  Oracle: numpy in float64 -- draws by cumulative sums, argmax, and
bincount, whose sequential sums the kernels reproduce bit for bit.  (A draw could
differ only where a uniform meets a cumulative share to its last bits, ~1e-13.)"""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _points(S, seed):
    rng = np.random.default_rng(seed)
    v = rng.standard_normal((S, 3)) * [0.02, 0.02, 0.0] + [0, 0, 1]
    v /= np.linalg.norm(v, axis=1, keepdims=True)
    w = rng.uniform(0.1, 1.0, S)
    return v, w / w.sum(), rng


@pytest.mark.parametrize("S, K", [(1, 1), (31, 5), (33, 33), (1023, 40), (1025, 200), (5414, 200), (12288, 30),
                                  (12289, 30), (70001, 9), (50000, 170)])
def test_paths_match_numpy(S, K):
    from tod_generation_mapbased_beam_b200.beam_cluster import _GpuKMeans

    v, w, rng = _points(S, S + K)
    km = _GpuKMeans(v, w, K)
    u = rng.random(K)
    cent = km.seed(u)
    near = None
    for k in range(K):
        p = w if k == 0 else w * np.maximum(1.0 - near, 0.0) ** 2
        p = w if p.sum() == 0 else p
        c = np.cumsum(p)
        pick = min(S - 1, int(np.argmax(c / c[-1] > u[k])))
        assert np.array_equal(cent[k], v[pick]), k
        s = v @ cent[k]
        near = s if near is None else np.maximum(near, s)
        if k == 40:  # the rest are drawn the same way
            break
    km.assign(cent)
    lab = km.labels.cpu().numpy()
    sim = v @ cent.T
    # the chosen centroid is the best to the last bits, and the first among equals
    assert np.all(sim[np.arange(S), lab] >= sim.max(axis=1) - 4e-16)
    exact = np.sort(sim, axis=1)[:, -2:] if K > 1 else None
    clear = np.ones(S, bool) if K == 1 else exact[:, 1] - exact[:, 0] > 4e-16
    assert np.array_equal(lab[clear], np.argmax(sim, axis=1)[clear])
    sums = km.cluster_sums()
    for c in range(3):
        assert np.array_equal(sums[:, c], np.bincount(lab, w * v[:, c], minlength=K))
    assert np.array_equal(sums[:, 3], np.bincount(lab, w, minlength=K))


def test_equal_similarities_keep_the_first_centroid():
    from tod_generation_mapbased_beam_b200.beam_cluster import _GpuKMeans

    v, w, _ = _points(300, 3)
    km = _GpuKMeans(v, w, 11)
    c = np.repeat(v[:1], 11, axis=0)
    c[:3] = v[1:2]
    c[3:] = v[1:2]
    km.assign(c)
    assert not km.labels.cpu().numpy().any()
