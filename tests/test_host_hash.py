"""The host fingerprint behind the drop-in's upload checks: any change of a word,
a tail byte, an order or a length changes it, and it depends on nothing else."""

import numpy as np
import pytest

from tod_generation_mapbased_beam_b200 import _native


def _hash(a, seed=0):
    return _native.lib().todgpu_host_hash(a.ctypes.data, a.nbytes, seed)


@pytest.mark.parametrize("n", [0, 1, 7, 8, 9, 63, 64, 65, 127, 128, 200, 4096 + 5])
def test_every_byte_counts(n):
    rng = np.random.default_rng(n)
    a = rng.integers(0, 256, n, dtype=np.uint8)
    base = _hash(a)
    assert _hash(a.copy()) == base
    seen = {base}
    for i in range(0, n, max(1, n // 97)):
        for bit in (0, 7):
            b = a.copy()
            b[i] ^= 1 << bit
            seen.add(_hash(b))
    assert len(seen) == 1 + 2 * len(range(0, n, max(1, n // 97)))
    if n > 1:
        assert _hash(a[:-1].copy()) != base
        assert _hash(np.concatenate([a, [0]]).astype(np.uint8)) != base
    assert n == 0 or _hash(a, 1) != base


def test_sign_flips_and_exchanges():
    """Two changes that cancel in a sum or product: signs of several values of one
    lane (every eighth word), and exchanged values."""
    a = np.random.default_rng(1).standard_normal(512)
    base = _hash(a)
    for idx in ([0, 8], [3, 11, 19, 27], slice(None), slice(0, None, 8)):
        b = a.copy()
        b[idx] *= -1
        assert _hash(b) != base
    for i, j in ((0, 8), (0, 1), (5, 509)):
        b = a.copy()
        b[[i, j]] = b[[j, i]]
        assert _hash(b) != base
