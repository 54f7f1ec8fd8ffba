"""The host fingerprint and changes that cancel in a simpler one: pairs of flipped
bits in words one lane, one block or one pair apart."""

import numpy as np
import pytest

from tod_generation_mapbased_beam_b200 import _native


def _hash(a):
    return _native.lib().todgpu_host_hash(a.ctypes.data, a.nbytes, 0)


@pytest.mark.parametrize("kind", ["random", "zeros", "ones", "floats"])
@pytest.mark.parametrize("apart", [1, 2, 8, 64])
def test_flipped_bit_pairs(kind, apart):
    n = 192
    rng = np.random.default_rng(apart)
    a = {"random": rng.integers(0, 1 << 63, n, dtype=np.uint64), "zeros": np.zeros(n, np.uint64),
         "ones": np.full(n, np.uint64(2**64 - 1)), "floats": rng.standard_normal(n).view(np.uint64)}[kind]
    base = _hash(a)
    for j in (3, 62):
        for hi in range(64):
            seen = set()
            for lo in range(64):
                b = a.copy()
                b[j] ^= np.uint64(1 << hi)
                b[j + apart] ^= np.uint64(1 << lo)
                seen.add(_hash(b))
            assert len(seen) == 64 and base not in seen


def test_the_pair_that_cancelled():
    a = np.random.default_rng(0).integers(0, 1 << 63, 64, dtype=np.uint64)
    b = a.copy()
    b[3] ^= np.uint64(1 << 63)
    b[11] ^= np.uint64(1 << 26)
    assert _hash(b) != _hash(a)


def test_blocks_in_another_order():
    a = np.random.default_rng(2).standard_normal((6, 64))
    seen = {_hash(a), _hash(a[::-1].copy()), _hash(a[[1, 0, 2, 3, 4, 5]].copy()), _hash(a[[0, 1, 2, 3, 5, 4]].copy()),
            _hash(np.repeat(a[:1], 6, 0)), _hash(np.repeat(a[:1], 5, 0))}
    assert len(seen) == 6
