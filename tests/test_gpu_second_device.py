"""A second GPU in the same process: kernels that ask for more than 48 KB of dynamic
shared memory ask on every device they run on."""

import numpy as np
import pytest
import torch

from tod_generation_mapbased_beam_b200 import _native
from tod_generation_mapbased_beam_b200.beam_cluster import _GpuKMeans
from tod_generation_mapbased_beam_b200.kernels import gather_accum_angles


@pytest.mark.gpu
def test_second_device_gives_the_first_ones_results():
    if torch.cuda.device_count() < 2:
        pytest.skip("needs two GPUs")
    rng = np.random.default_rng(1)
    v = rng.standard_normal((9000, 3)) * 0.1 + [0, 0, 1]  # 72 KB of probabilities
    v /= np.linalg.norm(v, axis=1, keepdims=True)
    w, u = rng.uniform(0.1, 1.0, 9000), rng.uniform(0, 1, 12)
    sky = rng.standard_normal((3, 12 * 512 * 512))
    ang = [rng.uniform(0.5, 2.5, 40) for _ in range(3)]
    got = []
    for dev in (0, 1):
        with torch.cuda.device(dev):
            cent = _GpuKMeans(v, w, 12).seed(u)
            tod = torch.zeros((3, 40), dtype=torch.float64, device="cuda")
            gather_accum_angles(_native.BILINEAR, v, *ang, 0.0, 0.0, 512, sky, w.astype(np.float32), tod, 1, 2)
            got.append((cent, tod.cpu().numpy()))
    for a, b in zip(*got):
        assert np.array_equal(a, b) and np.abs(a).max() > 0
