"""Which beam tensors a gather reads where they are: (S, 3) ones of the parameters'
type on the GPU the call runs on.  Everything else is moved, converted and
reshaped first, or refused."""

import numpy as np
import pytest
import torch

from tod_generation_mapbased_beam_b200 import _native
from tod_generation_mapbased_beam_b200.kernels import gather_accum, gather_accum_angles, resident_beam

CPU, OTHER = torch.device("cpu"), torch.device("meta")


def test_resident_beam_needs_device_type_and_shape():
    v = torch.zeros((4, 3), dtype=torch.float64)
    assert resident_beam(v, np.float64, CPU) is v
    planar = torch.zeros((3, 4), dtype=torch.float64).t()
    assert resident_beam(planar, np.float64, CPU) is planar
    assert resident_beam(torch.empty((4, 3), dtype=torch.float64, device=OTHER), np.float64, CPU) is None
    assert resident_beam(v, np.float32, CPU) is None
    for shape in ((4, 2), (3, 4), (2, 6), (12,), (2, 2, 3)):
        assert resident_beam(torch.zeros(shape, dtype=torch.float64), np.float64, CPU) is None
    assert resident_beam(v.numpy(), np.float64, CPU) is None


@pytest.mark.gpu
def test_beam_shapes():
    """Vectors in another shape of the same values give the same TOD; a tensor that
    does not hold three components a pixel is refused before any launch."""
    nside, S, B = 32, 90, 5
    rng = np.random.default_rng(1)
    v = rng.normal(size=(S, 3)) * 0.02 + [0, 0, 1]
    v = torch.from_numpy(v / np.linalg.norm(v, axis=1, keepdims=True)).cuda()
    bv = torch.full((S,), 1.0 / S, device="cuda")
    sky = torch.from_numpy(rng.normal(size=(3, 12 * nside * nside))).cuda()
    ang = [torch.from_numpy(rng.uniform(0.5, 2.5, B)).cuda() for _ in range(3)]

    def angles(vec):
        tod = torch.zeros((3, B), dtype=torch.float64, device="cuda")
        return gather_accum_angles(_native.BILINEAR, vec, *ang, 0.0, 0.0, nside, sky, bv, tod, 1, 2)

    ref = angles(v)
    for same in (v.reshape(S // 3, 9), v.reshape(-1), v.t().contiguous().t(), v.cpu()):
        assert torch.equal(angles(same), ref)
    for bad in (v[:, :2].contiguous(), v[:, :2], v[: S - 1]):
        with pytest.raises((RuntimeError, ValueError)):
            angles(bad)
    one = [torch.ones(B, dtype=torch.float64, device="cuda") for _ in range(4)]
    tri = [torch.ones((B, 3), dtype=torch.float64, device="cuda") for _ in range(2)]
    for bad in (v[:, :2].contiguous(), v[: S - 1]):
        with pytest.raises((RuntimeError, ValueError)):
            gather_accum(_native.BILINEAR, bad, tri[0], one[0], one[1], tri[1], one[2], one[3], nside, sky, bv, B, S,
                         torch.zeros((3, B), dtype=torch.float64, device="cuda"), 1, 2)
