"""Float64 records of a planar map: every component count, ragged and strided maps."""

import pytest
import torch

from tod_generation_mapbased_beam_b200.kernels import pack_map


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("C", [1, 2, 3, 4])
@pytest.mark.parametrize("N", [1, 12, 127, 129, 12 * 37 * 37, 5_000_001])
def test_records(C, N, dtype):
    m = torch.randn((C, N + 3), dtype=dtype, device="cuda")[:, :N]
    got = pack_map(m, "f64").data
    want = torch.zeros((N, 4), dtype=torch.float64, device="cuda")
    want[:, :C] = m.t().double()
    assert torch.equal(got, want)
