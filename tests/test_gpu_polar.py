"""GPU test of the gather at the poles, where the ring weights amplify the
rounding of a query's z by nside / sin theta: random pole-crossing cases with
the reference's float32 parameters agree with the oracle as cases elsewhere do,
with and without footprint tables."""

import numpy as np
import pytest
import torch

import oracle
from test_gpu_parity import TOD_RTOL, _random_case, _rel
from tod_generation_mapbased_beam_b200 import _native

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,S,nside,radius,pole,seeds", [
    (256, 300, 64, 1.0, True, (0, 32, 61, 87, 92, 127)), (64, 400, 256, 8.0, False, (10, 21, 42, 65, 110, 125)),
    (128, 257, 256, 0.5, True, (1, 2, 3))])
def test_pole_crossing_cases_match_oracle(B, S, nside, radius, pole, seeds):
    from tod_generation_mapbased_beam_b200.kernels import gather_accum

    for seed in seeds:
        params, mp, bv = _random_case(B, S, nside, seed=seed, beam_radius_deg=radius, pole=pole)
        cpu = np.zeros((3, B))
        oracle.gather_accum_fused(*params, nside, mp, bv, B, S, cpu, 1, 2)
        outs = []
        for flags in (0, _native.FLAG_NO_TABLES, _native.FLAG_WIDE_CTAS):
            tod = torch.zeros((3, B), dtype=torch.float64, device="cuda")
            gather_accum(_native.BILINEAR, *params, nside, mp, bv, B, S, tod, 1, 2, flags=flags)
            outs.append(tod.cpu().numpy())
        assert _rel(outs[0], cpu, 0.0) <= TOD_RTOL, seed
        np.testing.assert_array_equal(outs[0], outs[1])
        np.testing.assert_array_equal(outs[0], outs[2])
