"""A kept piece plan belongs to one beam size and nside: another beam's would leave
out pixels without a word, or run into jobs of no pixels after others were added."""

import numpy as np
import pytest
import torch

from tod_generation_mapbased_beam_b200 import _native
from tod_generation_mapbased_beam_b200.kernels import _check_plan, gather_accum_angles, piece_footprints


def _disc(S, seed=1):
    rng = np.random.default_rng(seed)
    r, a = np.radians(9.0) * np.sqrt(rng.uniform(0, 1, S)), rng.uniform(0, 2 * np.pi, S)
    return torch.from_numpy(np.stack([np.sin(r) * np.cos(a), np.sin(r) * np.sin(a), np.cos(r)], -1))


@pytest.mark.parametrize("S", [16385, 17408, 17409, 40000])
def test_plan_is_checked(S):
    plan = piece_footprints(_disc(S), 64)
    assert len(plan.slots) == -(-S // 1024) and _check_plan(plan, S, 64) is plan
    for s, nside in ((S - 1, 64), (S + 1, 64), (S - 1024, 64), (S + 1024, 64), (S, 128)):
        with pytest.raises(ValueError):
            _check_plan(plan, s, nside)
    for other in (tuple(plan), (plan.slots, plan.reach), plan._replace(slots=plan.slots[:-1])):
        with pytest.raises(ValueError):
            _check_plan(other, S, 64)


@pytest.mark.gpu
@pytest.mark.parametrize("other", [16385, 20000])
def test_gather_refuses_another_beams_plan(other):
    nside, S, B = 64, 18000, 4
    vec = _disc(S).cuda()
    sky = torch.from_numpy(np.random.default_rng(2).standard_normal((3, 12 * nside * nside))).cuda()
    bv = torch.full((S,), 1.0 / S, device="cuda")
    ang = [torch.from_numpy(np.random.default_rng(3).uniform(0.5, 2.5, B)).cuda() for _ in range(3)]
    tod = torch.zeros((3, B), dtype=torch.float64, device="cuda")
    with pytest.raises(ValueError):
        gather_accum_angles(_native.BILINEAR, vec, *ang, 0.0, 0.0, nside, sky, bv, tod, 1, 2,
                            pieces=piece_footprints(_disc(other).cuda(), nside))
    assert not tod.any()
    gather_accum_angles(_native.BILINEAR, vec, *ang, 0.0, 0.0, nside, sky, bv, tod, 1, 2,
                        pieces=piece_footprints(vec, nside))
    again = torch.zeros_like(tod)
    gather_accum_angles(_native.BILINEAR, vec, *ang, 0.0, 0.0, nside, sky, bv, again, 1, 2)
    assert tod.any() and torch.equal(tod, again)
