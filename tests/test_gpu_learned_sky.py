"""A sky refilled in place: the float64 forms of LearnedTailTOD read the caller's
tensor in every call."""

from types import SimpleNamespace

import numpy as np
import pytest
import torch

from tod_generation_mapbased_beam_b200 import workloads as W
from tod_generation_mapbased_beam_b200.learned import LearnedTailTOD
from tod_generation_mapbased_beam_b200.sky import alm2map, cl_tt, random_alm


def _beam(S, lo_deg, hi_deg, seed):
    rng = np.random.default_rng(seed)
    r, a = np.radians(rng.uniform(lo_deg, hi_deg, S)), rng.uniform(0, 2 * np.pi, S)
    v = np.stack([np.sin(r) * np.cos(a), np.sin(r) * np.sin(a), np.cos(r)], -1)
    return SimpleNamespace(vec_orig=v, beam_vals=np.full(S, 1.0 / S, np.float32))


@pytest.mark.gpu
@pytest.mark.parametrize("S", [700, 16384 + 700])
@pytest.mark.parametrize("refill", ["copy", "alm2map"])
def test_refilled_sky_is_read(S, refill):
    nside = 32
    main, tail = _beam(300, 0.0, 2.0, 1), _beam(S, 5.0, 9.0, 2)
    scan = [torch.from_numpy(a).cuda() for a in W.spin_scan(25, 0.5)]
    sky = torch.from_numpy(W.white_sky(nside, 3)).cuda()
    lt = LearnedTailTOD(nside, sky, main, tail, main_map="f64")
    forms = (lt.plain_tail, lambda *a: lt.main_lobe(*a, exact=True), lt.main_lobe, lt.full_plain)
    before = [f(*scan) for f in forms]
    if refill == "copy":
        sky.copy_(torch.from_numpy(W.white_sky(nside, 4)))
    else:
        for c in range(3):
            alm2map(random_alm(cl_tt(48), 5 + c), nside, 48, sky, c)
    fresh = LearnedTailTOD(nside, sky, main, tail, main_map="f64")
    for f, g, old in zip(forms, (fresh.plain_tail, lambda *a: fresh.main_lobe(*a, exact=True), fresh.main_lobe,
                                 fresh.full_plain), before):
        assert torch.equal(f(*scan), g(*scan))
        assert not torch.equal(f(*scan), old)
