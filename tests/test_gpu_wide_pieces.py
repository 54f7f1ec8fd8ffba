"""Pieces of a wide beam whose footprints are too large for a table: windows without
one, the direct evaluation's TOD bit for bit."""

import numpy as np
import pytest
import torch

from tod_generation_mapbased_beam_b200 import _native, kernels
from tod_generation_mapbased_beam_b200.kernels import (_PIECE_NO_TABLE, _PIECE_SLOTS, gather_accum_angles, patch_order,
                                                       piece_footprints)


def _beam(S, lo, hi, patches, seed=1):
    rng = np.random.default_rng(seed)
    r, a = np.radians(rng.uniform(lo, hi, S)), rng.uniform(0, 2 * np.pi, S)
    v = np.stack([np.sin(r) * np.cos(a), np.sin(r) * np.sin(a), np.cos(r)], -1)
    return v[patch_order(v)] if patches else v


def test_requests():
    S = 16384 + 700
    tabled = piece_footprints(torch.from_numpy(_beam(S, 3.0, 5.0, True)), 256)
    assert tabled.slots.max() <= _PIECE_SLOTS and tabled.slots.min() > 2
    wide = piece_footprints(torch.from_numpy(_beam(S, 3.0, 20.0, True)), 1024)
    assert wide.slots.min() >= _PIECE_NO_TABLE and wide.reach == 0.0 and wide.window_reach > 0.03
    # in no order every piece is the whole beam: beyond any window at this nside
    none = piece_footprints(torch.from_numpy(_beam(S, 3.0, 40.0, False)), 2048)
    assert np.all(none.slots == 2) and none.window_reach == 0.0


@pytest.mark.gpu
@pytest.mark.parametrize("mode", [_native.BILINEAR, _native.NEAREST])
@pytest.mark.parametrize("C, c_q, c_u", [(1, -1, -1), (3, 1, 2)])
@pytest.mark.parametrize("nside, lo, hi, patches", [(1024, 3.0, 20.0, True), (512, 0.0, 12.0, False),
                                                    (2048, 3.0, 40.0, False), (32, 60.0, 120.0, True)])
@pytest.mark.parametrize("own", [True, False])
def test_wide_pieces_match_direct(nside, lo, hi, patches, C, c_q, c_u, mode, own, monkeypatch):
    S, B = 16384 + 700, 20
    if own:  # a launch of their own takes thousands of samples otherwise
        monkeypatch.setattr(kernels, "_PIECE_OWN_LAUNCH", 1)
    vec = torch.from_numpy(_beam(S, lo, hi, patches)).cuda()
    rng = np.random.default_rng(2)
    bv = torch.from_numpy(rng.uniform(0, 1e-4, S).astype(np.float32)).cuda()
    ang = [torch.from_numpy(x).cuda() for x in (np.arccos(rng.uniform(-1, 1, B)), rng.uniform(0, 6.28, B),
                                                 rng.uniform(0, 6.28, B))]
    g = torch.Generator("cuda").manual_seed(3)
    sky = torch.randn((C, 12 * nside * nside), generator=g, device="cuda", dtype=torch.float64)
    outs = []
    for flags in (0, _native.FLAG_NO_TABLES):
        tod = torch.zeros((C, B), dtype=torch.float64, device="cuda")
        gather_accum_angles(mode, vec, *ang, 0.0, 0.0, nside, sky, bv, tod, c_q, c_u, flags=flags)
        outs.append(tod)
    assert torch.equal(*outs) and outs[0].abs().max() > 0
