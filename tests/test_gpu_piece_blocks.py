"""Wide beams run in pieces with outputs of their own: long batches go through in
blocks of samples, so the scratch is bounded, with the same TOD."""

import numpy as np
import pytest
import torch

from tod_generation_mapbased_beam_b200 import _native, kernels


def _case(S, B, nside=32):
    rng = np.random.default_rng(S)
    r, a = np.radians(rng.uniform(10.0, 20.0, S)), rng.uniform(0, 2 * np.pi, S)
    vec = torch.from_numpy(np.stack([np.sin(r) * np.cos(a), np.sin(r) * np.sin(a), np.cos(r)], -1)).cuda()
    bv = torch.full((S,), 1.0 / S, device="cuda")
    ang = [torch.from_numpy(rng.uniform(0.3, 2.8, B)).cuda() for _ in range(3)]
    sky = torch.from_numpy(rng.standard_normal((3, 12 * nside * nside))).cuda()

    def run(plan):
        tod = torch.ones((4, B), dtype=torch.float64, device="cuda")[:3]
        return kernels.gather_accum_angles(_native.BILINEAR, vec, *ang, 0.0, 0.0, nside, sky, bv, tod, 1, 2,
                                           pieces=plan)

    return run, kernels.piece_footprints(vec, nside)


@pytest.mark.gpu
@pytest.mark.parametrize("B", [1, 15, 16, 17, 47, 48, 49, 100])
def test_blocks_give_the_same_tod(B, monkeypatch):
    run, plan = _case(16384 + 1100, B)
    whole = run(plan)
    # three tiles a block: 18 pieces, 3 components, 8 bytes
    monkeypatch.setattr(kernels, "_PIECE_SCRATCH", 18 * 3 * 8 * 48)
    assert torch.equal(run(plan), whole)
    monkeypatch.setattr(kernels, "_PIECE_SCRATCH", 1)  # at least one tile
    assert torch.equal(run(plan), whole)


@pytest.mark.gpu
def test_scratch_is_bounded(monkeypatch):
    """98 pieces, 100,000 samples: 230 MB of outputs if they were held whole."""
    S, B = 98 * 1024, 100_000
    run, plan = _case(S, B, nside=8)
    monkeypatch.setattr(kernels, "_PIECE_SCRATCH", 1 << 26)
    torch.cuda.synchronize()
    held = torch.cuda.memory_allocated()
    torch.cuda.reset_peak_memory_stats()
    run(plan)
    torch.cuda.synchronize()
    rotations, tod, sums = 10 * 8 * B, 4 * 8 * B, 2 * 3 * 8 * B
    copies = 2 * 3 * 8 * S  # of the beam vectors
    assert torch.cuda.max_memory_allocated() - held <= (1 << 26) + rotations + tod + sums + copies + (16 << 20)
