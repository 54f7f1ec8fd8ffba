"""The plain tail over records made in the call: the planar map's TOD bit for bit, and
the sky as it is at each call."""

from types import SimpleNamespace

import numpy as np
import pytest
import torch

from tod_generation_mapbased_beam_b200 import learned
from tod_generation_mapbased_beam_b200 import workloads as W


@pytest.mark.gpu
@pytest.mark.parametrize("S", [900, 16384 + 900])
def test_records_follow_the_sky(S, monkeypatch):
    rng = np.random.default_rng(1)
    r, a = np.radians(rng.uniform(5.0, 9.0, S)), rng.uniform(0, 2 * np.pi, S)
    beam = SimpleNamespace(vec_orig=np.stack([np.sin(r) * np.cos(a), np.sin(r) * np.sin(a), np.cos(r)], -1),
                           beam_vals=np.full(S, 1.0 / S, np.float32))
    scan = [torch.from_numpy(x).cuda() for x in W.spin_scan(30, 0.5)]
    sky = torch.from_numpy(W.white_sky(256, 3)).cuda()
    lt = learned.LearnedTailTOD(256, sky, beam, beam)

    def both():
        out = []
        for least in (30 * S, 30 * S + 1):
            monkeypatch.setattr(learned, "_RECORD_EVALS", least)
            assert (lt._tail_sky(30) is sky) == (least > 30 * S)
            out.append(lt.plain_tail(*scan))
        assert torch.equal(*out)
        return out[0]

    before = both()
    sky.copy_(torch.from_numpy(W.white_sky(256, 4)))
    assert not torch.equal(both(), before)
