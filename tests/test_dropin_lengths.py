"""The drop-in's host pointing has one entry per sample: arrays of other lengths are
refused, never cut or repeated."""

import numpy as np
import pytest
import torch

from tod_generation_mapbased_beam_b200 import tod_core
from tod_generation_mapbased_beam_b200 import tod_rotations as R
from tod_generation_mapbased_beam_b200.kernels import boresight_phi_host


def _inputs(B):
    rng = np.random.default_rng(B)
    return rng.normal(0, 0.3, (B, 3)), rng.uniform(0, 6, B), rng.uniform(0.5, 2.5, B), rng.uniform(0, 6, B)


def test_packed_parameters_are_the_fields():
    B = 7
    params = R._rotation_params(*_inputs(B))
    buf = tod_core._pack_params(params, B, True)
    for got, want in zip(tod_core._param_views(torch.from_numpy(buf), B), params):
        assert np.array_equal(got.numpy(), want)
    assert np.array_equal(buf[-B:], boresight_phi_host(params[3]))
    for i in range(6):
        short = list(params)
        short[i] = params[i][:1]
        with pytest.raises(ValueError):
            tod_core._pack_params(short, B, True)


@pytest.mark.gpu
def test_dropin_refuses_other_lengths():
    nside, B = 16, 6
    rng = np.random.default_rng(0)
    v = rng.normal(size=(20, 3)) * 0.02 + [0, 0, 1]
    v = (v / np.linalg.norm(v, axis=1, keepdims=True)).astype(np.float32)
    data = dict(vec_orig=v, beam_vals=np.full(20, 0.05, np.float32), comp_indices=[0, 1, 2],
                mp_stacked=rng.normal(size=(3, 12 * nside * nside)))
    rot, ph, th, ps = _inputs(B)

    def call(rot, ph, th, ps):
        return tod_core.beam_tod_batch(nside, None, data, rot, ph, th, ps)

    ref = call(rot, ph, th, ps)
    rot2, ph2, th2, ps2 = (np.concatenate([a, a]) for a in (rot, ph, th, ps))
    for bad in ((rot2, ph, th, ps), (rot, ph, th2, ps), (rot, ph, th, ps2), (rot[:3], ph, th, ps),
                (rot, ph, th[:1], ps), (rot, ph, th, ps[:1])):
        with pytest.raises((ValueError, RuntimeError)):
            call(*bad)
    # a single sample's roll may be a plain number
    one = call(rot[:1], ph[:1], th[:1], float(ps[0]))
    assert np.array_equal(one[0], ref[0][:1]) and np.array_equal(one[2], ref[2][:1])
    assert np.array_equal(call(rot.tolist(), ph, th.tolist(), ps.tolist())[1], ref[1])
