"""GPU test of a batch whose jobs' own shapes differ: it runs as one launch per
shape where each has tiles enough and as one launch where not, with the TOD of
one gather per detector bit for bit either way."""

import numpy as np
import pytest
import torch

from tod_generation_mapbased_beam_b200 import workloads as W
from tod_generation_mapbased_beam_b200.batched import DetectorBatch
from tod_generation_mapbased_beam_b200.kernels import beam_order, gather_accum_angles, pack_map

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lengths", [(30000, 30000, 31000), (30000, 500, 31000), (500, 0, 700)])
@pytest.mark.parametrize("tile", [1, 16])
@pytest.mark.parametrize("graph", [False, True])
def test_jobs_of_different_shapes_equal_single_launches(lengths, tile, graph):
    nside = 512
    sky = pack_map(torch.from_numpy(W.white_sky(nside, 3, dtype=np.float32)).cuda(), "f32")
    dets = []
    for k, (fwhm, n) in enumerate(zip((60.0, 150.0, 100.0), lengths)):
        beam = W.pole_gaussian_beam(fwhm, 256, 0.99, search_fwhm=1.5)
        th, ph, ps = W.spin_scan(n, 100.0, t0=100.0 * k, phi0=0.5 * k)
        dets.append(dict(vec_orig=beam.vec_orig, beam_vals=beam.beam_vals, theta=th, phi=ph, psi=ps, center=(0.0, 0.0)))
    batch = DetectorBatch(nside, sky, dets, tile=tile, graph=graph)
    got = [o.cpu().numpy() for o in batch.run()]
    for d, g in zip(dets, got):
        o = beam_order(d["vec_orig"])
        tod = torch.zeros((3, len(d["theta"])), dtype=torch.float64, device="cuda")
        if len(d["theta"]):
            gather_accum_angles(0, np.asarray(d["vec_orig"])[o], d["theta"], d["phi"], d["psi"], 0.0, 0.0, nside, sky,
                                np.asarray(d["beam_vals"])[o], tod, 1, 2)
        np.testing.assert_array_equal(g, tod.cpu().numpy())
