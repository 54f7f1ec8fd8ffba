"""Beams whose footprint has no table of pixel values: sparse ones (a table would hold
more slots than the beam reads), footprints larger than one CTA's shared memory, I
alone in passes.  The pixel loops that read the map give the direct evaluation's TOD
bit for bit, and in a batch such a beam does not take the others' table."""

import ctypes

import numpy as np
import pytest
import torch

import oracle
from tod_generation_mapbased_beam_b200 import _native
from tod_generation_mapbased_beam_b200 import workloads as W
from tod_generation_mapbased_beam_b200.batched import DetectorBatch
from tod_generation_mapbased_beam_b200.kernels import footprint_slots, gather_accum, gather_accum_angles, pack_map

TOD_RTOL = 1e-10  # device pointing in float64 against the oracle
INTERP = {"bilinear": _native.BILINEAR, "nearest": _native.NEAREST}


def _wants(nside, S, slots, C=3, qu=True, mode="bilinear", map_dtype=_native.F64, table=16):
    """(rings, slots) that a launch of these arguments reserves."""
    a = _native.GatherArgs()
    a.abi_version, a.interp, a.nside, a.B, a.S, a.C = _native.ABI_VERSION, INTERP[mode], nside, 8, S, C
    a.c_q, a.c_u = (1, 2) if qu else (-1, -1)
    a.params_dtype, a.map_dtype, a.map_stride, a.tod_stride = _native.F64, map_dtype, 12 * nside * nside, 8
    for f in ("vec_orig", "axes", "cos_a", "sin_a", "ax_pts", "cos_p", "sin_p", "beam_vals", "map", "tod"):
        setattr(a, f, 16)  # (not read)
    a.ring_table, a.tab_slots = table, slots
    rings, got = ctypes.c_int32(), ctypes.c_int32()
    _native.check(_native.lib().todgpu_gather_wants(ctypes.byref(a), ctypes.byref(rings), ctypes.byref(got)))
    return rings.value, got.value


def _rings(slots):
    return int(np.ceil(3.0 * np.sqrt(slots / 3.15))) + 6


def test_tables_only_where_they_pay():
    n = footprint_slots(2048, np.radians(0.5) + 3.0 / 2048)  # 30' at nside 2048
    assert 1200 < n < 1350
    assert _wants(2048, 1600, n) == (_rings(n), n)
    assert _wants(2048, 100, n)[1] == 0
    assert _wants(2048, 1600, n, C=1, qu=False)[1] == n and _wants(2048, 100, n, C=1, qu=False)[1] == 0
    big = footprint_slots(8192, np.radians(0.5) + 3.0 / 8192)  # 17,000: more than a CTA holds
    assert _wants(8192, 16000, big) == (_rings(big), 0)
    assert _wants(8192, 1000, big, C=1, qu=False) == (_rings(big), 0)
    assert _wants(4096, 1000, 9500, map_dtype=_native.PACKED_F32)[1] == 0
    assert _wants(4096, 16000, 9500, map_dtype=_native.PACKED_F32)[1] == 9500
    # nearest: turned values only, and no more slots than pixels
    assert _wants(2048, n, n, mode="nearest")[1] == n and _wants(2048, n - 1, n, mode="nearest")[1] == 0
    assert _wants(2048, n, n, mode="nearest", C=1, qu=False) == (_rings(n), 0)
    # in passes: the default table where a pass's share of the footprint fits it
    assert _wants(1024, 100000, 10 * 2048)[1] == 2048
    assert _wants(1024, 60000, 140000) == (448, 0)
    assert _wants(1024, 100000, 10 * 2048, C=1, qu=False)[1] == 0
    assert _wants(2048, 1600, n, table=None) == (1, 0)


def _disc(S, radius_deg, seed):
    rng = np.random.default_rng(seed)
    r = np.radians(radius_deg) * np.sqrt(rng.uniform(0, 1, S))
    a = rng.uniform(0, 2 * np.pi, S)
    bv = rng.uniform(0.1, 1.0, S).astype(np.float32)
    return np.stack([np.sin(r) * np.cos(a), np.sin(r) * np.sin(a), np.cos(r)], -1), bv / bv.sum()


def _pointing(B, seed):
    rng = np.random.default_rng(seed)
    th = np.concatenate([np.arccos(rng.uniform(-1, 1, B - 6)), [0.0, 0.004, 0.05, np.pi, np.pi - 0.004, 3.0]])
    return th, rng.uniform(0, 2 * np.pi, B), rng.uniform(0, 2 * np.pi, B)


# nside 1 to 4: rings of four pixels; S = 1, 255 .. 513: the remainders of the lanes
CASES = [(1, 60.0, 3), (2, 20.0, 1), (4, 5.0, 7), (512, 1.0, 1), (512, 1.0, 255), (512, 1.0, 257), (512, 1.0, 300),
         (1024, 2.0, 513), (1024, 6.0, 900), (2048, 12.0, 400), (1024, 3.0, 2100)]


@pytest.mark.gpu
@pytest.mark.parametrize("kind, C, c_q, c_u", [("planar", 3, 1, 2), ("planar", 1, -1, -1), ("planar32", 4, 3, 0),
                                               ("f64", 2, -1, -1), ("f32", 3, 1, 2), ("bf16", 1, -1, -1)])
@pytest.mark.parametrize("nside, radius, S", CASES)
def test_map_loop_is_the_direct_evaluation(nside, radius, S, kind, C, c_q, c_u):
    B = 60
    vec, bv = _disc(S, radius, 1)
    ang = _pointing(B, 2)
    sky = np.random.default_rng(3).standard_normal((C, 12 * nside * nside))
    dev = torch.from_numpy(sky).cuda()
    mp = dev if kind == "planar" else dev.float() if kind == "planar32" else pack_map(dev, kind)
    th, ph, ps = ang
    rot, beta = oracle.rotation_vectors_f64(0.0, 0.0, ph, th)
    params = oracle.rotation_params_f64(rot, ph, th, ps - beta)
    for mode in INTERP:
        outs = []
        for flags in (0, _native.FLAG_NO_TABLES, _native.FLAG_WIDE_CTAS):
            tod = torch.zeros((C, B), dtype=torch.float64, device="cuda")
            gather_accum_angles(INTERP[mode], vec, *ang, 0.0, 0.0, nside, mp, bv, tod, c_q, c_u, flags=flags)
            outs.append(tod.cpu().numpy())
            ref = torch.zeros((C, B), dtype=torch.float64, device="cuda")
            gather_accum(INTERP[mode], vec.astype(np.float32), *[np.asarray(p, np.float32) for p in params], nside, mp, bv,
                         B, S, ref, c_q, c_u, flags=flags)
            outs.append(ref.cpu().numpy())
        for k in (2, 3, 4, 5):
            assert np.array_equal(outs[k % 2], outs[k])
        assert all(np.abs(o).max() > 0 for o in outs)
        if mode == "bilinear" and kind == "planar":
            want = np.zeros((C, B))
            oracle.gather_accum_fused(vec, *params, nside, sky, bv, B, S, want, c_q, c_u, f64=True)
            # (the last bits of the two pointings differ: not at the poles themselves)
            err = np.abs(outs[0] - want)[:, : B - 6].max() / np.abs(want).max()
            assert err <= TOD_RTOL


@pytest.mark.gpu
@pytest.mark.parametrize("C, c_q, c_u", [(1, -1, -1), (3, 1, 2)])
@pytest.mark.parametrize("radius", [1.5, 12.0])
def test_passes(C, c_q, c_u, radius):
    """More than 16384 pixels with float32 parameters: passes of 1024 or 4096."""
    nside, S, B = 256, 16384 + 4097, 24
    vec, bv = _disc(S, radius, 4)
    th, ph, ps = _pointing(B, 5)
    rot, beta = oracle.rotation_vectors_f64(0.0, 0.0, ph, th)
    params = [np.asarray(p, np.float32) for p in oracle.rotation_params_f64(rot, ph, th, ps - beta)]
    sky = torch.from_numpy(np.random.default_rng(6).standard_normal((C, 12 * nside * nside))).cuda()
    for mode in INTERP.values():
        outs = []
        for flags in (0, _native.FLAG_NO_TABLES, _native.FLAG_WIDE_CTAS):
            tod = torch.zeros((C, B), dtype=torch.float64, device="cuda")
            gather_accum(mode, vec.astype(np.float32), *params, nside, sky, bv, B, S, tod, c_q, c_u, flags=flags)
            outs.append(tod.cpu().numpy())
        assert np.array_equal(outs[0], outs[1]) and np.array_equal(outs[0], outs[2]) and np.abs(outs[0]).max() > 0


@pytest.mark.gpu
@pytest.mark.parametrize("mode", ["bilinear", "nearest"])
@pytest.mark.parametrize("n_wide", [40, 3000])  # joins the others' launch; has one of its own
def test_batch_with_a_beam_without_a_table(mode, n_wide):
    nside = 512
    sky = W.white_sky(nside, 7)
    dets = []
    for d, (S, radius, n) in enumerate([(900, 0.5, 500), (700, 7.0, n_wide), (1200, 0.6, 300), (5, 0.6, n_wide)]):
        vec, bv = _disc(S, radius, d)
        th, ph, ps = W.spin_scan(n, 0.5)
        dets.append(dict(vec_orig=vec, beam_vals=bv, theta=th, phi=ph, psi=ps, center=(0.0, 0.0)))
    run = lambda ds: [o.cpu().numpy() for o in _run(DetectorBatch(nside, sky, ds, interp_mode=mode, tile=1, graph=False))]
    whole = run(dets)
    for d, got in zip(dets, whole):
        assert np.array_equal(got, run([d])[0]) and np.abs(got).max() > 0


def _run(batch):
    batch.run()
    torch.cuda.synchronize()
    return batch.out
