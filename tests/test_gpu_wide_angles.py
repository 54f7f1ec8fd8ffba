"""Beams of many degrees, footprints about the poles and rings of few pixels: the
pixel loops' form with atan2 and acos gives the direct evaluation's TOD bit for bit,
and the CPU oracle's to the bound of the other tests of device pointing."""

import math

import numpy as np
import pytest
import torch

import oracle
from tod_generation_mapbased_beam_b200 import _native
from tod_generation_mapbased_beam_b200.kernels import gather_accum, gather_accum_angles, pack_map

TOD_RTOL = 1e-10  # device pointing in float64 against the oracle
INTERP = {"bilinear": _native.BILINEAR, "nearest": _native.NEAREST}


def _disc(S, radius_deg, seed):
    rng = np.random.default_rng(seed)
    r = np.radians(radius_deg) * np.sqrt(rng.uniform(0, 1, S))
    a = rng.uniform(0, 2 * np.pi, S)
    bv = rng.uniform(0.1, 1.0, S).astype(np.float32)
    return np.stack([np.sin(r) * np.cos(a), np.sin(r) * np.sin(a), np.cos(r)], -1), bv / bv.sum()


def _pointing(B, seed, where):
    rng = np.random.default_rng(seed)
    th = {"sky": np.arccos(rng.uniform(-1, 1, B)),
          "poles": np.where(rng.uniform(0, 1, B) < 0.5, rng.uniform(0, 0.3, B), np.pi - rng.uniform(0, 0.3, B))}[where]
    return th, rng.uniform(0, 2 * np.pi, B), rng.uniform(0, 2 * np.pi, B)


def _oracle(mode, vec, bv, ang, nside, sky, c_q, c_u):
    th, ph, ps = ang
    rot, beta = oracle.rotation_vectors_f64(0.0, 0.0, ph, th)
    params = oracle.rotation_params_f64(rot, ph, th, ps - beta)
    out = np.zeros((sky.shape[0], len(th)))
    fn = oracle.gather_accum_fused if mode == "bilinear" else oracle.gather_accum_nearest
    fn(vec, *params, nside, sky, bv, len(th), vec.shape[0], out, c_q, c_u, f64=True)
    return out


def _gather(mode, vec, bv, ang, nside, mp, c_q, c_u, C, flags=0):
    tod = torch.zeros((C, len(ang[0])), dtype=torch.float64, device="cuda")
    gather_accum_angles(INTERP[mode], vec, *ang, 0.0, 0.0, nside, mp, bv, tod, c_q, c_u, flags=flags)
    return tod.cpu().numpy()


@pytest.mark.gpu
@pytest.mark.parametrize("mode", ["bilinear", "nearest"])
@pytest.mark.parametrize("where", ["sky", "poles"])
@pytest.mark.parametrize("nside", [1, 4, 16, 39, 40, 64, 256])
@pytest.mark.parametrize("radius", [0.5, 3.4, 3.6, 7.0, 12.0, 40.0, 90.0])
def test_wide_beams_match_direct_and_oracle(mode, where, nside, radius):
    S, B = 700, 120
    vec, bv = _disc(S, radius, 1)
    ang = _pointing(B, 2, where)
    sky = np.random.default_rng(3).standard_normal((3, 12 * nside * nside))
    dev = torch.from_numpy(sky).cuda()
    got = _gather(mode, vec, bv, ang, nside, dev, 1, 2, 3)
    assert np.array_equal(got, _gather(mode, vec, bv, ang, nside, dev, 1, 2, 3, _native.FLAG_NO_TABLES))
    assert np.array_equal(got, _gather(mode, vec, bv, ang, nside, dev, 1, 2, 3, _native.FLAG_WIDE_CTAS))
    ref = _oracle(mode, vec, bv, ang, nside, sky, 1, 2)
    err = np.abs(got - ref).max(axis=0) / np.abs(ref).max()
    if mode == "nearest":  # a pixel may flip where the two pointings' last bits decide a tie
        assert np.mean(err > TOD_RTOL) <= 0.05
    else:
        assert err.max() <= TOD_RTOL


@pytest.mark.gpu
@pytest.mark.parametrize("mode", ["bilinear", "nearest"])
@pytest.mark.parametrize("C, c_q, c_u", [(1, -1, -1), (3, 2, 0), (4, 1, 3)])
@pytest.mark.parametrize("kind", ["planar", "planar32", "f64", "f32", "bf16"])
def test_layouts(mode, C, c_q, c_u, kind):
    nside, S, B = 64, 500, 60
    vec, bv = _disc(S, 15.0, 4)
    ang = _pointing(B, 5, "sky")
    sky = torch.from_numpy(np.random.default_rng(6).standard_normal((C, 12 * nside * nside))).cuda()
    mp = sky if kind == "planar" else sky.float() if kind == "planar32" else pack_map(sky, kind)
    got = _gather(mode, vec, bv, ang, nside, mp, c_q, c_u, C)
    assert np.array_equal(got, _gather(mode, vec, bv, ang, nside, mp, c_q, c_u, C, _native.FLAG_NO_TABLES))
    assert np.abs(got).max() > 0


@pytest.mark.gpu
@pytest.mark.parametrize("mode", ["bilinear", "nearest"])
@pytest.mark.parametrize("nside, radius", [(16, 10.0), (128, 9.0), (256, 1.0)])
def test_reference_typing(mode, nside, radius):
    """Float32 parameters, whose z follows the reference's rounding beyond |z| = 0.9."""
    S, B = 500, 90
    vec, bv = _disc(S, radius, 7)
    th, ph, ps = _pointing(B, 8, "poles")
    rot, beta = oracle.rotation_vectors_f64(0.0, 0.0, ph, th)
    params = [np.asarray(p, np.float32) for p in oracle.rotation_params_f64(rot, ph, th, ps - beta)]
    sky = torch.from_numpy(np.random.default_rng(9).standard_normal((3, 12 * nside * nside))).cuda()
    outs = []
    for flags in (0, _native.FLAG_NO_TABLES):
        tod = torch.zeros((3, B), dtype=torch.float64, device="cuda")
        gather_accum(INTERP[mode], vec.astype(np.float32), *params, nside, sky, bv, B, S, tod, 1, 2, flags=flags)
        outs.append(tod.cpu().numpy())
    assert np.array_equal(outs[0], outs[1]) and np.abs(outs[0]).max() > 0
    cpu = np.zeros((3, B))
    fn = oracle.gather_accum_fused if mode == "bilinear" else oracle.gather_accum_nearest
    fn(vec.astype(np.float32), *params, nside, sky.cpu().numpy(), bv, B, S, cpu, 1, 2)
    err = np.abs(outs[0] - cpu).max(axis=0) / np.abs(cpu).max()
    assert np.mean(err > 1e-12) <= (0.05 if mode == "nearest" else 0.02) and math.isfinite(err.max())
