"""The gather's per-sample windows and tables at the sizes where they can go wrong.

Every sample's footprint is laid out as a window of rings and a table of turned map
values in shared memory; beam pixels that they do not hold are evaluated directly.
Window and table decide speed only, so the TOD must equal the direct evaluation's
(FLAG_NO_TABLES) bit for bit, and the CPU oracle's to the bound of the other tests
of device pointing in float64 (the oracle's own terms carry rounding errors of up to
3e-12 of the largest magnitude where a footprint holds a pole)."""

import math

import numpy as np
import pytest
import torch

import oracle
from tod_generation_mapbased_beam_b200 import _native
from tod_generation_mapbased_beam_b200.kernels import (footprint_slots, gather_accum, gather_accum_angles, pack_map,
                                                       patch_order, planar_beam)

TOD_RTOL = 1e-10


def _disc(S, radius_deg, seed, offset_deg=0.0):
    rng = np.random.default_rng(seed)
    r = np.radians(radius_deg) * np.sqrt(rng.uniform(0, 1, S))
    a = rng.uniform(0, 2 * np.pi, S)
    v = np.stack([np.sin(r) * np.cos(a), np.sin(r) * np.sin(a), np.cos(r)], -1)
    o = math.radians(offset_deg)
    v = np.stack([v[:, 0] * math.cos(o) + v[:, 2] * math.sin(o), v[:, 1], v[:, 2] * math.cos(o) - v[:, 0] * math.sin(o)],
                 -1)
    bv = rng.uniform(0.1, 1.0, S).astype(np.float32)
    return v, bv / bv.sum()


def _pointing(B, seed, where):
    rng = np.random.default_rng(seed)
    th = {"sky": rng.uniform(0.05, np.pi - 0.05, B),
          "belt edge": np.arccos(2 / 3) + rng.uniform(-0.05, 0.05, B),
          "south edge": np.pi - np.arccos(2 / 3) + rng.uniform(-0.05, 0.05, B),
          "poles": np.where(rng.uniform(0, 1, B) < 0.5, rng.uniform(0, 0.2, B), np.pi - rng.uniform(0, 0.2, B)),
          "seam": rng.uniform(0.5, 2.6, B)}[where]
    ph = rng.normal(0, 5e-3, B) % (2 * np.pi) if where == "seam" else rng.uniform(0, 2 * np.pi, B)
    return th, ph, rng.uniform(0, 2 * np.pi, B)


def _sky(nside, seed, C=3):
    return torch.from_numpy(np.random.default_rng(seed).standard_normal((C, 12 * nside * nside))).cuda()


def _angles(interp, vec, bv, ang, nside, mp, c_q, c_u, flags=0, C=3):
    tod = torch.zeros((C, len(ang[0])), dtype=torch.float64, device="cuda")
    gather_accum_angles(interp, vec, *ang, 0.0, 0.0, nside, mp, bv, tod, c_q, c_u, flags=flags)
    return tod.cpu().numpy()


def _oracle(mode, vec, bv, ang, nside, sky, c_q, c_u):
    th, ph, ps = ang
    rot, beta = oracle.rotation_vectors_f64(0.0, 0.0, ph, th)
    params = oracle.rotation_params_f64(rot, ph, th, ps - beta)
    out = np.zeros((sky.shape[0], len(th)))
    fn = oracle.gather_accum_fused if mode == "bilinear" else oracle.gather_accum_nearest
    fn(vec, *params, nside, sky.cpu().numpy(), bv, len(th), vec.shape[0], out, c_q, c_u, f64=True)
    return out


INTERP = {"bilinear": _native.BILINEAR, "nearest": _native.NEAREST}


@pytest.mark.gpu
@pytest.mark.parametrize("mode", ["bilinear", "nearest"])
@pytest.mark.parametrize("where", ["sky", "belt edge", "south edge", "poles", "seam"])
@pytest.mark.parametrize("radius, offset", [(0.7, 0.0), (0.7, 1.0), (4.0, 0.0)])
def test_regions_match_direct_and_oracle(mode, where, radius, offset):
    nside, S, B = 256, 600, 173
    vec, bv = _disc(S, radius, 1, offset)
    ang = _pointing(B, 2, where)
    sky = _sky(nside, 3)
    got = _angles(INTERP[mode], vec, bv, ang, nside, sky, 1, 2)
    assert np.array_equal(got, _angles(INTERP[mode], vec, bv, ang, nside, sky, 1, 2, _native.FLAG_NO_TABLES))
    ref = _oracle(mode, vec, bv, ang, nside, sky, 1, 2)
    err = np.abs(got - ref).max(axis=0) / np.abs(ref).max()
    if mode == "nearest":  # a pixel may flip where the two pointings' last bits decide a tie
        assert np.mean(err > TOD_RTOL) <= 0.02
    else:
        assert err.max() <= TOD_RTOL


@pytest.mark.gpu
@pytest.mark.parametrize("mode", ["bilinear", "nearest"])
@pytest.mark.parametrize("S", [1, 2, 127, 128, 129, 255, 256, 257, 511, 512, 513, 769])
@pytest.mark.parametrize("B", [1, 15, 33])
def test_beam_and_batch_remainders(mode, S, B):
    """Beam sizes about the summation lanes and pixel pairs, batches about the
    sixteen samples prepared together; 128- and 256-thread CTAs."""
    nside = 128
    vec, bv = _disc(S, 1.0, 4)
    ang = _pointing(B, 5, "sky")
    sky = _sky(nside, 6)
    outs = [_angles(INTERP[mode], vec, bv, ang, nside, sky, 1, 2, f)
            for f in (0, _native.FLAG_NO_TABLES, _native.FLAG_WIDE_CTAS)]
    assert np.abs(outs[0]).max() > 0
    assert np.array_equal(outs[0], outs[1]) and np.array_equal(outs[0], outs[2])


@pytest.mark.gpu
@pytest.mark.parametrize("mode", ["bilinear", "nearest"])
@pytest.mark.parametrize("kind", ["planar", "planar32", "f64", "f32", "bf16"])
@pytest.mark.parametrize("C, c_q, c_u", [(1, -1, -1), (2, -1, -1), (2, 0, 1), (3, 2, 0), (4, 1, 3), (4, -1, -1)])
def test_component_layouts(mode, kind, C, c_q, c_u):
    nside, S, B = 128, 300, 40
    vec, bv = _disc(S, 1.5, 7)
    ang = _pointing(B, 8, "sky")
    sky = _sky(nside, 9, C)
    mp = sky if kind == "planar" else sky.float() if kind == "planar32" else pack_map(sky, kind)
    got = _angles(INTERP[mode], vec, bv, ang, nside, mp, c_q, c_u, C=C)
    assert np.array_equal(got, _angles(INTERP[mode], vec, bv, ang, nside, mp, c_q, c_u, _native.FLAG_NO_TABLES, C=C))
    # each output is the map's own component turned with the others' as the oracle does
    ref = _oracle(mode, vec, bv, ang, nside, sky, c_q, c_u)
    tol = {"planar": TOD_RTOL, "f64": TOD_RTOL, "planar32": 1e-6, "f32": 1e-6, "bf16": 2e-2}[kind]
    err = np.abs(got - ref).max(axis=0) / np.abs(ref).max()
    assert np.mean(err > tol) <= (0.05 if mode == "nearest" else 0.0)


@pytest.mark.gpu
@pytest.mark.parametrize("mode", ["bilinear", "nearest"])
@pytest.mark.parametrize("dtype", [np.float32, np.float64])
def test_planar_vectors_give_the_same_tod(mode, dtype):
    nside, S, B = 256, 700, 50
    vec, bv = _disc(S, 1.0, 10)
    th, ph, ps = _pointing(B, 11, "sky")
    rot, beta = oracle.rotation_vectors_f64(0.0, 0.0, ph, th)
    params = [np.asarray(p, dtype) for p in oracle.rotation_params_f64(rot, ph, th, ps - beta)]
    sky = _sky(nside, 12)
    v = torch.from_numpy(vec.astype(dtype)).cuda()
    assert planar_beam(v, 1)[1] == 0 and planar_beam(planar_beam(v)[0], 1)[1] == _native.FLAG_BEAM_PLANAR
    outs = []
    for beam in (v, planar_beam(v)[0]):
        tod = torch.zeros((3, B), dtype=torch.float64, device="cuda")
        gather_accum(INTERP[mode], beam, *params, nside, sky, bv, B, S, tod, 1, 2)
        outs.append(tod.cpu().numpy())
    assert np.array_equal(outs[0], outs[1])


@pytest.mark.gpu
@pytest.mark.parametrize("mode", ["bilinear", "nearest"])
@pytest.mark.parametrize("precompute", [True, False])
def test_beam_in_chunks(mode, precompute):
    """More than 16384 beam pixels: chunks of the beam with their own centres and
    frames, the last one ragged -- as jobs of their own (precompute) or one after
    another in one launch."""
    nside, S, B = 64, 16384 + 1029, 20
    vec, bv = _disc(S, 9.0, 13)
    ang = _pointing(B, 14, "sky")
    sky = _sky(nside, 15)
    outs = []
    for flags in (0, _native.FLAG_NO_TABLES):
        tod = torch.ones((3, B), dtype=torch.float64, device="cuda")
        gather_accum_angles(INTERP[mode], vec, *ang, 0.0, 0.0, nside, sky, bv, tod, 1, 2, flags=flags,
                            precompute=precompute)
        outs.append(tod.cpu().numpy())
    assert np.array_equal(outs[0], outs[1])
    got = outs[0] - 1.0
    ref = _oracle(mode, vec, bv, ang, nside, sky, 1, 2)
    err = np.abs(got - ref).max(axis=0) / np.abs(ref).max()
    assert np.mean(err > TOD_RTOL) <= (0.2 if mode == "nearest" else 0.0)


@pytest.mark.gpu
@pytest.mark.parametrize("mode", ["bilinear", "nearest"])
def test_non_finite_beam_pixels_leave_the_others_alone(mode):
    """A NaN or infinite beam vector spoils only its own terms (bilinear: skipped
    and counted), with and without tables."""
    nside, S, B = 64, 300, 9
    vec, bv = _disc(S, 2.0, 16)
    ang = _pointing(B, 17, "sky")
    sky = _sky(nside, 18)
    bad = vec.copy()
    bad[17, 0] = np.nan
    bad[40] = np.inf
    outs = [_angles(INTERP[mode], bad, bv, ang, nside, sky, 1, 2, f) for f in (0, _native.FLAG_NO_TABLES)]
    assert np.array_equal(outs[0], outs[1], equal_nan=True)
    if mode == "bilinear":
        keep = np.ones(S, bool)
        keep[[17, 40]] = False
        ref = _oracle(mode, vec[keep], bv[keep], ang, nside, sky, 1, 2)
        assert np.abs(outs[0] - ref).max() <= TOD_RTOL * np.abs(ref).max()
        err = torch.zeros(1, dtype=torch.int64, device="cuda")
        tod = torch.zeros((3, B), dtype=torch.float64, device="cuda")
        gather_accum_angles(_native.BILINEAR, bad, *ang, 0.0, 0.0, nside, sky, bv, tod, 1, 2, err_count=err)
        assert int(err.item()) == 2 * B


def test_patch_order_makes_compact_runs():
    """Runs of 1024 pixels of a full disc in patch_order are patches: their radius
    stays within twice a square patch's half diagonal, 0.71 sqrt(run's share of
    the area); every pixel appears once."""
    S, radius = 40000, 5.0
    vec, _ = _disc(S, radius, 21)
    order = patch_order(vec)
    assert np.array_equal(np.sort(order), np.arange(S))
    half_diagonal = math.sqrt(math.pi * math.radians(radius) ** 2 * 1024 / S / 2)
    for a in range(0, S, 1024):
        p = vec[order[a:a + 1024]]
        c = p.sum(axis=0) / np.linalg.norm(p.sum(axis=0))
        assert np.arccos(np.clip((p @ c).min(), -1, 1)) <= 2 * half_diagonal


def _ring(n, i):
    """z and pixel count of RING ring i."""
    if i < n:
        return 1 - i * i / (3.0 * n * n), 4 * i
    if i <= 3 * n:
        return (2 * n - i) * 2.0 / (3.0 * n), 4 * n
    j = 4 * n - i
    return -(1 - j * j / (3.0 * n * n)), 4 * j


def _ring_above(n, z):
    az = abs(z)
    if az > 2.0 / 3.0:
        ir = int(n * math.sqrt(3 * (1 - az)))
        return 4 * n - ir - 1 if z < 0 else ir
    return int(n * (2 - 1.5 * z))


@pytest.mark.parametrize("nside, radius", [(1024, 0.011), (2048, 0.0138), (512, 0.02), (128, 0.04), (256, 0.09),
                                           (4096, 0.01), (1024, 0.0005)])
def test_request_covers_every_footprint(nside, radius):
    """The slots and rings a footprint takes (footprint_window of the gather,
    restated) stay within kernels.footprint_slots and the rings reserved for it
    (ring_cap_for), wherever the footprint lies and whatever its longitude."""
    reach = math.ceil((radius + 3 / nside + 2e-5) / 1e-4) * 1e-4
    rb, sp = radius + 1e-5, 0.9 / nside
    want = footprint_slots(nside, reach)
    rng = np.random.default_rng(1)
    worst = 0
    for th in np.linspace(0.1 + rb + 1e-6, math.pi - 0.1 - rb - 1e-6, 301):
        a, b = max(1, _ring_above(nside, math.cos(th - rb))), _ring_above(nside, math.cos(th + rb)) + 1
        phi = rng.uniform(0, 2 * math.pi)
        total = 0
        for i in range(a, b + 1):
            z, n = _ring(nside, i)
            sth, dphi = math.sqrt(1 - z * z), 2 * math.pi / n
            shifted = i < nside or i > 3 * nside or (i - nside) % 2 == 0
            x = (phi - (dphi / 2 if shifted else 0.0)) / dphi
            d = max(0.0, abs(math.acos(z) - th) - sp)
            q = max(0.0, math.sin(rb / 2) ** 2 - math.sin(d / 2) ** 2) / math.sin(th) / (sth - sp)
            half = 2.04 * math.asin(min(1.0, math.sqrt(q))) / dphi
            total += min(n, 2 * int(x - math.floor(x) + half) + 3)
        worst = max(worst, total)
        assert b - a + 1 <= math.ceil(3.0 * math.sqrt(want / 3.15)) + 6
    assert worst <= want <= 1.15 * worst + 16
