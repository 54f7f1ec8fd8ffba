"""What a user of this framework has it compute, as measurable cases.

Every case goes through a public entry point: the drop-in ``beam_tod_batch``, the
kernel-level ``_gather_accum_fused_jit``, the device-pointing ``beam_tod_angles`` and
``gather_accum_angles``, the day driver, the detector batch, the far-sidelobe tail by
the plain method and by its network (inference and training), and beam clustering.

:func:`prepare` builds what a program holds before the call (sky, beam, pointing,
plans), from the seed alone; :func:`run` is one pass; :func:`exact` is the same result
in 64-bit torch or numpy without this package's code.  Scans stay away from the poles
(the spin scan spans 40 to 140 degrees in colatitude), so the reference stencil below
needs no pole rule.
"""

import math

import numpy as np
import torch

from tod_generation_mapbased_beam_b200 import _native, beam_cluster, tod_bilinear, tod_core
from tod_generation_mapbased_beam_b200 import tod_rotations as rotations
from tod_generation_mapbased_beam_b200 import workloads
from tod_generation_mapbased_beam_b200.batched import DetectorBatch
from tod_generation_mapbased_beam_b200.driver import DayRunner
from tod_generation_mapbased_beam_b200.kernels import beam_order, gather_accum_angles, pack_map
from tod_generation_mapbased_beam_b200.learned import LearnedTailTOD
from tod_generation_mapbased_beam_b200.tailnet import TailNet

PI = math.pi
RMS = (100e-6, 31.6e-6, 31.6e-6)  # I, Q, U of the sky [K]
F32, F64 = torch.float32, torch.float64


def listed():
    return [
        # The smallest call: one small batch of the nside 128 workload (elliptical 1.5/1.8
        # degree beam shared by I and Q, no spin-2), everything in host memory, as a
        # program written for the reference calls it.
        dict(name="dropin_small", kind="dropin", nside=128, fwhm=108.0, fwhm2=90.0, beam_nside=256, cut=0.99,
             comps="IQ", map="f64", map_on="host", mode="bilinear", n=64),
        # One batch of the reference's day loop: its batch size, its float32 sky (kept on
        # the GPU by the caller), host pointing in, float32 host TOD out.
        dict(name="dropin_batch", kind="dropin", nside=1024, fwhm=30.0, fwhm2=30.0, beam_nside=2048, cut=0.99,
             comps="IQU", map="f32", map_on="gpu", mode="bilinear", n=32768),
        # The fused kernel on prepared float32 parameters and a float64 sky: the parity
        # form of the 30' benchmark beam.
        dict(name="fused_f64", kind="fused", nside=1024, fwhm=30.0, beam_nside=2048, cut=0.99, map="f64",
             n=120011),
        # Device pointing, nearest mode: the quick-look form of the same day.
        dict(name="angles_nearest", kind="angles", nside=1024, fwhm=30.0, beam_nside=2048, cut=0.99, map="f64",
             mode="nearest", n=100003),
        # A stretch of a day end to end: host scan in, host float64 TOD out.
        dict(name="day_run", kind="day", nside=1024, fwhm=30.0, beam_nside=2048, cut=0.99, map="f64",
             mode="bilinear", n=1200007),
        # Precision form: nside 2048 sky in packed float32 records, 30' beam pixelised
        # finely (9,530 pixels), float32 Kahan sums.
        dict(name="precision_f32", kind="angles", nside=2048, fwhm=30.0, beam_nside=4096, cut=0.999, map="pf32",
             mode="bilinear", n=20011),
        # The bfloat16 record variant at a lower resolution and a wider beam.
        dict(name="precision_bf16", kind="angles", nside=512, fwhm=45.0, beam_nside=1024, cut=0.99, map="pbf16",
             mode="bilinear", n=50021),
        # Many detectors with their own beams, offsets and uneven scan lengths in one
        # launch over a float32 sky.
        dict(name="detectors", kind="detectors", nside=2048, beam_nside=2048, map="f32", detectors=6, n_min=4001,
             n_max=60013, tile=16),
        # Far sidelobes of one beam (10-20 degree annulus, 284k pixels) by the plain
        # float64 method: the targets and the judge of the learned tail.
        dict(name="plain_tail", kind="tail", nside=1024, beam_nside=1024, map="f64", n=301),
        # The learned tail in use: the network's prediction added into a TOD.
        dict(name="tail_network", kind="network", n_freq=256, width=256, depth=4, n=500009),
        # The learned tail in training: loss and gradient of one batch.
        dict(name="tail_training", kind="training", n_freq=256, width=256, depth=4, n=8192),
        # Beam preparation: the weak tail of a beam clustered (host lists in and out).
        dict(name="cluster_tail", kind="cluster", fwhm=30.0, beam_nside=4096, cut=0.999, tail=0.05, clusters=200),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case of the same ranges: sizes over their logarithm, odd ones too, the work
    bounded by the listed cases' largest (about 2e9 beam-pixel evaluations)."""
    kind = rng.choice(["dropin", "dropin", "fused", "angles", "angles", "angles", "day", "detectors", "tail",
                       "network", "training", "cluster"])
    mode = rng.choice(["bilinear", "bilinear", "nearest"])
    if kind == "network":
        return dict(kind=kind, n_freq=rng.choice([64, 128, 256]), width=rng.choice([128, 256]),
                    depth=rng.randint(2, 5), n=_log(rng, 1000, 500000))
    if kind == "training":
        return dict(kind=kind, n_freq=rng.choice([64, 128, 256]), width=rng.choice([128, 256]),
                    depth=rng.randint(2, 5), n=128 * _log(rng, 8, 128))
    if kind == "cluster":
        return dict(kind=kind, fwhm=rng.uniform(25.0, 35.0), beam_nside=rng.choice([2048, 4096]), cut=0.999,
                    tail=rng.uniform(0.02, 0.08), clusters=_log(rng, 20, 250))
    if kind == "tail":
        nside = rng.choice([256, 512, 1024])
        return dict(kind=kind, nside=nside, beam_nside=nside, map="f64",
                    n=min(2000, _log(rng, 40, 300 * (1024 // nside) ** 2)))
    if kind == "detectors":
        nside = rng.choice([512, 1024, 2048])
        lo = _log(rng, 500, 4000)
        return dict(kind=kind, nside=nside, beam_nside=2048, map=rng.choice(["f32", "pf32"]),
                    detectors=rng.randint(2, 7), n_min=lo, n_max=lo * rng.randint(3, 14), tile=16)
    nside = rng.choice([128, 256, 512, 1024, 2048])
    fwhm = (30.0 if nside >= 1024 else 45.0 if nside >= 512 else 90.0) * rng.uniform(0.85, 1.2)
    beam_nside = nside * 2 if nside < 2048 else rng.choice([2048, 4096])
    cut = rng.choice([0.99, 0.999])
    pixels = _beam_of(dict(fwhm=fwhm, beam_nside=beam_nside, cut=cut)).S
    most = 2e9 / 2.0 / pixels
    case = dict(kind=kind, nside=nside, fwhm=fwhm, beam_nside=beam_nside, cut=cut)
    if kind == "dropin":
        return dict(case, fwhm2=fwhm * rng.uniform(0.8, 1.0), comps=rng.choice(["IQU", "IQU", "IQ", "I"]),
                    map=rng.choice(["f32", "f64"]), map_on="gpu", mode=mode, n=_log(rng, 1, min(60000, most)))
    if kind == "fused":
        return dict(case, map=rng.choice(["f64", "f64", "f32"]), n=_log(rng, 200, min(150000, most)))
    if kind == "angles":
        return dict(case, map=rng.choice(["f64", "pf32", "pbf16"]), mode=mode, n=_log(rng, 200, min(150000, most)))
    return dict(case, map=rng.choice(["f64", "f32"]), mode=mode, n=_log(rng, 5000, min(800000, most)))


# -- inputs ---------------------------------------------------------------------


def _beam_of(case):
    wide = 2.0 if case["cut"] > 0.99 else 1.5
    return workloads.pole_gaussian_beam(case["fwhm"], case["beam_nside"], case["cut"], case.get("fwhm2"),
                                        search_fwhm=wide)


def _sky(nside, seed, dtype):
    g = torch.Generator("cuda").manual_seed(seed)
    sky = torch.randn((3, 12 * nside * nside), generator=g, dtype=dtype, device="cuda")
    for c in range(3):
        sky[c] *= RMS[c]
    return sky


def _map(case, seed, comps=(0, 1, 2)):
    kind = case["map"]
    sky = _sky(case["nside"], seed, F32 if kind == "f32" else F64)
    if len(comps) < 3:
        sky = sky[list(comps)].contiguous()
    return pack_map(sky, kind[1:]) if kind in ("pf32", "pbf16") else sky


def _scan(n, seed):
    rng = np.random.default_rng(seed)
    return workloads.spin_scan(n, 100.0, t0=rng.uniform(0, 60.0), phi0=rng.uniform(0, 2 * PI))


def _gpu(*arrays):
    return [torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in arrays]


COMPS = {"I": [0], "IQ": [0, 1], "IQU": [0, 1, 2]}


def prepare(case, seed):
    kind = case["kind"]
    s = dict(case=case)
    if kind in ("network", "training"):
        net = TailNet(case["n_freq"], case["width"], case["depth"], 3, seed=seed)
        rng = np.random.default_rng(seed)
        n = case["n"]
        th, ph, ps = np.arccos(rng.uniform(-1, 1, n)), rng.uniform(0, 2 * PI, n), rng.uniform(0, 2 * PI, n)
        if kind == "network":
            net.shift, net.scale = np.array([1e-6, -2e-6, 5e-7]), np.array([3e-6, 1e-6, 2e-6])
            s["angles"] = _gpu(th, ph, ps)
        else:
            s["x"] = net.inputs(th, ph, ps)
            t = np.stack([np.sin(2 * th) * np.cos(ph), np.cos(2 * ps) * np.sin(th), np.sin(ph + ps)], -1)
            s["target"] = torch.from_numpy(t.astype(np.float32)).cuda()
        return dict(s, net=net)
    if kind == "cluster":
        beam = _beam_of(case)
        turn = np.random.default_rng(seed).uniform(0, 2 * PI)  # the beam's orientation on the sky
        vec = workloads.rotate_beam(beam.vec_orig, turn, 0.0, 0.0).astype(np.float32)
        return dict(s, vec=vec, vals=beam.beam_vals, seed=seed)
    if kind == "detectors":
        rng = np.random.default_rng(seed)
        m, dets = case["detectors"], []
        for d in range(m):
            f = d / max(1, m - 1)
            n = int(round(case["n_min"] * (case["n_max"] / case["n_min"]) ** f))
            beam = workloads.pole_gaussian_beam(25.0 + 10.0 * (1 - f), case["beam_nside"], 0.99,
                                                (25.0 + 10.0 * (1 - f)) * (1 - 0.1 * f), search_fwhm=1.5)
            th, ph, ps = _scan(n, int(rng.integers(1 << 30)))
            vec = workloads.rotate_beam(beam.vec_orig, rng.uniform(0, PI), math.radians(math.sqrt(rng.uniform())),
                                        rng.uniform(0, 2 * PI))
            dets.append(dict(vec_orig=vec, beam_vals=beam.beam_vals, theta=th, phi=ph, psi=ps, center=(0.0, 0.0)))
        mp = _map(case, seed)
        return dict(s, dets=dets, map=mp, batch=DetectorBatch(case["nside"], mp, dets, tile=case["tile"]))
    if kind == "tail":
        main, tail = workloads.config5_beams(beam_nside=case["beam_nside"], seed=5, fwhm_arcmin=60.0)
        sky = _sky(case["nside"], seed, F64)
        step = 7919  # pointings spread over the day
        scan = [a[::step].copy() for a in _scan(case["n"] * step, seed)]
        return dict(s, beam=tail, sky=sky, angles=_gpu(*scan), plan=LearnedTailTOD(case["nside"], sky, main, tail))
    comps = COMPS[case.get("comps", "IQU")]
    beam = _beam_of(case)
    th, ph, ps = _scan(case["n"], seed)
    mp = _map(case, seed, comps)
    s.update(beam=beam, map=mp, scan=(th, ph, ps))
    if kind in ("dropin", "fused"):
        rot, beta = rotations.precompute_rotation_vector_batch(beam.ra, beam.dec, ph, th)
        psis = -beta + ps
        if kind == "dropin":
            held = mp.cpu().numpy() if case["map_on"] == "host" else mp
            data = dict(vec_orig=beam.vec_orig, beam_vals=beam.beam_vals, comp_indices=comps, mp_stacked=held)
            return dict(s, data=data, rot=rot, psis=psis)
        order = beam_order(beam.vec_orig)
        params = rotations._rotation_params(rot, ph, th, psis)
        s["params"] = _gpu(beam.vec_orig[order], *params)
        s["vals"] = _gpu(beam.beam_vals[order])[0]
        s["bore"] = torch.from_numpy(np.arctan2(params[3][:, 1], params[3][:, 0])).cuda()
        s["held"] = pack_map(mp, "f64") if case["map"] == "f64" else mp
        return s
    data = dict(vec_orig=beam.vec_orig, beam_vals=beam.beam_vals, comp_indices=comps, ra=beam.ra, dec=beam.dec,
                mp_stacked=mp)
    if kind == "day":
        return dict(s, runner=DayRunner({"beam": data}, case["nside"], interp_mode=case["mode"], chunk=1 << 18))
    s["angles"] = _gpu(th, ph, ps)
    if case["map"] in ("f64", "f32"):
        return dict(s, data=data)
    order = beam_order(beam.vec_orig)
    s["vec"], s["vals"] = _gpu(beam.vec_orig[order].astype(np.float64), beam.beam_vals[order])
    return s


# -- one pass -------------------------------------------------------------------


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "dropin":
        th, ph, _ = s["scan"]
        return tod_core.beam_tod_batch(case["nside"], None, s["data"], s["rot"], ph, th, s["psis"],
                                       interp_mode=case["mode"])
    if kind == "fused":
        B, S = case["n"], s["beam"].S
        tod = torch.zeros((3, B), dtype=F64, device="cuda")
        tod_bilinear._gather_accum_fused_jit(*s["params"], case["nside"], s["held"], s["vals"], B, S, tod, 1, 2,
                                             bore_phi=s["bore"])
        return tod
    if kind == "angles":
        if "data" in s:
            return tod_core.beam_tod_angles(case["nside"], s["data"], *s["angles"], interp_mode=case["mode"],
                                            return_device=True)
        tod = torch.zeros((3, case["n"]), dtype=F64, device="cuda")
        interp = _native.BILINEAR if case["mode"] == "bilinear" else _native.NEAREST
        return gather_accum_angles(interp, s["vec"], *s["angles"], 0.0, 0.0, case["nside"], s["map"], s["vals"],
                                   tod, 1, 2)
    if kind == "day":
        return s["runner"].run(*s["scan"])
    if kind == "detectors":
        return s["batch"].run()
    if kind == "tail":
        return s["plan"].plain_tail(*s["angles"])
    if kind == "network":
        tod = torch.zeros((3, case["n"]), dtype=F64, device="cuda")
        return s["net"].accumulate(*s["angles"], tod)
    if kind == "training":
        return s["net"].loss_grad(s["x"], s["target"])
    return beam_cluster.cluster_beam_pixels(s["vec"], s["vals"], case["clusters"], tail_fraction=case["tail"],
                                            random_state=s["seed"], verbose=False)


# -- what one pass cannot do without ----------------------------------------------


def work(case):
    kind = case["kind"]
    if kind in ("network", "training"):
        f, h, d = case["n_freq"], case["width"], case["depth"]
        weights = 7 * f + 2 * f * h + (d - 1) * h * h + 3 * h
        passes = 1 if kind == "network" else 3
        row = 3 * 8 + 2 * 3 * 8 if kind == "network" else 7 * 4 + 3 * 4
        return {"bytes": case["n"] * row + weights * (2 if kind == "network" else 8),
                "flops": 2.0 * passes * weights * case["n"]}
    if kind == "cluster":
        pixels = _beam_of(case).S
        tail = 0.4 * pixels  # about the share of the pixels that holds a few percent of the weight
        return {"bytes": pixels * 16.0 + (pixels + case["clusters"]) * 16.0,
                "flops": 5.0 * tail * case["clusters"] * 20}
    rec = {"f64": 8, "f32": 4, "pf32": 4, "pbf16": 2}[case["map"]]
    if kind == "detectors":
        m = case["detectors"]
        ns = [case["n_min"] * (case["n_max"] / case["n_min"]) ** (d / max(1, m - 1)) for d in range(m)]
        samples = sum(ns)
        evals = sum(n * 1512 * ((25.0 + 10.0 * (1 - d / max(1, m - 1))) / 30.0) ** 2 for d, n in enumerate(ns))
        evals *= (case["beam_nside"] / 2048.0) ** 2
    elif kind == "tail":
        samples, evals = case["n"], case["n"] * 284000.0 * (case["beam_nside"] / 1024.0) ** 2
    else:
        samples = case["n"]
        evals = float(samples) * _beam_of(case).S
    comps = len(COMPS[case.get("comps", "IQU")])
    # the map's pixels that the footprints touch, at most the whole map
    touched = min(12.0 * case["nside"] ** 2, evals * 4)
    nearest = case.get("mode") == "nearest"
    # rotation 15, direction to ring and in-ring position 20, weights 12, mixing 2 per
    # neighbour and component
    flops = evals * ((45 + 2 * comps) if nearest else (47 + 8 * comps))
    return {"bytes": touched * comps * rec + samples * (12 + 8 * comps) + evals / samples * 16, "flops": flops}


# -- the same in 64 bits ------------------------------------------------------------


def _rodrigues(axis, angle):
    """(B, 3, 3) rotation by angle (B,) about unit axis (B, 3)."""
    c, s = torch.cos(angle)[:, None, None], torch.sin(angle)[:, None, None]
    x, y, z = axis.T
    o = torch.zeros_like(x)
    k = torch.stack([o, -z, y, z, o, -x, -y, x, o], -1).view(-1, 3, 3)
    eye = torch.eye(3, dtype=F64, device=axis.device)
    return eye * c + k * s + axis[:, :, None] * axis[:, None, :] * (1 - c)


def _pointing(theta, phi, psi):
    """Rotation matrices (B, 3, 3) and boresights (B, 3) for a beam centred on the pole."""
    th, ph, ps = (torch.as_tensor(a).to("cuda", F64) for a in (theta, phi, psi))
    t = torch.stack([torch.sin(th) * torch.cos(ph), torch.sin(th) * torch.sin(ph), torch.cos(th)], -1)
    zero = torch.zeros_like(ph)
    k = torch.stack([-torch.sin(ph), torch.cos(ph), zero], -1)
    north = torch.stack([torch.cos(ph) * torch.cos(th), torch.sin(ph) * torch.cos(th), -torch.sin(th)], -1)
    recentre = _rodrigues(k, th)
    w = recentre[:, :, 0]  # the pole's north (longitude 0: the x axis) carried along
    beta = torch.atan2((w * k).sum(-1), (w * north).sum(-1))
    return _rodrigues(t, ps - beta) @ recentre, t


def _ring(nside, ir):
    north, south = ir < nside, ir > 3 * nside
    i2 = 4 * nside - ir
    short = torch.where(north, ir, torch.where(south, i2, torch.full_like(ir, nside)))
    n = 4 * short
    npix = 12 * nside * nside
    belt = 2 * nside * (nside - 1) + (ir - nside) * 4 * nside
    first = torch.where(north, 2 * ir * (ir - 1), torch.where(south, npix - 2 * i2 * (i2 + 1), belt))
    shifted = north | south | ((ir - nside) % 2 == 0)
    dphi = 2 * PI / n.to(F64)
    cap = 1 - short.to(F64) ** 2 / (3.0 * nside * nside)
    z = torch.where(north, cap, torch.where(south, -cap, (2.0 / 3.0) * (2 - ir.to(F64) / nside)))
    return n, first, torch.where(shifted, 0.5 * dphi, torch.zeros_like(dphi)), dphi, z


def _spin2(z, phi, bore):
    zb, sb, pb = bore
    s = torch.sqrt(1 - z * z)
    half = 0.5 * (pb - phi)
    sh, ch = torch.sin(half), torch.cos(half)
    sd, cd, sh2 = 2 * sh * ch, 1 - 2 * sh * sh, sh * sh
    st2 = 0.25 * ((zb - z) ** 2 + (sb - s) ** 2)
    prod = s * sb
    num = 2 * sd * (zb + z) * (st2 + prod * sh2)
    den = 4 * st2 * (1 - st2) * cd - 4 * prod * zb * z * sh2 * sh2 + prod * sd * sd
    u = 1 / (num * num + den * den)
    return (den * den - num * num) * u, 2 * num * den * u


def _exact_tod(nside, vec, vals, rot, bores, planes, mode, spin2):
    """(C, B) TOD of one beam: planes (C, N), rot (B, 3, 3), boresights (B, 3)."""
    vec, vals = vec.to("cuda", F64), vals.to("cuda", F64)
    C, B, S = planes.shape[0], rot.shape[0], vec.shape[0]
    out = torch.zeros((C, B), dtype=F64, device="cuda")
    tile = min(S, 1 << 21)
    step = max(1, (1 << 22) // tile)
    for b0 in range(0, B, step):
        r, t = rot[b0:b0 + step], bores[b0:b0 + step]
        pb = torch.remainder(torch.atan2(t[:, 1], t[:, 0]), 2 * PI)[:, None]
        bore = (t[:, 2, None], torch.sqrt(1 - t[:, 2, None] ** 2), pb)
        for s0 in range(0, S, tile):
            v, w = vec[s0:s0 + tile], vals[s0:s0 + tile]
            x, y, z = (sum(r[:, i, j, None] * v[None, :, j] for j in range(3)) for i in range(3))
            phi = torch.remainder(torch.atan2(y, x), 2 * PI)
            z = z.clamp(-1, 1)
            polar = nside * torch.sqrt(3 * (1 - z.abs()))
            cap = torch.where(z < 0, 4 * nside - polar.long() - 1, polar.long())
            above = torch.where(z.abs() > 2.0 / 3.0, cap, (nside * (2 - 1.5 * z)).long())
            best, terms = None, None
            ta = None
            for g in (0, 1):
                n, first, phi0, dphi, zr = _ring(nside, above + g)
                tr = torch.acos(zr)
                if mode == "bilinear":
                    u = torch.remainder((phi - phi0) / dphi, n.to(F64))
                    if g == 0:
                        ta = tr
                        tb = torch.acos(_ring(nside, above + 1)[4])
                        wb = (torch.acos(z) - ta) / (tb - ta)
                    wr = wb if g else 1 - wb
                else:
                    u = torch.floor(phi * n.to(F64) / (2 * PI))
                i0 = torch.remainder(u.long(), n)
                frac = u - u.floor()
                for k in (0, 1):
                    ip = torch.remainder(i0 + k, n)
                    phc = phi0 + ip.to(F64) * dphi
                    if mode == "bilinear":
                        got = _terms(planes, first + ip, zr, phc, bore, spin2)
                        wk = wr * (frac if k else 1 - frac)
                        terms = [wk * q if terms is None else terms[c] + wk * q for c, q in enumerate(got)]
                    else:
                        cosd = torch.sqrt(x * x + y * y) * torch.sqrt(1 - zr * zr) * torch.cos(phi - phc) + z * zr
                        new = (cosd, first + ip, zr, phc)
                        best = new if best is None else tuple(torch.where(cosd > best[0], a, b)
                                                              for a, b in zip(new, best))
            if mode != "bilinear":
                terms = _terms(planes, best[1], best[2], best[3], bore, spin2)
            for c in range(C):
                out[c, b0:b0 + step] += (terms[c] * w).sum(-1)
    return out


def _terms(planes, pix, z, phi, bore, spin2):
    if not spin2:
        return [p[pix] for p in planes]
    c2, s2 = _spin2(z, phi, bore)
    q, u = planes[1][pix], planes[2][pix]
    return [planes[0][pix], q * c2 + u * s2, u * c2 - q * s2]


def _exact_network(net, x):
    feats = 2 * PI * (x.to(F64) @ net.freq.to(F64).T)
    a = torch.cat([torch.cos(feats), torch.sin(feats)], -1)
    layers = []
    for l in range(net.dims[2] + 1):
        w, b = (t.to(F64).clone().requires_grad_() for t in net.layer(l))
        layers += [w, b]
        a = a @ w.T + b
        if l < net.dims[2]:
            a = a * torch.sigmoid(a)
    return a, layers


def _exact_cluster(vec, vals, clusters, tail, seed):
    """Main lobe as it is, the weakest pixels holding `tail` of the weight as centroids of a
    weighted spherical k-means (k-means++ seeding, at most 150 rounds, 1e-5 rad)."""
    order = np.argsort(vals)
    m = min(max(1, int(np.searchsorted(np.cumsum(vals[order]), tail, side="right"))), len(vals) - 1)
    main, rest = order[m:], order[:m]
    v, w = vec[rest].astype(np.float64), vals[rest].astype(np.float64)
    k = min(clusters, m)
    if k < m:
        rng = np.random.default_rng(seed)
        cent, near = np.empty((k, 3)), None
        for j in range(k):
            p = w if j == 0 else w * np.maximum(1.0 - near, 0.0) ** 2
            c = np.cumsum(p)
            cent[j] = v[min(m - 1, int(np.searchsorted(c / c[-1], rng.random(), side="right")))]
            s = v @ cent[j]
            near = s if near is None else np.maximum(near, s)
        for _ in range(150):
            lab = np.argmax(v @ cent.T, axis=1)
            new = np.stack([np.bincount(lab, w * v[:, i], minlength=k) for i in range(3)], -1)
            empty = np.bincount(lab, w, minlength=k) == 0
            if empty.any():
                new[empty] = v[np.argmin((v @ cent.T).max(axis=1))]
            new /= np.linalg.norm(new, axis=1, keepdims=True)
            moved = np.clip((cent * new).sum(1), -1, 1).min()
            cent = new
            if moved > np.cos(1e-5):
                break
        lab = np.argmax(v @ cent.T, axis=1)
        v, w = cent, np.bincount(lab, w, minlength=k)
    out = np.concatenate([vals[main].astype(np.float64), w])
    return np.concatenate([vec[main].astype(np.float64), v]), out / out.sum(), None


def exact(case, seed):
    s = prepare(case, seed)
    kind = case["kind"]
    if kind in ("network", "training"):
        net = s["net"]
        if kind == "training":
            y, layers = _exact_network(net, s["x"])
            loss = ((y - s["target"].to(F64)) ** 2).mean()
            loss.backward()
            return loss.detach(), torch.cat([t.grad.reshape(-1) for t in layers])
        th, ph, ps = s["angles"]
        st = torch.sin(th)
        x = torch.stack([st * torch.cos(ph), st * torch.sin(ph), torch.cos(th), torch.cos(ps), torch.sin(ps),
                         torch.cos(2 * ps), torch.sin(2 * ps)], -1)
        scale, shift = (torch.from_numpy(a).cuda() for a in (net.scale, net.shift))
        with torch.no_grad():
            return torch.cat([(_exact_network(net, part)[0] * scale + shift).T for part in x.split(1 << 16)], 1)
    if kind == "cluster":
        return _exact_cluster(s["vec"], s["vals"], case["clusters"], case["tail"], seed)
    if kind == "detectors":
        planes = (s["map"] if torch.is_tensor(s["map"]) else s["map"].data[:, :3].T.contiguous()).to(F64)
        res = []
        for d in s["dets"]:
            rot, t = _pointing(d["theta"], d["phi"], d["psi"])
            res.append(_exact_tod(case["nside"], torch.from_numpy(d["vec_orig"]), torch.from_numpy(d["beam_vals"]),
                                  rot, t, planes, "bilinear", True))
        return res
    beam = s["beam"]
    vec, vals = torch.from_numpy(beam.vec_orig), torch.from_numpy(beam.beam_vals)
    if kind == "tail":
        rot, t = _pointing(*s["angles"])
        return _exact_tod(case["nside"], vec, vals, rot, t, s["sky"], "bilinear", True)
    mp = s["map"]
    planes = (mp if torch.is_tensor(mp) else mp.data[:, :3].T.contiguous()).to(F64)
    if kind == "fused":
        k, ca, sa, t, cp, sp = (a.to(F64) for a in s["params"][1:])
        rot = _rodrigues(t, torch.atan2(sp, cp)) @ _rodrigues(k, torch.atan2(sa, ca))
        return _exact_tod(case["nside"], vec, vals, rot, t, planes, "bilinear", True)
    if kind == "dropin":
        th, ph, _ = s["scan"]
        rv, th, ph, ps = (torch.from_numpy(np.asarray(a, np.float64)).cuda() for a in (s["rot"], th, ph, s["psis"]))
        angle = rv.norm(dim=1)
        t = torch.stack([torch.sin(th) * torch.cos(ph), torch.sin(th) * torch.sin(ph), torch.cos(th)], -1)
        rot = _rodrigues(t, ps) @ _rodrigues(rv / angle.clamp_min(1e-10)[:, None], angle)
        comps = COMPS[case["comps"]]
        tod = _exact_tod(case["nside"], vec, vals, rot, t, planes, case["mode"], len(comps) == 3)
        return {c: tod[i] for i, c in enumerate(comps)}
    rot, t = _pointing(*s["scan"])
    return _exact_tod(case["nside"], vec, vals, rot, t, planes, case["mode"], True)
