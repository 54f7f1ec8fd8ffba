"""Kernel-level entry points with the reference's Numba kernel ABI.

``gather_accum`` runs one fused gather/accumulate launch through
``todgpu_gather_accum``.  Arguments follow ``_gather_accum_fused_jit``
(tod_bilinear.py:205-222) and ``_gather_accum_nearest_jit``
(tod_nearest.py:21-38): beam-frame vectors, the six per-sample rotation
arrays, nside, the planar (C, N) map, beam weights, B, S, the (C, B) float64
output accumulated in place, and the Q/U component positions.

Inputs may be numpy arrays or torch tensors (CPU or CUDA).  When ``tod`` is a
numpy array it is copied to the GPU, accumulated there and copied back in
place, exactly like the reference mutates its argument; CUDA tensors are
updated in place without a host round trip.

Precision follows the parameter dtype, as it does in the reference (Numba
specialises the kernel on it): float32 parameters are combined with the
reference's float32/float64 operand typing (bit-parity form), float64
parameters give an all-float64 computation.
"""

from __future__ import annotations

import ctypes
import math
import weakref
from typing import NamedTuple

import numpy as np
import torch

from . import _native
from ._device import dtype_of, is_tensor, ptr, require_cuda, stream_handle, to_device

_PARAM_NAMES = ("vec_orig", "axes", "cos_a", "sin_a", "ax_pts", "cos_p", "sin_p")


def _param_dtype(arrs):
    dts = {dtype_of(a) for a in arrs}
    if dts == {np.dtype(np.float32)}:
        return np.float32
    if dts == {np.dtype(np.float64)}:
        return np.float64
    raise TypeError("vec_orig and the rotation parameter arrays must all be float32 "
                    f"(reference typing) or all float64; got {sorted(str(d) for d in dts)}")


def boresight_phi_host(ax_pts) -> np.ndarray:
    """atan2f(ax_pts[:,1], ax_pts[:,0]) with the host C library (float32),
    the boresight longitude the reference kernels compute
    (tod_bilinear.py:308, tod_nearest.py:87)."""
    if is_tensor(ax_pts):
        ax_pts = ax_pts.detach().to("cpu")
        a = np.ascontiguousarray(ax_pts.numpy(), dtype=np.float32)
    else:
        a = np.ascontiguousarray(np.asarray(ax_pts), dtype=np.float32)
    a = a.reshape(-1, 3)
    out = np.empty(a.shape[0], dtype=np.float32)
    _native.check(_native.lib().todgpu_boresight_phi_host(
        a.ctypes.data_as(ctypes.c_void_p), a.shape[0], out.ctypes.data_as(ctypes.c_void_p), 0))
    return out


_RING_TABLES = {}
_REACH_STEP = 1e-4  # ring tables are built for reaches rounded up to this step [rad]


_REACH = {}  # (tensor identity, version, nside) -> (reach, weak reference to the tensor)


def beam_reach(vec_orig, nside):
    """Angular radius [rad] that every stencil neighbour of the rotated beam
    stays within around the rotated beam centre: the beam's radius about its
    mean direction plus 3/nside (stencil reach) plus float32 slack.  The
    kernel derives the same bound from the beam on the device and uses the
    ring table's spin-2 slots only if the table covers it.  For a CUDA tensor
    the value is remembered (until the tensor changes or is freed), so repeated
    calls do not copy the beam back to the host."""
    key = None
    if is_tensor(vec_orig):
        key = (id(vec_orig), vec_orig.data_ptr(), vec_orig._version, tuple(vec_orig.shape), int(nside))
        hit = _REACH.get(key)
        if hit is not None and hit[1]() is vec_orig:
            return hit[0]
    r = _beam_reach(vec_orig, nside)
    if key is not None:
        try:
            _REACH[key] = (r, weakref.ref(vec_orig, lambda _r, k=key: _REACH.pop(k, None)))
        except TypeError:
            pass
    return r


def patch_order(vec_orig):
    """Order of a wide beam's pixels in which every run of ``_PIECE`` is a compact
    patch: the plane orthogonal to the beam's mean direction is halved along its
    longer side, at a multiple of ``_PIECE`` pixels, until a part is one run.  (Runs
    of the Morton order, and of the Hilbert curve, jump across a beam with holes:
    of the pieces of a 10-20 degree annulus 11% and 52% fit 3000 table slots, of
    these 87%.)
    For beams that run in pieces (:func:`gather_accum_angles`)."""
    v = vec_orig.detach().cpu().numpy() if is_tensor(vec_orig) else np.asarray(vec_orig)
    v = np.asarray(v, np.float64).reshape(-1, 3)
    if v.shape[0] <= _PIECE:
        return np.arange(v.shape[0], dtype=np.int64)
    # level by level, all parts at once (on the GPU where there is one)
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    xy = torch.from_numpy(np.stack(_tangent_plane(v))).to(dev)
    order = torch.arange(v.shape[0], device=dev)
    lens = [v.shape[0]]
    while max(lens) > _PIECE:
        size = torch.tensor(lens, device=dev)
        part = torch.repeat_interleave(torch.arange(len(lens), device=dev), size)
        q = xy[:, order]
        at = part.expand(2, -1)
        blank = torch.zeros((2, len(lens)), dtype=q.dtype, device=dev)
        wide = (blank.scatter_reduce(1, at, q, "amax", include_self=False)
                - blank.scatter_reduce(1, at, q, "amin", include_self=False)).argmax(dim=0)
        by = torch.argsort(torch.where(wide[part] == 0, q[0], q[1]), stable=True)
        order = order[by[torch.argsort(part[by], stable=True)]]
        halves = [((n + _PIECE - 1) // _PIECE // 2 * _PIECE, n) for n in lens]
        lens = [k for m, n in halves for k in ((m, n - m) if m > 0 else (n,))]
    return order.cpu().numpy()


def _beam_reach(vec_orig, nside):
    v = vec_orig.detach().cpu().numpy() if is_tensor(vec_orig) else np.asarray(vec_orig)
    v = np.asarray(v, np.float64).reshape(-1, 3)
    if v.shape[0] == 0:
        return 0.0
    c = v.sum(axis=0)
    nc = np.linalg.norm(c)
    c = c / nc if nc > 0 else np.array([0.0, 0.0, 1.0])
    vn = np.linalg.norm(v, axis=1)
    with np.errstate(invalid="ignore", divide="ignore"):
        d = np.where(vn > 0, (v @ c) / vn, -1.0)
    r = float(np.arccos(np.clip(d.min(), -1.0, 1.0)))
    return r + 3.0 / float(nside) + 2e-5


def _spread16(a):
    """The low 16 bits of a with a zero bit inserted after each."""
    a = a & 0xFFFF
    a = (a | (a << 8)) & 0x00FF00FF
    a = (a | (a << 4)) & 0x0F0F0F0F
    a = (a | (a << 2)) & 0x33333333
    a = (a | (a << 1)) & 0x55555555
    return a


def _tangent_plane(v):
    """Coordinates of unit vectors (n, 3) in the plane orthogonal to their mean."""
    c = v.sum(axis=0)
    nc = np.linalg.norm(c)
    c = c / nc if nc > 0 else np.array([0.0, 0.0, 1.0])
    a = np.zeros(3)
    a[int(np.argmin(np.abs(c)))] = 1.0
    e1 = np.cross(c, a)
    e1 /= np.linalg.norm(e1)
    return v @ e1, v @ np.cross(c, e1)


def beam_order(vec_orig):
    """Order of a beam's pixels that puts neighbours on the sky next to each
    other: the Morton (Z) order of their coordinates in the plane orthogonal to
    the beam's mean direction, 16 bits per axis.  Consecutive pixels go to
    neighbouring threads of a warp, whose stencils then share memory sectors
    of the map (a 30' beam pixelised at nside 4096 over an nside 2048 map made
    16 sectors per gather request in its ring order).  Only the order of the
    sum over beam pixels changes."""
    v = vec_orig.detach().cpu().numpy() if is_tensor(vec_orig) else np.asarray(vec_orig)
    v = np.asarray(v, np.float64).reshape(-1, 3)
    n = v.shape[0]
    if n < 2:
        return np.arange(n, dtype=np.int64)
    code = np.zeros(n, dtype=np.int64)
    for shift, x in enumerate(_tangent_plane(v)):
        lo, hi = x.min(), x.max()
        q = np.clip(((x - lo) / max(hi - lo, 1e-300) * 65535.0).astype(np.int64), 0, 65535)
        code |= _spread16(q) << shift
    return np.argsort(code, kind="stable")


_TABLE_REACH = {}  # data_ptr of a cached ring table -> the reach it was built for


def table_slots(nside, reach):
    """Upper bound of the map pixels in a footprint disc of radius ``reach`` [rad]
    away from the poles: per ring the disc's stretch with 2% margin, rounded up to
    2k + 1 pixels -- at most 1.02 x 3 (reach nside)^2 for the disc plus 3 per ring
    over at most 3 reach nside + 4 rings -- with 5% more and 32 to spare; 0 from
    0.05 rad.  A generous request: the gather lays its footprints out more tightly
    (:func:`footprint_slots`)."""
    r = float(reach)
    n = float(nside)
    if not r < 0.05:
        return 0
    x = r * n
    need = 1.02 * 3.0 * x * x + 3.0 * (3.0 * x + 4.0)
    return int(min(1 << 20, math.ceil(1.05 * need) + 32))


def footprint_slots(nside, reach):
    """Table slots of a footprint away from the poles as the gather lays it out:
    ``reach`` [rad] is a ring table's (the beam's radius plus 3/nside), x = radius
    times nside; per ring 2 H + 3 slots on average for a beam disc of half-width H
    pixels, each ring taking the disc's width one ring spacing nearer its centre --
    1.02 x 3 x^2 + 13.2 x + 12 -- with 3% more and 8 to spare (4 to 10% above what
    footprints of x = 3 to 60 fill).  ``reach`` may be an array."""
    x = np.maximum(0.0, np.asarray(reach, np.float64) - 3.0 / float(nside)) * float(nside)
    slots = np.minimum(1 << 20, np.ceil(1.03 * (1.02 * 3.0 * x * x + 13.2 * x + 12.0)) + 8)
    return int(slots) if slots.ndim == 0 else slots.astype(np.int64)


def table_slots_for(table, nside):
    """``footprint_slots`` for a table made by :func:`ring_table` (0, the
    library's default, for any other table or none)."""
    if table is None:
        return 0
    reach = _TABLE_REACH.get(table.data_ptr()) if is_tensor(table) else None
    return 0 if reach is None else footprint_slots(nside, reach)


def ring_table(nside, reach, device=None):
    """Device ring table for ``nside`` covering footprints up to ``reach``
    (built once and cached per device, nside and rounded reach)."""
    dev = device if device is not None else require_cuda()
    reach_q = min(np.pi, np.ceil(reach / _REACH_STEP) * _REACH_STEP)
    key = (dev.index if isinstance(dev, torch.device) else int(dev), int(nside), round(reach_q / _REACH_STEP))
    t = _RING_TABLES.get(key)
    if t is None:
        nbytes = int(_native.lib().todgpu_ring_table_bytes(int(nside)))
        if nbytes == 0:
            raise _native.TodGpuError(_native.ENSIDE, f"nside {nside} out of range")
        t = torch.empty(nbytes // 8, dtype=torch.float64, device=dev)
        _native.check(_native.lib().todgpu_ring_table_build(int(nside), float(reach_q), t.data_ptr(),
                                                            nbytes, stream_handle()))
        _RING_TABLES[key] = t
        _TABLE_REACH[t.data_ptr()] = float(reach_q)
    return t


# Evaluations (samples x beam pixels) from which a call makes its beam vectors
# planar: the copy takes some 5 us, interleaved vectors cost the gather a tenth
# of its time (three strided reads of 12 or 24 bytes a pixel) -- 40 us here.
_PLANAR_EVALS = 1 << 24


def planar_beam(vec, evals=None):
    """(vectors, flag) for a gather of ``evals`` evaluations over a CUDA (S, 3)
    tensor ``vec``: as they are if they are planar already (the (S, 3) view of a
    (3, S) tensor, as ``tod_core.device_beam`` keeps them), made planar for a
    large gather (``evals`` None: always), else interleaved.  flag is
    ``FLAG_BEAM_PLANAR`` or 0; the vectors' data pointer goes into vec_orig."""
    S = vec.shape[0]
    if S > 1 and vec.stride() == (1, S):
        return vec, _native.FLAG_BEAM_PLANAR
    if S > 1 and (evals is None or evals >= _PLANAR_EVALS):
        return vec.t().contiguous().t(), _native.FLAG_BEAM_PLANAR
    return vec.contiguous(), 0


def resident_beam(vec_orig, np_dtype, device):
    """``vec_orig`` itself when it is a (S, 3) tensor of ``np_dtype`` on
    ``device`` -- in any strides, for :func:`planar_beam` -- else None: anything
    else (another GPU's tensor too) goes through ``to_device``."""
    if (is_tensor(vec_orig) and vec_orig.device == device and dtype_of(vec_orig) == np.dtype(np_dtype)
            and vec_orig.dim() == 2 and vec_orig.shape[1] == 3):
        return vec_orig
    return None


def _row_stride(t):
    """Row stride of a (rows, n) tensor with unit column stride; a single
    row's stride is free in torch (a ``[None, :]`` view may carry 0), so it
    is taken as n."""
    return t.stride(0) if t.shape[0] > 1 else t.shape[1]


def _set_map(a, mp):
    if isinstance(mp, PackedMap):
        a.map_dtype = mp.map_dtype
        a.map = mp.data.data_ptr()
        a.map_stride = mp.npix
    else:
        a.map_dtype = _native.F32 if mp.dtype == torch.float32 else _native.F64
        a.map = mp.data_ptr()
        a.map_stride = _row_stride(mp)


def _ncomp(mp):
    return mp.C if isinstance(mp, PackedMap) else mp.shape[0]


def make_args(interp, nside, B, S, C, c_q, c_u, params, pdt, bore_phi, beam, mp, tod,
              err=None, flags=0, table=None):
    a = _native.GatherArgs()
    a.abi_version = _native.ABI_VERSION
    a.interp = interp
    a.nside = int(nside)
    a.B = int(B)
    a.S = int(S)
    a.C = int(C)
    a.c_q = int(c_q)
    a.c_u = int(c_u)
    a.params_dtype = _native.F32 if pdt == np.float32 else _native.F64
    _set_map(a, mp)
    (a.vec_orig, a.axes, a.cos_a, a.sin_a, a.ax_pts, a.cos_p, a.sin_p) = [ptr(t) for t in params]
    a.bore_phi = ptr(bore_phi)
    a.beam_vals = ptr(beam)
    a.tod = ptr(tod)
    a.tod_stride = _row_stride(tod)
    a.err_count = ptr(err)
    a.flags = int(flags)
    a.ring_table = ptr(table)
    a.tab_slots = table_slots_for(table, nside)
    return a


class PackedMap:
    """A map with one record of 4 components per pixel: float32 (16 B) or
    bfloat16 (8 B) for the precision form, float64 (32 B) for the float64
    path with a pixel's components side by side (same results as the planar
    float64 map).  Built by :func:`pack_map`."""

    def __init__(self, data: torch.Tensor, C: int, kind: str):
        self.data = data
        self.C = int(C)
        self.kind = kind  # "f32" or "bf16"

    @property
    def map_dtype(self):
        return {"f32": _native.PACKED_F32, "bf16": _native.PACKED_BF16, "f64": _native.PACKED_F64}[self.kind]

    @property
    def npix(self):
        return self.data.shape[0]

    @property
    def device(self):
        return self.data.device


def pack_map(mp_stacked, kind="f32"):
    """Pack a planar (C, N) map (numpy or torch, float32/float64, C <= 4) into
    per-pixel records on the GPU (todgpu_pack_map): "f32" or "bf16" for the
    precision form, "f64" for the float64 path."""
    if kind not in ("f32", "bf16", "f64"):
        raise ValueError("kind must be 'f32', 'bf16' or 'f64'")
    mp = _map_tensor(mp_stacked)
    C, N = mp.shape
    if C > 4:
        raise ValueError("at most 4 components per record")
    dt = {"f32": torch.float32, "bf16": torch.bfloat16, "f64": torch.float64}[kind]
    out = torch.empty((N, 4), dtype=dt, device=mp.device)
    _native.check(_native.lib().todgpu_pack_map(
        mp.data_ptr(), _native.F32 if mp.dtype == torch.float32 else _native.F64, C, N, _row_stride(mp),
        {"f32": _native.PACKED_F32, "bf16": _native.PACKED_BF16, "f64": _native.PACKED_F64}[kind], out.data_ptr(),
        stream_handle()))
    return PackedMap(out, C, kind)


def _map_tensor(mp_stacked):
    if isinstance(mp_stacked, PackedMap):
        return mp_stacked
    dt = dtype_of(mp_stacked)
    if dt not in (np.dtype(np.float32), np.dtype(np.float64)):
        raise TypeError(f"mp_stacked must be float32 or float64, got {dt}")
    mp = to_device(mp_stacked, dt.type)
    if mp.dim() != 2:
        raise ValueError("mp_stacked must be a (C, N) array")
    return mp


def gather_accum(interp, vec_orig, axes, cos_a, sin_a, ax_pts, cos_p, sin_p, nside, mp_stacked,
                 beam_vals, B, S, tod, c_q=-1, c_u=-1, bore_phi=None, err_count=None, flags=0):
    """One fused launch; see the module docstring.  Returns ``tod``.

    ``err_count``: optional int64 CUDA tensor of one element that receives the
    number of (sample, beam pixel) terms skipped because a stencil pixel fell
    outside the map (only possible for non-finite pointing).
    ``flags``: ``_native.FLAG_NO_TABLES`` evaluates every ring quantity and
    spin-2 angle directly instead of from the per-sample footprint tables
    (identical results; for testing)."""
    dev = require_cuda()
    B = int(B)
    S = int(S)
    nside = int(nside)
    raw = (vec_orig, axes, cos_a, sin_a, ax_pts, cos_p, sin_p)
    pdt = _param_dtype(raw)
    shapes = [(S, 3), (B, 3), (B,), (B,), (B, 3), (B,), (B,)]
    given = resident_beam(vec_orig, pdt, dev)
    if given is None or given.shape[0] != S:
        given = to_device(vec_orig, pdt, (S, 3))
    vec, planar = planar_beam(given, B * S)
    params = [vec] + [to_device(x, pdt, sh) for x, sh in zip(raw[1:], shapes[1:])]
    if dtype_of(beam_vals) != np.dtype(np.float32):
        raise TypeError("beam_vals must be float32 (the reference casts beam weights to float32)")
    beam = to_device(beam_vals, np.float32, (S,))
    mp = _map_tensor(mp_stacked)
    C = _ncomp(mp)
    if pdt == np.float32 and bore_phi is None and B > 0:
        bore_phi = boresight_phi_host(ax_pts if not is_tensor(ax_pts) else params[4])
    bphi = to_device(bore_phi, np.float32, (B,)) if (bore_phi is not None and pdt == np.float32) else None

    host_tod = None
    if is_tensor(tod) and tod.is_cuda:
        if tod.dtype != torch.float64 or tod.dim() != 2 or tod.stride(1) != 1:
            raise ValueError("tod must be a float64 (C, B) tensor with unit stride along B")
        dtod = tod
    else:
        host_tod = tod
        arr = tod.numpy() if is_tensor(tod) else tod
        if arr.dtype != np.float64 or arr.ndim != 2:
            raise ValueError("tod must be a float64 (C, B) array")
        dtod = torch.from_numpy(np.ascontiguousarray(arr)).to(params[0].device)
    if tuple(dtod.shape) != (C, B):
        raise ValueError(f"tod has shape {tuple(dtod.shape)}, expected {(C, B)}")

    table = None
    if not flags & _native.FLAG_NO_TABLES and B > 0 and S > 0:
        table = ring_table(nside, beam_reach(vec_orig, nside), params[0].device)
    args = make_args(interp, nside, B, S, C, c_q, c_u, params, pdt, bphi, beam, mp, dtod,
                     err_count, flags | planar, table)
    _native.check(_native.lib().todgpu_gather_accum(ctypes.byref(args), stream_handle()))
    if host_tod is not None:
        res = dtod.cpu().numpy()
        if is_tensor(host_tod):
            host_tod.copy_(torch.from_numpy(res))
        else:
            host_tod[...] = res
    return tod


def bilinear_stencils(vec_orig, axes, cos_a, sin_a, ax_pts, cos_p, sin_p, nside, B, S):
    """Per-(b, s) bilinear pixels (4, B*S) int64 and weights (4, B*S) float64 of
    the fused path, as CUDA tensors."""
    require_cuda()
    B = int(B)
    S = int(S)
    raw = (vec_orig, axes, cos_a, sin_a, ax_pts, cos_p, sin_p)
    pdt = _param_dtype(raw)
    shapes = [(S, 3), (B, 3), (B,), (B,), (B, 3), (B,), (B,)]
    params = [to_device(x, pdt, sh) for x, sh in zip(raw, shapes)]
    dev = params[0].device
    pix = torch.empty((4, B * S), dtype=torch.int64, device=dev)
    wgt = torch.empty((4, B * S), dtype=torch.float64, device=dev)
    a = _native.GatherArgs()
    a.abi_version = _native.ABI_VERSION
    a.nside = int(nside)
    a.B = B
    a.S = S
    a.params_dtype = _native.F32 if pdt == np.float32 else _native.F64
    (a.vec_orig, a.axes, a.cos_a, a.sin_a, a.ax_pts, a.cos_p, a.sin_p) = [ptr(t) for t in params]
    _native.check(_native.lib().todgpu_bilinear_stencils(ctypes.byref(a), pix.data_ptr(),
                                                         wgt.data_ptr(), stream_handle()))
    return pix, wgt


def beam_center_angles(ra, dec, center_idx=None):
    """(phi_c, theta_c) of the beam centre: the grid centre by default, as
    tod_rotations.py:251-261 chooses it."""
    ra = np.asarray(ra)
    dec = np.asarray(dec)
    if center_idx is None:
        center_idx = (ra.shape[0] // 2, ra.shape[1] // 2)
    return float(ra[center_idx]), float(np.pi / 2 - dec[center_idx])


def _angles_on_device(theta, phi, psi):
    adt = dtype_of(theta)
    adt = np.float32 if adt == np.dtype(np.float32) else np.float64
    th = to_device(theta, adt).reshape(-1)
    ph = to_device(phi, adt).reshape(-1)
    ps = to_device(psi, adt).reshape(-1)
    if ph.shape[0] != th.shape[0] or ps.shape[0] != th.shape[0]:
        raise ValueError("theta, phi and psi must have the same length")
    return adt, th, ph, ps


def pointing_buffers(B, device):
    """Uninitialised float64 (axes (B, 3), cos_a, sin_a, ax_pts (B, 3), cos_p,
    sin_p) for :func:`pointing_params`."""
    axes = torch.empty((B, 3), dtype=torch.float64, device=device)
    pts = torch.empty((B, 3), dtype=torch.float64, device=device)
    cos_a, sin_a, cos_p, sin_p = (torch.empty(B, dtype=torch.float64, device=device) for _ in range(4))
    return axes, cos_a, sin_a, pts, cos_p, sin_p


def pointing_params(theta, phi, psi, center_phi, center_theta, out=None):
    """Float64 rotation parameters (axes (B, 3), cos_a, sin_a, ax_pts (B, 3),
    cos_p, sin_p) of every sample, derived on the device from the pointing
    angles and the beam centre -- the reference's
    precompute_rotation_vector_batch + _rotation_params
    (tod_rotations.py:219-333) in float64, one thread per sample.  A float64
    gather on them equals the angles-mode gather bit for bit.  ``out``: six
    contiguous float64 CUDA tensors of at least B samples to fill (e.g. from
    :func:`pointing_buffers`); returned as given."""
    require_cuda()
    adt, th, ph, ps = _angles_on_device(theta, phi, psi)
    B = th.shape[0]
    if out is None:
        out = pointing_buffers(B, th.device)
    elif len(out) != 6 or any(not (is_tensor(t) and t.is_cuda and t.dtype == torch.float64 and t.is_contiguous()
                                   and t.shape[0] >= B) for t in out):
        raise ValueError("out must be six contiguous float64 CUDA tensors of at least B samples")
    axes, cos_a, sin_a, pts, cos_p, sin_p = out
    _native.check(_native.lib().todgpu_pointing_params(
        th.data_ptr(), ph.data_ptr(), ps.data_ptr(), _native.F32 if adt == np.float32 else _native.F64, B,
        float(center_phi), float(center_theta), axes.data_ptr(), cos_a.data_ptr(), sin_a.data_ptr(),
        pts.data_ptr(), cos_p.data_ptr(), sin_p.data_ptr(), stream_handle()))
    return out


# Beams of more pixels than this run as pieces of _PIECE consecutive pixels, each
# a job of its own of the batched gather with its own footprint.
_PIECE_MIN = 16384
_PIECE = 1024
# Largest footprint a piece gets a table for: three CTAs of 256 threads share an SM up
# to there (284k pixels of an annulus, 301 samples: 4.72 ms; 5.06 at 3000, 5.11 at
# 4400, 6.8 at 8192, where one CTA has the SM; pieces of 512 or 2048 pixels 5.9, 6.7).
_PIECE_SLOTS = 2600
# Wider pieces ask for a window without a table, as the gather's rule gives it: for more
# slots than four times their pixels.  (With neither, every pixel went through the direct
# evaluation: 60,000 pixels of 3 to 12 degrees, nside 1024, 8000 samples, I alone, nearest
# 17.7 ms, now 7.4.)  Up to the slots of 700 window rings, which three CTAs of 256 threads
# hold, and where they are tiles enough for the launch of their own that the library then
# makes (16 an SM): fewer share the others' launch, where a window gains them nothing
# (71,000 pixels, nside 512, 80 samples: 512 us, 560 with the windows).
_PIECE_NO_TABLE = 4 * _PIECE + 1
_PIECE_WINDOW = 170_000
_PIECE_OWN_LAUNCH = 16 * 148
_PIECE_TILE = 16  # samples per work tile of a piece's job
_PIECE_SCRATCH = 1 << 28  # bytes of the pieces' own outputs: 116,000 samples of 96 pieces, I, Q and U


class PiecePlan(NamedTuple):
    """:func:`piece_footprints` of a beam of S pixels over a map of one nside."""

    slots: np.ndarray  # requested slots of every piece
    reach: float       # the largest footprint with a table [rad]
    S: int
    nside: int
    window_reach: float  # the largest with a window [rad]


def _check_plan(plan, S, nside):
    """A plan made for another beam would leave out pixels or read past the beam's."""
    if not isinstance(plan, PiecePlan) or plan.S != S or plan.nside != int(nside) or len(plan.slots) != -(-S // _PIECE):
        raise ValueError(f"pieces must be piece_footprints of this beam ({S} pixels) and nside {int(nside)}")
    return plan


def piece_footprints(vec, nside):
    """:class:`PiecePlan` of a wide beam, a CUDA (S, 3) tensor: the angle from a
    piece's mean direction to its farthest pixel, found on the device; pieces too
    wide for a table ask for more slots than one may have (a window alone), and those too
    wide for that for 2.  A plan that a program keeps with its beam
    (``gather_accum_angles(pieces=...)``)."""
    S = vec.shape[0]
    n = (S + _PIECE - 1) // _PIECE
    at = torch.arange(n * _PIECE, device=vec.device).clamp_(max=S - 1)
    p = vec[at].view(n, _PIECE, 3)
    c = torch.nn.functional.normalize(p.sum(dim=1), dim=1)
    low = torch.einsum("nkc,nc->nk", torch.nn.functional.normalize(p, dim=2), c).amin(dim=1)
    r = np.arccos(np.clip(low.cpu().numpy(), -1.0, 1.0))
    r = np.where(np.isfinite(r), r, np.pi) + 3.0 / float(nside) + 2e-5
    slots = footprint_slots(nside, r)
    tabled, window = slots <= _PIECE_SLOTS, slots <= _PIECE_WINDOW
    slots = np.where(tabled, slots, np.where(window, np.maximum(slots, _PIECE_NO_TABLE), 2))
    most = lambda which: float(r[which].max()) if which.any() else 0.0
    return PiecePlan(slots.astype(np.int32), most(tabled), S, int(nside), most(window))


def _gather_pieces(args, vec, beam, nside, tod, pieces):
    """The gather of ``args`` (all but its beam set) over a wide beam, in pieces:
    launches of up to 96 pieces into outputs of their own, added into ``tod`` in
    order.  A far-sidelobe beam's footprint holds 1e5 to 1e6 map pixels, a
    piece's a patch that fits a table in shared memory; as jobs the pieces also
    spread over the GPU where the samples alone would not.  Pieces of like
    footprints share a launch, whose table is sized for the largest.  Long batches
    run in blocks of samples, so the pieces' outputs stay within _PIECE_SCRATCH (the
    sums are a sample's own: the same in any block)."""
    S = vec.shape[0]
    plan = pieces if pieces is not None else piece_footprints(vec, nside)
    C, B = tod.shape
    most = min(96, len(plan.slots))
    block = min(B, max(_PIECE_TILE, _PIECE_SCRATCH // (most * C * 8) // _PIECE_TILE * _PIECE_TILE))
    wide = plan.slots >= _PIECE_NO_TABLE
    own = min(96, int(wide.sum())) * -(-block // _PIECE_TILE) >= _PIECE_OWN_LAUNCH
    slots, reach = (plan.slots, plan.window_reach) if own else (np.where(wide, 2, plan.slots), plan.reach)
    flat = vec.contiguous()  # (pieces of a planar beam are not planar beams)
    args.flags &= ~_native.FLAG_BEAM_PLANAR
    if not args.flags & _native.FLAG_NO_TABLES and reach > 0.0:
        args.ring_table = ring_table(nside, reach, vec.device).data_ptr()
    elif not args.flags & _native.FLAG_NO_TABLES:
        args.ring_table = ring_table(nside, 3.0 / float(nside), vec.device).data_ptr()
    part = torch.empty((most, C, block), dtype=torch.float64, device=vec.device)
    size = ctypes.sizeof(_native.GatherArgs)
    jobs = np.tile(np.frombuffer(bytes(args), np.uint8), (len(slots), 1))
    field = lambda name, dt: np.ndarray(len(slots), dt, jobs, getattr(_native.GatherArgs, name).offset, (size,))
    first = np.arange(len(slots), dtype=np.int64) * _PIECE
    field("vec_orig", np.uint64)[:] = flat.data_ptr() + first * 24
    field("beam_vals", np.uint64)[:] = beam.data_ptr() + first * 4
    field("S", np.int64)[:] = np.minimum(_PIECE, S - first)
    field("tab_slots", np.int32)[:] = slots
    # (those without a table first: the longest)
    jobs = np.ascontiguousarray(jobs[np.argsort(np.where(slots <= _PIECE_SLOTS, slots, 0), kind="stable")])
    for b0 in range(0, B, block):
        nb = min(block, B - b0)
        for name in ("axes", "cos_a", "sin_a", "ax_pts", "cos_p", "sin_p"):
            field(name, np.uint64)[:] = getattr(args, name) + 8 * b0 * (3 if name in ("axes", "ax_pts") else 1)
        field("B", np.int64)[:] = nb
        field("tod", np.uint64)[:] = part.data_ptr() + (np.arange(len(slots)) % most) * (C * nb * 8)
        field("tod_stride", np.int64)[:] = nb
        for j0 in range(0, len(slots), most):
            n = min(most, len(slots) - j0)
            sums = part.view(-1)[:n * C * nb].view(n, C, nb)
            sums.zero_()
            _native.check(_native.lib().todgpu_gather_accum_batched(
                ctypes.cast(jobs[j0:].ctypes.data, ctypes.POINTER(_native.GatherArgs)), n, _PIECE_TILE,
                stream_handle()))
            tod[:, b0:b0 + nb] += sums.sum(dim=0)


def gather_accum_angles(interp, vec_orig, theta, phi, psi, center_phi, center_theta, nside,
                        mp_stacked, beam_vals, tod, c_q=-1, c_u=-1, err_count=None, flags=0,
                        static_table=False, precompute=True, pieces=None):
    """One fused launch with the pointing given as angles: every CTA derives
    the sample's rotation on the device in float64 from (theta, phi, psi) and
    the beam centre (no float32 parameter rounding).  ``tod`` must be a float64
    (C, B) CUDA tensor; it is accumulated in place.  ``theta, phi, psi`` may be
    float32 or float64 (a float32 scan is widened exactly on the device).

    ``precompute`` (default) derives the rotations first with
    :func:`pointing_params` (one thread per sample, 80 bytes of scratch per
    sample) and runs the gather in its float64-parameter mode: the same TOD bit
    for bit, with the per-sample rotation taken off the gather's critical path.
    ``precompute=False`` (and ``static_table=True``, which allocates nothing)
    derive the rotation inside the gather.

    ``pieces``: :func:`piece_footprints` of a beam of more than 16384 pixels, for a
    program that keeps it (found in each call otherwise); a plan of another beam
    size or nside is a ValueError."""
    # (a copy or view of a resident beam would be another tensor to beam_reach)
    given = resident_beam(vec_orig, np.float64, require_cuda())
    if given is None:
        given = to_device(vec_orig, np.float64).reshape(-1, 3)
    S = given.shape[0]
    if pieces is not None:
        _check_plan(pieces, S, nside)
    adt, th, ph, ps = _angles_on_device(theta, phi, psi)
    B = th.shape[0]
    vec, planar = planar_beam(given, B * S)
    rot = pointing_params(th, ph, ps, center_phi, center_theta) if precompute and not static_table else None
    beam = to_device(beam_vals, np.float32, (S,))
    mp = _map_tensor(mp_stacked)
    C = _ncomp(mp)
    if not (is_tensor(tod) and tod.is_cuda and tod.dtype == torch.float64 and tod.dim() == 2
            and tod.stride(1) == 1 and tuple(tod.shape) == (C, B)):
        raise ValueError(f"tod must be a float64 CUDA tensor of shape {(C, B)} with unit stride")
    a = _native.GatherArgs()
    a.abi_version = _native.ABI_VERSION
    a.interp = interp
    a.nside = int(nside)
    a.B = B
    a.S = S
    a.C = C
    a.c_q = int(c_q)
    a.c_u = int(c_u)
    _set_map(a, mp)
    a.vec_orig = vec.data_ptr()
    if rot is not None:
        a.params_dtype = _native.F64
        (a.axes, a.cos_a, a.sin_a, a.ax_pts, a.cos_p, a.sin_p) = [t.data_ptr() for t in rot]
    else:
        a.params_dtype = _native.ANGLES
        a.theta, a.phi, a.psi = th.data_ptr(), ph.data_ptr(), ps.data_ptr()
        a.angles_dtype = _native.F32 if adt == np.float32 else _native.F64
        a.center_phi = float(center_phi)
        a.center_theta = float(center_theta)
    a.beam_vals = beam.data_ptr()
    a.tod = tod.data_ptr()
    a.tod_stride = _row_stride(tod)
    a.err_count = ptr(err_count)
    a.flags = int(flags) | planar
    lib = _native.lib()
    if S > _PIECE_MIN and rot is not None and B > 0 and not (isinstance(mp, PackedMap) and mp.kind != "f64"):
        _gather_pieces(a, given, beam, nside, tod, pieces)
        return tod
    if static_table:
        _native.check(lib.todgpu_gather_accum_static(ctypes.byref(a), stream_handle()))
        return tod
    if not flags & _native.FLAG_NO_TABLES and B > 0 and S > 0:
        table = ring_table(nside, beam_reach(given, nside), vec.device)
        a.ring_table = table.data_ptr()
        a.tab_slots = table_slots_for(table, nside)
    _native.check(lib.todgpu_gather_accum(ctypes.byref(a), stream_handle()))
    return tod
