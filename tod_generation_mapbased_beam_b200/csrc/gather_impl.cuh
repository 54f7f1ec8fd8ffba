// gather_impl.cuh -- fused beam-convolution TOD kernels for B200 (sm_100a):
// device code and launch templates, shared by the translation units that
// instantiate them (gather_map_*.cu, one per map element type) and by the C
// ABI (tod_api.cu).
//
// Work decomposition ("footprint" kernel): a persistent grid of CTAs (128 or
// 256 threads) walks the samples; a CTA takes one sample
// at a time and
//   1. has its rotation, footprint centre and range of RING rings prepared, for
//      sixteen samples at a time by sixteen lanes of one warp (prepare_sample);
//   2. lays out the window of rings the footprint (beam radius + stencil
//      reach) can touch, each ring's stretch of the footprint disc and the
//      ring in the sample's own longitude frame (footprint_window);
//   3. evaluates the map once per footprint pixel into shared memory: I, and Q
//      and U turned into the boresight's frame (fill_table; a map pixel is
//      shared by ~10 (beam pixel, neighbour) pairs of a sample) -- where that
//      pays (table_pays); other launches are kernels of their own, without it;
//   4. strides its threads over the beam pixels: rotation into the frame ->
//      longitude by a short series -> ring and in-ring position from the window
//      -> weighted sum of four table entries, or of four map pixels
//      (bilinear_loop), or the nearest one (nearest_loop);
//   5. reduces the per-lane sums (256 summation lanes in either CTA shape) in a
//      fixed order and adds them into tod[c, b] (one writer per sample: no
//      atomics, bit-reproducible runs, the same TOD in every shape).
// A pixel that the window or the table does not hold takes bilinear_direct /
// nearest_exact, which do the same operations on the same values without
// them: windows and tables only decide speed, never results.
//
// Compiled with -fmad=false: the pixel decisions and the FP64 accumulation
// reproduce the reference's uncontracted arithmetic.
#pragma once

#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <climits>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <mutex>
#include <string>
#include <thread>
#include <type_traits>
#include <vector>

#include "healpix_ring.cuh"
#include "todgpu.h"

namespace todgpu {

// Rings per footprint window: of a call that names no footprint, of a call's
// request at most, and of a beam in chunks without a table (three CTAs of 256 threads
// an SM still hold that window).
constexpr int kRingCap = 192, kRingMax = 2048, kRingChunk = 448;
constexpr int kTabCapDefault = 2048;  // table slots per sample when the caller asks for none
constexpr long long kMaxNside = 16384;
// Summation lanes of the gather: the beam pixels of a sample are summed in
// this many strided partial sums, combined in a fixed order whatever the CTA's
// thread count, so CTAs of 128 and 256 threads give the same TOD bit for bit.
constexpr int kSumLanes = 256;
// Registers per thread and the threads that then fit an SM (in CTAs of 128).
// Measured at 64 / 72 / 80 / 96: the 30' float64 beam 2.59 / 2.57 / 2.59 / 2.65
// ms, detectors over a float32 map 4.69 / 4.51 / 4.44 / 5.2 ms, packed float32
// records 1.91 / 1.97 / 1.94 / 2.5 ms: the pixel loops spill a few registers
// below 72, and above it too few warps are left.
constexpr int kRegs = 72;
constexpr int kThreadsSM = 65536 / kRegs / 128 * 128;

// Bytes of a window's rings and their slot ends.
__host__ __device__ constexpr size_t window_bytes(int ring_cap) {
  return (84 * (size_t)ring_cap + 15) & ~size_t(15);
}
// Bytes of the slot -> ring index of a table (one entry per 32 slots).
__host__ __device__ constexpr size_t ring_of_bytes(int tab_cap) {
  return (2 * ((size_t)tab_cap / 32 + 1) + 15) & ~size_t(15);
}

// Message of the calling thread's last failure (defined in tod_api.cu).
extern thread_local std::string g_last_error;

inline int fail(int code, const std::string& msg) {
  g_last_error = msg;
  return code;
}

inline int cuda_fail(cudaError_t e, const char* what) {
  return fail(TODGPU_ECUDA, std::string(what) + ": " + cudaGetErrorString(e));
}

struct KArgs {
  long long nside, npix, B, S;
  int C, c_q, c_u;
  int tab_cap;               // table slots in shared memory
  int tab_req;               // slots the caller asks for (0: default)
  const void* ring_table;    // RingRec[4 nside] or nullptr
  const void* vec;
  const void* axes;
  const void* cos_a;
  const void* sin_a;
  const void* pts;
  const void* cos_p;
  const void* sin_p;
  const float* bore_phi;
  const void* theta;         // pointing angles (angles mode)
  const void* phi;
  const void* psi;
  int angles_f32;            // angles are float32 (else float64)
  double cvx, cvy, cvz;      // beam-centre unit vector (angles mode)
  double cnx, cny, cnz;      // its local north
  const float* beam;
  const void* map;
  long long map_stride;
  double* tod;
  long long tod_stride;
  unsigned long long* err;
  int flags_wide;            // the caller asks for CTAs of at least 256 threads
  int ring_cap;              // window rings the launch has room for
  int vec_ss;                // beam vectors: component i of pixel s at vec[s vec_ss + i vec_si]
  long long vec_si;
};

// Pointing modes of the per-sample rotation.
constexpr int kParamsRef32 = 0;  // reference float32 parameter arrays
constexpr int kParamsF64 = 1;    // float64 parameter arrays
constexpr int kAngles = 2;       // (theta, phi, psi) + beam centre, derived on the device

__host__ __device__ constexpr bool f64_params(int pm) { return pm == kParamsF64; }

template <int PM>
__device__ __forceinline__ double angle_at(const KArgs& a, const void* p, long long b) {
  return a.angles_f32 ? (double)static_cast<const float*>(p)[b] : static_cast<const double*>(p)[b];
}

// Rotation from pointing angles (theta, phi, psi), in float64: the Rodrigues
// vector taking the beam centre c to the boresight t and the polarisation
// offset beta (tod_rotations.py:219-303), then the parameters of
// tod_rotations.py:306-333 without any float32 rounding.
__device__ __forceinline__ SampleRot rot_from_angle_values(const KArgs& a, double th, double ph, double ps) {
  double st, ct, sp, cp;
  sincos(th, &st, &ct);
  sincos(ph, &sp, &cp);
  const double tx = st * cp, ty = st * sp, tz = ct;    // boresight
  const double nx = cp * ct, ny = sp * ct, nz = -st;   // its north
  const double ex = -sp, ey = cp;                      // its east
  double kx = a.cvy * tz - a.cvz * ty;
  double ky = a.cvz * tx - a.cvx * tz;
  double kz = a.cvx * ty - a.cvy * tx;
  const double kn = sqrt((kx * kx + ky * ky) + kz * kz);
  if (kn > 1e-10) {
    kx /= kn;
    ky /= kn;
    kz /= kn;
  } else {
    kx = ky = kz = 0.0;
  }
  const double ang = acos(clamp1(a.cvx * tx + a.cvy * ty + a.cvz * tz));
  double sa, ca;
  sincos(ang, &sa, &ca);
  const double dkn = kx * a.cnx + ky * a.cny + kz * a.cnz;
  const double oma = 1.0 - ca;
  const double wx = a.cnx * ca + (ky * a.cnz - kz * a.cny) * sa + kx * dkn * oma;
  const double wy = a.cny * ca + (kz * a.cnx - kx * a.cnz) * sa + ky * dkn * oma;
  const double wz = a.cnz * ca + (kx * a.cny - ky * a.cnx) * sa + kz * dkn * oma;
  double beta = atan2(wx * ex + wy * ey + wz * 0.0, wx * nx + wy * ny + wz * nz);
  if (beta < 0.0) beta += kTwoPi;
  SampleRot r;
  r.kx = kx;
  r.ky = ky;
  r.kz = kz;
  r.ca = ca;
  r.sa = sa;
  r.px = tx;
  r.py = ty;
  r.pz = tz;
  sincos(ps - beta, &r.sp, &r.cp);
  return r;
}

__device__ __forceinline__ SampleRot rot_from_angles(const KArgs& a, long long b) {
  return rot_from_angle_values(a, angle_at<kAngles>(a, a.theta, b), angle_at<kAngles>(a, a.phi, b),
                               angle_at<kAngles>(a, a.psi, b));
}

// The per-sample pointing inputs as numbered fields.  Reference float32
// parameters: 0-2 axes, 3 cos_a, 4 sin_a, 5-7 ax_pts, 8 cos_p, 9 sin_p, 10 the
// boresight longitude (when given); float64 parameters: fields 0-9 as
// doubles; angles: 0 theta, 1 phi, 2 psi.  field_ptr gives a field's address
// (nullptr when absent).
template <int PM>
__device__ __forceinline__ const void* field_ptr(const KArgs& a, long long b, int i) {
  if constexpr (PM == kAngles) {
    const void* p = i == 0 ? a.theta : (i == 1 ? a.phi : a.psi);
    return a.angles_f32 ? (const void*)(static_cast<const float*>(p) + b)
                        : (const void*)(static_cast<const double*>(p) + b);
  } else {
    using T = typename std::conditional<PM == kParamsRef32, float, double>::type;
    if (i < 3) return static_cast<const T*>(a.axes) + 3 * b + i;
    if (i == 3) return static_cast<const T*>(a.cos_a) + b;
    if (i == 4) return static_cast<const T*>(a.sin_a) + b;
    if (i < 8) return static_cast<const T*>(a.pts) + 3 * b + (i - 5);
    if (i == 8) return static_cast<const T*>(a.cos_p) + b;
    if (i == 9) return static_cast<const T*>(a.sin_p) + b;
    if (PM == kParamsRef32 && i == 10 && a.bore_phi != nullptr) return a.bore_phi + b;
    return nullptr;
  }
}

// Rotation of a sample from its fields, got(i) returning field i (float for
// the reference typing, double otherwise).
template <int PM, class Get>
__device__ __forceinline__ SampleRot rot_from_fields(const KArgs& a, const Get& got) {
  SampleRot r;
  if constexpr (PM == kAngles) {
    r = rot_from_angle_values(a, got(0), got(1), got(2));
  } else if constexpr (f64_params(PM)) {
    r.kx = got(0);
    r.ky = got(1);
    r.kz = got(2);
    r.ca = got(3);
    r.sa = got(4);
    r.px = got(5);
    r.py = got(6);
    r.pz = got(7);
    r.cp = got(8);
    r.sp = got(9);
  } else {
    r.fkx = got(0);
    r.fky = got(1);
    r.fkz = got(2);
    r.fca = got(3);
    r.fsa = got(4);
    r.kx = (double)r.fkx;
    r.ky = (double)r.fky;
    r.kz = (double)r.fkz;
    r.ca = (double)r.fca;
    r.sa = (double)r.fsa;
    r.px = (double)got(5);
    r.py = (double)got(6);
    r.pz = (double)got(7);
    r.cp = (double)got(8);
    r.sp = (double)got(9);
  }
  return r;
}

// Boresight (z, sin theta, phi) of the spin-2 angle.  Float32 parameters use
// the reference's typing: sin theta from a float32 square, phi from float32
// atan2 (host libm value when provided).
template <int PM, class Get>
__device__ __forceinline__ void boresight_from_fields(const KArgs& a, const SampleRot& rot, const Get& got, double& z,
                                                      double& sth, double& phi) {
  if constexpr (PM == kAngles) {
    z = clamp1(rot.pz);
    sth = sqrt(max0(1.0 - rot.pz * rot.pz));
    phi = atan2(rot.py, rot.px);
  } else if constexpr (f64_params(PM)) {
    const double pz = got(7);
    z = clamp1(pz);
    sth = sqrt(max0(1.0 - pz * pz));
    phi = atan2((double)got(6), (double)got(5));
  } else {
    const float bz = got(7);
    const float bz2 = bz * bz;
    z = clamp1((double)bz);
    sth = sqrt(max0(1.0 - (double)bz2));
    if (a.bore_phi != nullptr)
      phi = (double)got(10);
    else
      phi = (double)(float)atan2((double)got(6), (double)got(5));
  }
  if (phi < 0.0) phi += kTwoPi;
}

// Field getter reading global memory.
template <int PM>
struct GlobalFields {
  const KArgs& a;
  long long b;
  __device__ __forceinline__ auto operator()(int i) const {
    if constexpr (PM == kParamsRef32)
      return *static_cast<const float*>(field_ptr<PM>(a, b, i));
    else if constexpr (PM == kAngles)
      return a.angles_f32 ? (double)*static_cast<const float*>(field_ptr<PM>(a, b, i))
                          : *static_cast<const double*>(field_ptr<PM>(a, b, i));
    else
      return *static_cast<const double*>(field_ptr<PM>(a, b, i));
  }
};

template <int PM>
__device__ __forceinline__ SampleRot load_rot(const KArgs& a, long long b) {
  return rot_from_fields<PM>(a, GlobalFields<PM>{a, b});
}

// ---------------------------------------------------------------------------
// Map element types.  Planar float/double maps are the reference's
// mp_stacked (C, N); the precision form packs a pixel's components into one
// record: PackF32 = 4 x float32 (16 B), PackBF16 = 4 x bfloat16 (8 B).  The
// precision form also keeps cos 2d / sin 2d in float32 and accumulates in
// float32 with Kahan compensation; pixel decisions and weights stay float64.
// PackF64 = 4 x float64 (32 B, one sector) is the float64 path's layout with
// a pixel's components together: every value and operation as for a planar
// float64 map, so the results are the same bit for bit.
// ---------------------------------------------------------------------------

struct PackF32 {};
struct PackBF16 {};
struct PackF64 {};

template <typename MapT>
struct MapTraits {
  static constexpr bool packed = false;
};
template <>
struct MapTraits<PackF32> {
  static constexpr bool packed = true;
};
template <>
struct MapTraits<PackBF16> {
  static constexpr bool packed = true;
};

__device__ __forceinline__ float bf16_lo(unsigned v) { return __uint_as_float(v << 16); }
__device__ __forceinline__ float bf16_hi(unsigned v) { return __uint_as_float(v & 0xffff0000u); }

template <typename MapT>
__device__ __forceinline__ float4 load_rec(const void* map, long long p) {
  if constexpr (std::is_same<MapT, PackF32>::value) {
    return __ldg(static_cast<const float4*>(map) + p);
  } else {
    const uint2 r = __ldg(static_cast<const uint2*>(map) + p);
    return make_float4(bf16_lo(r.x), bf16_hi(r.x), bf16_lo(r.y), bf16_hi(r.y));
  }
}

// Per-thread accumulators: float64 (parity path) or float32 with Kahan
// compensation (precision form).
struct Acc64 {
  double v[4] = {0.0, 0.0, 0.0, 0.0};
  __device__ __forceinline__ void add(int c, double x) { v[c] += x; }
  __device__ __forceinline__ double total(int c) const { return v[c]; }
};
struct AccKahan {
  float s[4] = {0.f, 0.f, 0.f, 0.f};
  float e[4] = {0.f, 0.f, 0.f, 0.f};  // running compensation (minus the lost low bits)
  __device__ __forceinline__ void add(int c, float x) {
    const float y = x - e[c];
    const float t = s[c] + y;
    e[c] = (t - s[c]) - y;
    s[c] = t;
  }
  __device__ __forceinline__ double total(int c) const { return (double)s[c] - (double)e[c]; }
};

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// ---------------------------------------------------------------------------
// Ring table (global memory, built once per nside and footprint reach).
// ---------------------------------------------------------------------------

// One RING ring.  Record 0 is a header: z = nside, ta = reach [rad].
struct __align__(16) RingRec {
  double z;         // ring centre z
  double sth;       // sqrt(max(0, 1 - z^2))
  double phi0;      // longitude of the first pixel
  double dphi;      // pixel spacing
  double ta;        // acos(z)
  double inv_dta;   // 1 / (ta(ir + 1) - ta), correctly rounded (0 for the last ring)
  int unused0;
  int n;            // pixels in the ring
  double inv_dphi;  // 1 / dphi, correctly rounded
  long long first;  // first pixel index
  int cap;          // table slots reserved for this ring
  int unused;
};
static_assert(sizeof(RingRec) == 80, "RingRec must be 80 bytes");
static_assert(offsetof(RingRec, phi0) == 16 && offsetof(RingRec, ta) == 32 && offsetof(RingRec, unused0) == 48,
              "RingRec pairs must sit on 16-byte boundaries");

// The geometry of ring ir (all fields but cap), the values the ring table holds.
__device__ __forceinline__ RingRec make_ring(long long nside, long long ir) {
  const RingInfo ri = hp_ring_info(nside, ir, 12 * nside * nside);
  RingRec r;
  r.z = hp_ring_z(nside, ir);
  r.ta = acos(r.z);
  r.sth = sqrt(max0(1.0 - r.z * r.z));
  r.phi0 = ri.phi0;
  r.dphi = ri.dphi;
  r.first = ri.first;
  r.unused0 = 0;
  r.n = (int)ri.n;
  r.inv_dphi = 1.0 / ri.dphi;
  r.inv_dta = ir < 4 * nside - 1 ? 1.0 / (acos(hp_ring_z(nside, ir + 1)) - r.ta) : 0.0;
  r.cap = 0;
  r.unused = 0;
  return r;
}

// Ring provider backed by the global ring table.
struct TableRings {
  const RingRec* t;
  __device__ __forceinline__ RingData operator()(long long ir) const {
    const RingRec* r = t + ir;
    RingData d;
    d.z = __ldg(&r->z);
    d.ta = __ldg(&r->ta);
    d.phi0 = __ldg(&r->phi0);
    d.dphi = __ldg(&r->dphi);
    d.first = __ldg(&r->first);
    d.n = __ldg(&r->n);
    return d;
  }
  __device__ __forceinline__ double sth(long long ir, const RingData&) const { return __ldg(&t[ir].sth); }
};

// ---------------------------------------------------------------------------
// Per-sample state in shared memory.
// ---------------------------------------------------------------------------

// One sample, prepared by one thread for all.  The bilinear path works in the
// sample's frame: longitudes are measured from phi_u, the longitude of the
// rotated beam centre u, so a beam pixel's longitude is a small angle (an
// arctangent series of six terms) and every stencil position a small number
// relative to its ring's own origin.  m maps a beam vector (float64
// parameters: the vector itself; reference float32 parameters: the vector
// after the reference's float32-typed recentring) to (x, y, z) of that frame:
// longitude phi_u + atan2(y, x), z the sky's.
struct __align__(16) SampleBlock {
  double m[9];
  double oma;                                                // 1 - cos a
  float fkx, fky, fkz, fca, fsa;                             // reference float32 recentring
  int wide;                                                  // the pixel loop's form is kWide
  int far;                                                   // without a table: also where Q and U are turned there
  float fpad;
  double bz, bsth, bdl;                                      // boresight: z, sin theta, longitude - phi_u in [-pi, pi]
  double phi_u, theta_u;                                     // rotated beam centre
  int ir_lo, nr;                                             // window rings (nr = 0: none)
  double cu, su;                                             // cos, sin of theta_u
  double px, py, pz, cp, sp;                                 // reference float32 roll (polar_z)
};
static_assert(sizeof(SampleBlock) == 224 && offsetof(SampleBlock, cu) == 160 && offsetof(SampleBlock, px) == 176 &&
                  offsetof(SampleBlock, fkx) == 80,
              "SampleBlock layout");

// The reference's own two-step rotation (k, a; p, psi), for the nearest
// rule's exact path.
struct ExactBlock {
  double px, py, pz, cp, sp;
  double kx, ky, kz, ca, sa;
};

// Samples prepared together, one lane each: the preparation is a serial chain
// of some 500 float64 operations, so sixteen lanes of one warp run it side by
// side.
constexpr int kPrep = 16;

// One ring of a sample's window: the ring in the sample's frame (origin k0 +
// f0 in units of pixels: the longitude phi_u lies f0 past pixel k0), its
// stretch of the footprint and its geometry.  The stretch is the cnt pixels
// from -(cnt - 1) / 2 about k0; pixel j (relative to k0) has table slot base +
// j; slots = base << 16 | cnt - 1 (both below 65536 where a table is used).
// 80 bytes: 16-byte reads of eight neighbouring rings fall on different
// banks.  The pixel loop reads 36 bytes of the ring above and 20 of the one
// below (28 and 12 in the belt): every 4 bytes a lane reads cost a
// shared-memory wavefront.
struct __align__(16) RingWin {
  double f0, inv_dphi;
  double rta, inv_dta;  // acos(z) - theta_u; 1 / (acos(z of the next ring) - acos(z))
  double z, sth;
  long long first;
  double dphi;
  unsigned slots;
  int k0, n, pad;
};
static_assert(sizeof(RingWin) == 80 && offsetof(RingWin, rta) == 16 && offsetof(RingWin, z) == 32 &&
                  offsetof(RingWin, first) == 48 && offsetof(RingWin, slots) == 64,
              "RingWin layout");

// Table slot of pixel j; true when pixels j .. j + count - 1 all have one.
__device__ __forceinline__ bool slot_of(unsigned slots, int j, int count, int& slot) {
  const int top = (int)(slots & 0xffffu);
  slot = (int)(slots >> 16) + j;
  return (unsigned)(j + (top >> 1)) < (unsigned)(top + 2 - count);
}

// The boresight: z and sin theta.
struct Bore {
  double z, sth;
};

// Longitude of the boresight less that of pixel j (relative to k0) of a ring
// whose origin is f0.
__device__ __forceinline__ double pixel_dphi(double bdl, double f0, int j, double dphi) {
  return fma(f0 - (double)j, dphi, bdl);
}

__device__ __forceinline__ unsigned smem_u32(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }

// Shared-memory loads that stay inside the pixel loop (the values are the
// same for every pixel of a sample; loading them per pixel keeps them out of
// the registers the evaluation needs).
__device__ __forceinline__ double2 lds_d2(unsigned p) {
  double2 v;
  asm volatile("ld.shared.v2.f64 {%0, %1}, [%2];" : "=d"(v.x), "=d"(v.y) : "r"(p));
  return v;
}
__device__ __forceinline__ double lds_d1(unsigned p) {
  double v;
  asm volatile("ld.shared.f64 %0, [%1];" : "=d"(v) : "r"(p));
  return v;
}
__device__ __forceinline__ float4 lds_f4(unsigned p) {
  float4 v;
  asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(p));
  return v;
}
__device__ __forceinline__ uint4 lds_u4(unsigned p) {
  uint4 v;
  asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(p));
  return v;
}
__device__ __forceinline__ unsigned lds_u1(unsigned p) {
  unsigned v;
  asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(p));
  return v;
}

// ---------------------------------------------------------------------------
// Elementary functions of small arguments.
// ---------------------------------------------------------------------------

constexpr double kNearTan = 0.125;   // largest |tan| / angle of the series below
constexpr double kNearSin = 0.0625;  // largest |sin| of colat_near's

// y / x for x > 0 finite: hardware reciprocal estimate, one Newton step and a
// residual correction (Markstein, IBM J. Res. Dev. 34(1), 1990).
__device__ __forceinline__ double div_near(double y, double x) {
  double r;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(x));
  r = fma(r, fma(-x, r, 1.0), r);
  const double q = y * r;
  return fma(fma(-x, q, y), r, q);
}

// sqrt(s) for s > 0: reciprocal square-root estimate and Goldschmidt's
// iteration with a residual correction (same reference).
__device__ __forceinline__ double sqrt_near(double s) {
  double y;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(s));
  double g = s * y, h = 0.5 * y;
  const double r = fma(-g, h, 0.5);
  g = fma(g, r, g);
  h = fma(h, r, h);
  return fma(fma(-g, g, s), h, g);
}

// atan(t) for |t| <= kNearTan: Taylor series through t^15 (the first term left
// out, t^17 / 17, is below 3e-17 there).
__device__ __forceinline__ double atan_near(double t) {
  const double w = t * t;
  double p = fma(w, -1.0 / 15.0, 1.0 / 13.0);
  p = fma(w, p, -1.0 / 11.0);
  p = fma(w, p, 1.0 / 9.0);
  p = fma(w, p, -1.0 / 7.0);
  p = fma(w, p, 1.0 / 5.0);
  p = fma(w, p, -1.0 / 3.0);
  return fma(t * w, p, t);
}

// sin and cos of |x| <= kNearTan by their Taylor series (the first terms left out
// are below 2.4e-17 of the sine and 3e-20).
__device__ __forceinline__ void sincos_near(double x, double& s, double& c) {
  const double w = x * x;
  double p = fma(w, 1.0 / 362880.0, -1.0 / 5040.0);
  p = fma(w, p, 1.0 / 120.0);
  p = fma(w, p, -1.0 / 6.0);
  s = fma(x * w, p, x);
  double q = fma(w, -1.0 / 3628800.0, 1.0 / 40320.0);
  q = fma(w, q, -1.0 / 720.0);
  q = fma(w, q, 1.0 / 24.0);
  q = fma(w, q, -0.5);
  c = fma(w, q, 1.0);
}

// x > 0 and |t| < kNearTan for t = y / x by div_near, on the high words (a t
// that is not finite -- x zero, denormal, infinite or NaN -- fails).
__device__ __forceinline__ bool lon_is_near(double x, double t) {
  return __double2hiint(x) >= 0 && (__double2hiint(t) & 0x7fffffff) < 0x3fc00000;
}
// Longitude of (x, y) in the sample's frame.
__device__ __forceinline__ double frame_lon(double x, double y) {
  const double t = div_near(y, x);
  return lon_is_near(x, t) ? atan_near(t) : atan2(y, x);
}

// cos 2d / sin 2d of the frame rotation between a pixel centre and the
// boresight for longitudes up to kNearTan apart (false beyond: spin2_far).
// Reference float32 parameters: the haversine form of spin2_c2s2 (the
// reference forms the boresight's sin theta from a float32 square, so its z
// and sin theta disagree by 6e-8, and only the same
// form of N and D gives the same angle).  Float64 pointing: the same ratio
// N / D with the common factor 2h divided out,
//   N : D = (z + z_b) sin dphi : sin theta sin theta_b + (1 + z z_b) cos dphi,
// half the operations and well conditioned (D is near 2 for a nearby pixel).
template <int PM>
__device__ __forceinline__ bool spin2_small(double z, double sth, double dphi, const Bore& bo, double& c2d,
                                            double& s2d) {
  if ((__double2hiint(dphi) & 0x7fffffff) >= 0x3fc00000) return false;  // |dphi| >= kNearTan
  double N, D;
  if constexpr (PM == kParamsRef32) {
    if (dphi == 0.0 && bo.sth == sth && bo.z == z) {
      c2d = 1.0;
      s2d = 0.0;
      return true;
    }
    double sh, ch;
    sincos_near(dphi * 0.5, sh, ch);
    const double sin_dphi = 2.0 * ch * sh;
    const double sh2 = sh * sh;
    const double cos_dphi = fma(-2.0, sh2, 1.0);
    const double dz = bo.z - z, ds = bo.sth - sth;
    const double st2 = 0.25 * fma(dz, dz, ds * ds);
    const double S = sth * bo.sth, S2 = S * sh2;
    N = 2.0 * sin_dphi * ((bo.z + z) * (st2 + S2));
    const double q = 4.0 * st2;
    D = fma(q - q * st2, cos_dphi, fma(S * sin_dphi, sin_dphi, -4.0 * (bo.z * z) * (S2 * sh2)));
  } else {
    double s, c;
    sincos_near(dphi, s, c);
    N = s * (bo.z + z);
    D = fma(fma(bo.z, z, 1.0), c, sth * bo.sth);
  }
  const double n2 = N * N;
  const double u = div_near(1.0, fma(D, D, n2));
  c2d = fma(D, D, -n2) * u;
  s2d = 2.0 * N * D * u;
  return true;
}
static __device__ __noinline__ double2 spin2_far(double z, double sth, double dphi, double bz, double bsth) {
  double2 r;
  spin2_c2s2(z, sth, 0.0, bz, bsth, dphi, r.x, r.y);
  return r;
}

// Position of the frame's origin longitude on a ring: phi_u lies f0 in [0, 1)
// pixels past pixel k0 (mod the ring's length).
__device__ __forceinline__ void ring_origin(double phi_u, double phi0, double dphi, double inv_dphi, int& k0,
                                            double& f0) {
  const double x = phi_u - phi0;
  const double k = floor(x * inv_dphi);
  f0 = fma(-k, dphi, x) * inv_dphi;
  k0 = (int)k;
}

// ---------------------------------------------------------------------------
// Per-sample preparation (one lane per sample, out of line).
// ---------------------------------------------------------------------------

// 3 x 3 matrix of r -> r cos t + (k x r) sin t + k (k . r) (1 - cos t).
__device__ __forceinline__ void rodrigues_matrix(double x, double y, double z, double c, double s, double omc,
                                                 double* m) {
  const double ox = omc * x, oy = omc * y, oz = omc * z;
  m[0] = fma(ox, x, c);
  m[1] = fma(ox, y, -(s * z));
  m[2] = fma(ox, z, s * y);
  m[3] = fma(oy, x, s * z);
  m[4] = fma(oy, y, c);
  m[5] = fma(oy, z, -(s * x));
  m[6] = fma(oz, x, -(s * y));
  m[7] = fma(oz, y, s * x);
  m[8] = fma(oz, z, c);
}

template <int PM, bool TABLE>
__device__ __noinline__ void prepare_sample(const KArgs& a, long long b, bool has_qu, double cx, double cy, double cz,
                                            double rbeam, bool window, double polar, SampleBlock& sb,
                                            ExactBlock* eb) {
  const GlobalFields<PM> got{a, b};
  const SampleRot r = rot_from_fields<PM>(a, got);
  if (eb != nullptr) {
    eb->px = r.px;
    eb->py = r.py;
    eb->pz = r.pz;
    eb->cp = r.cp;
    eb->sp = r.sp;
    eb->kx = r.kx;
    eb->ky = r.ky;
    eb->kz = r.kz;
    eb->ca = r.ca;
    eb->sa = r.sa;
  }
  const double omp = 1.0 - r.cp, oma = 1.0 - r.ca;
  sb.oma = oma;
  if constexpr (PM == kParamsRef32) {
    sb.fkx = r.fkx;
    sb.fky = r.fky;
    sb.fkz = r.fkz;
    sb.fca = r.fca;
    sb.fsa = r.fsa;
    sb.px = r.px;
    sb.py = r.py;
    sb.pz = r.pz;
    sb.cp = r.cp;
    sb.sp = r.sp;
  }
  double bphi = 0.0;
  if (has_qu) {
    double z, sth;
    boresight_from_fields<PM>(a, r, got, z, sth, bphi);
    sb.bz = z;
    sb.bsth = sth;
  }
  double A[9], M[9];
  rodrigues_matrix(r.px, r.py, r.pz, r.cp, r.sp, omp, A);
  rodrigues_matrix(r.kx, r.ky, r.kz, r.ca, r.sa, oma, M);
  double ux, uy, uz;
  {
    const double wx = fma(M[0], cx, fma(M[1], cy, M[2] * cz));
    const double wy = fma(M[3], cx, fma(M[4], cy, M[5] * cz));
    const double wz = fma(M[6], cx, fma(M[7], cy, M[8] * cz));
    ux = fma(A[0], wx, fma(A[1], wy, A[2] * wz));
    uy = fma(A[3], wx, fma(A[4], wy, A[5] * wz));
    uz = fma(A[6], wx, fma(A[7], wy, A[8] * wz));
  }
  double phi_u = atan2(uy, ux);
  if (phi_u < 0.0) phi_u += kTwoPi;
  double s, c;
  sincos(phi_u, &s, &c);
  // rows of the roll turned by -phi_u about z, then times the recentring
#pragma unroll
  for (int j = 0; j < 3; ++j) {
    const double a0 = A[j], a1 = A[3 + j];
    A[j] = fma(c, a0, s * a1);
    A[3 + j] = fma(c, a1, -(s * a0));
  }
#pragma unroll
  for (int i = 0; i < 3; ++i)
#pragma unroll
    for (int j = 0; j < 3; ++j)
      sb.m[3 * i + j] = PM == kParamsRef32
                            ? A[3 * i + j]
                            : fma(A[3 * i], M[j], fma(A[3 * i + 1], M[3 + j], A[3 * i + 2] * M[6 + j]));
  sb.phi_u = phi_u;
  double bdl = bphi - phi_u;
  if (bdl > kPi)
    bdl -= kTwoPi;
  else if (bdl < -kPi)
    bdl += kTwoPi;
  sb.bdl = bdl;
  const double theta_u = acos(clamp1(uz));
  sb.theta_u = theta_u;
  sincos(theta_u, &sb.su, &sb.cu);
  int ir_lo = 0, nr = 0;
  const double th_lo = theta_u - rbeam, th_hi = theta_u + rbeam;
  if (window && isfinite(phi_u) && isfinite(uz) && th_lo >= polar && th_hi <= kPi - polar) {
    long long lo = th_lo <= 0.0 ? 1 : hp_ring_above(a.nside, cos(th_lo));
    long long hi = th_hi >= kPi ? 4 * a.nside - 1 : hp_ring_above(a.nside, cos(th_hi)) + 1;
    lo = max(lo, 1LL);
    hi = min(hi, 4 * a.nside - 1);
    if (hi >= lo && hi - lo + 1 <= a.ring_cap) {
      ir_lo = (int)lo;
      nr = (int)(hi - lo + 1);
    }
  }
  sb.ir_lo = ir_lo;
  sb.nr = nr;
  // where the short series end; the nearest rule's cosine holds for half a pixel of
  // rings of 157 pixels (kCosSmallMax)
  sb.wide = rbeam > kNearSin - 0.001 || rbeam > (kNearTan - 0.001) * sb.su ||
            (eb != nullptr && nr > 0 && 4 * min(ir_lo, (int)(4 * a.nside) - (ir_lo + nr - 1)) < 158) ||
            (eb != nullptr && a.nside < 40);
  if (!TABLE) sb.far = sb.wide || (has_qu && fabs(bdl) * sb.su + rbeam > kNearTan * sb.su);
}

// Two beam pixels (or one) in the sample's frame.  The rotation is read from
// shared memory for every pair: held in registers (18, and 7 more for the
// reference typing) it left room for a third fewer warps.
template <int N>
__device__ __forceinline__ void to_frame(unsigned sb, const double (&v)[N][3], double* x, double* y, double* z) {
  const double2 m0 = lds_d2(sb), m1 = lds_d2(sb + 16);
#pragma unroll
  for (int k = 0; k < N; ++k) x[k] = fma(m0.x, v[k][0], fma(m0.y, v[k][1], m1.x * v[k][2]));
  const double2 m2 = lds_d2(sb + 32);
#pragma unroll
  for (int k = 0; k < N; ++k) y[k] = fma(m1.y, v[k][0], fma(m2.x, v[k][1], m2.y * v[k][2]));
  const double2 m3 = lds_d2(sb + 48);
  const double m8 = lds_d1(sb + 64);
#pragma unroll
  for (int k = 0; k < N; ++k) z[k] = fma(m3.x, v[k][0], fma(m3.y, v[k][1], m8 * v[k][2]));
}
template <int N>
__device__ __forceinline__ void rotate_frame(unsigned sb, const double* const* vec, const int (&at)[N], double* x,
                                             double* y, double* z) {
  double v[N][3];
#pragma unroll
  for (int k = 0; k < N; ++k)
#pragma unroll
    for (int i = 0; i < 3; ++i) v[k][i] = __ldg(vec[i] + at[k]);
  to_frame<N>(sb, v, x, y, z);
}
// Reference typing: the recentring's products and sums are float32, as in
// rot_ref32 (the same bits), the roll and the frame float64.
__device__ __forceinline__ void recentre32(unsigned sb, float vx, float vy, float vz, double* v) {
  const float4 fk = lds_f4(sb + 80);  // fkx, fky, fkz, fca
  const float fsa = __uint_as_float(lds_u1(sb + 96));
  const double oma = lds_d1(sb + 72);
  const float dkv = fk.x * vx + fk.y * vy + fk.z * vz;
  const float ax = vx * fk.w + (fk.y * vz - fk.z * vy) * fsa;
  const float ay = vy * fk.w + (fk.z * vx - fk.x * vz) * fsa;
  const float az = vz * fk.w + (fk.x * vy - fk.y * vx) * fsa;
  v[0] = (double)ax + (double)(fk.x * dkv) * oma;
  v[1] = (double)ay + (double)(fk.y * dkv) * oma;
  v[2] = (double)az + (double)(fk.z * dkv) * oma;
}
template <int N>
__device__ __forceinline__ void rotate_frame(unsigned sb, const float* const* vec, const int (&at)[N], double* x,
                                             double* y, double* z) {
  double v[N][3];
#pragma unroll
  for (int k = 0; k < N; ++k) recentre32(sb, __ldg(vec[0] + at[k]), __ldg(vec[1] + at[k]), __ldg(vec[2] + at[k]), v[k]);
  to_frame<N>(sb, v, x, y, z);
}

// Near a pole the colatitude is ill-conditioned in z (an error of 1e-16 becomes
// 1e-16 / sin theta, and the ring weight's 1.2 nside times that), so the
// reference's own rounding of z shows there: with z from the matrix one random
// pole-crossing case of twenty differed from it by more than 1e-12 (300 seeds,
// nside 64 and 256).  Beyond |z| = kPolarZ z is therefore formed by rot_ref32's
// operations in its order.  Float64 pointing has no such typing to follow.
constexpr double kPolarZ = 0.9;
__device__ __forceinline__ bool is_polar(double z) { return fabs(z) > kPolarZ; }
__device__ __forceinline__ double polar_z(unsigned sb, const float* const* vec, int at) {
  double v[3];
  recentre32(sb, __ldg(vec[0] + at), __ldg(vec[1] + at), __ldg(vec[2] + at), v);
  const double2 pxy = lds_d2(sb + 176), pzc = lds_d2(sb + 192);
  const double sp = lds_d1(sb + 208);
  const double dpr = pxy.x * v[0] + pxy.y * v[1] + pzc.x * v[2];
  return v[2] * pzc.y + (pxy.x * v[1] - pxy.y * v[0]) * sp + pzc.x * dpr * (1.0 - pzc.y);
}
__device__ __forceinline__ double polar_z(unsigned, const double* const*, int) { return 0.0; }

// The reference's own rotation of a beam pixel (rot_ref32 / rot_f64).
__device__ __forceinline__ void rotate_exact(const SampleBlock* sb, const ExactBlock* eb, float vx, float vy, float vz,
                                             double& ox, double& oy, double& oz) {
  SampleRot r;
  r.px = eb->px;
  r.py = eb->py;
  r.pz = eb->pz;
  r.cp = eb->cp;
  r.sp = eb->sp;
  r.fkx = sb->fkx;
  r.fky = sb->fky;
  r.fkz = sb->fkz;
  r.fca = sb->fca;
  r.fsa = sb->fsa;
  rot_ref32(r, vx, vy, vz, ox, oy, oz);
}
__device__ __forceinline__ void rotate_exact(const SampleBlock*, const ExactBlock* eb, double vx, double vy, double vz,
                                             double& ox, double& oy, double& oz) {
  SampleRot r;
  r.px = eb->px;
  r.py = eb->py;
  r.pz = eb->pz;
  r.cp = eb->cp;
  r.sp = eb->sp;
  r.kx = eb->kx;
  r.ky = eb->ky;
  r.kz = eb->kz;
  r.ca = eb->ca;
  r.sa = eb->sa;
  rot_f64(r, vx, vy, vz, ox, oy, oz);
}

// Beam centre direction (normalised mean of the beam vectors [s0, s1)) and the
// largest angle between it and any of them; by the whole CTA.  The mean is
// summed by the first 128 threads whatever the CTA's size, so that every CTA
// shape measures longitudes in the same frame, bit for bit.
constexpr int kMeanLanes = 128;
template <int PM>
__device__ void beam_extent(const KArgs& a, int s0, int s1, double* s_red, double& cx, double& cy, double& cz,
                            double& radius) {
  using VecT = typename std::conditional<PM == kParamsRef32, float, double>::type;
  const VecT* vec = static_cast<const VecT*>(a.vec);
  const long long si = a.vec_si;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, NT = blockDim.x;
  double sx = 0.0, sy = 0.0, sz = 0.0;
  __syncthreads();  // earlier users of s_red are done
  if (tid < kMeanLanes) {
#pragma unroll 4
    for (int s = s0 + tid; s < s1; s += kMeanLanes) {
      const VecT* v = vec + (long long)s * a.vec_ss;
      sx += (double)v[0];
      sy += (double)v[si];
      sz += (double)v[2 * si];
    }
    sx = warp_sum(sx);
    sy = warp_sum(sy);
    sz = warp_sum(sz);
    if (lane == 0) {
      s_red[warp * 4 + 0] = sx;
      s_red[warp * 4 + 1] = sy;
      s_red[warp * 4 + 2] = sz;
    }
  }
  __syncthreads();
  sx = sy = sz = 0.0;
  for (int i = 0; i < kMeanLanes / 32; ++i) {
    sx += s_red[i * 4 + 0];
    sy += s_red[i * 4 + 1];
    sz += s_red[i * 4 + 2];
  }
  const double nrm = sqrt(sx * sx + sy * sy + sz * sz);
  if (nrm > 0.0 && nrm < 1e300) {
    cx = sx / nrm;
    cy = sy / nrm;
    cz = sz / nrm;
  } else {
    cx = 0.0;
    cy = 0.0;
    cz = 1.0;
  }
  double mind = 1.0;
#pragma unroll 4
  for (int s = s0 + tid; s < s1; s += NT) {
    const VecT* v = vec + (long long)s * a.vec_ss;
    const double vx = v[0], vy = v[si], vz = v[2 * si];
    const double vn = sqrt(vx * vx + vy * vy + vz * vz);
    const double d = vn > 0.0 ? (vx * cx + vy * cy + vz * cz) / vn : -1.0;
    mind = fmin(mind, d);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) mind = fmin(mind, __shfl_xor_sync(0xffffffffu, mind, o));
  __syncthreads();
  if (lane == 0) s_red[warp] = mind;
  __syncthreads();
  mind = 1.0;
  for (int i = 0; i < NT / 32; ++i) mind = fmin(mind, s_red[i]);
  __syncthreads();
  radius = acos(clamp1(mind));
}

// ---------------------------------------------------------------------------
// Values of one map pixel as the accumulation uses them: every component,
// with Q and U turned into the boresight's frame.
// ---------------------------------------------------------------------------

constexpr int kLayoutGeneric = 0;  // runtime C, c_q, c_u
constexpr int kLayoutIQU = 1;      // C = 3, Q at 1, U at 2

template <int LAYOUT>
struct Chan {
  int C, q, u;
  Chan() = default;
  __device__ __forceinline__ explicit Chan(const KArgs& a) : C(a.C), q(a.c_q), u(a.c_u) {}
};
template <>
struct Chan<kLayoutIQU> {
  static constexpr int C = 3, q = 1, u = 2;
  Chan() = default;
  __device__ __forceinline__ explicit Chan(const KArgs&) {}
};

template <typename MapT>
using ValT = typename std::conditional<MapTraits<MapT>::packed, float, double>::type;

template <typename R>
struct Vals {
  R v[4];
};

// q turned by (c2, s2) and u turned by (c2, s2): the products of the reference
// (tod_bilinear.py:440-470), float32 for packed float32/bfloat16 records.
__device__ __forceinline__ double turn_q(double q, double u, double c2, double s2) { return fma(q, c2, u * s2); }
__device__ __forceinline__ double turn_u(double q, double u, double c2, double s2) { return fma(u, c2, -q * s2); }
__device__ __forceinline__ float turn_q(float q, float u, double c2, double s2) {
  return fmaf(q, (float)c2, u * (float)s2);
}
__device__ __forceinline__ float turn_u(float q, float u, double c2, double s2) {
  return fmaf(u, (float)c2, -q * (float)s2);
}

template <typename R>
__device__ __forceinline__ R pick4(const R* v, int c) {
  return c == 0 ? v[0] : (c == 1 ? v[1] : (c == 2 ? v[2] : v[3]));
}

struct MapRef {
  const void* map;
  long long stride;
};

template <typename MapT, int LAYOUT>
__device__ __forceinline__ Vals<ValT<MapT>> raw_vals(const Chan<LAYOUT>& ch, const MapRef& m, long long p) {
  Vals<ValT<MapT>> o{{0, 0, 0, 0}};
  if constexpr (MapTraits<MapT>::packed) {
    const float4 r = load_rec<MapT>(m.map, p);
    o.v[0] = r.x;
    o.v[1] = r.y;
    o.v[2] = r.z;
    o.v[3] = r.w;
  } else if constexpr (std::is_same<MapT, PackF64>::value) {
    const double2 lo = __ldg(static_cast<const double2*>(m.map) + 2 * p);
    o.v[0] = lo.x;
    o.v[1] = lo.y;
    if (ch.C > 2) {
      const double2 hi = __ldg(static_cast<const double2*>(m.map) + 2 * p + 1);
      o.v[2] = hi.x;
      o.v[3] = hi.y;
    }
  } else {
#pragma unroll
    for (int c = 0; c < 4; ++c)
      if (c < ch.C) o.v[c] = (double)__ldg(static_cast<const MapT*>(m.map) + (long long)c * m.stride + p);
  }
  return o;
}

template <typename MapT, int LAYOUT>
__device__ __forceinline__ Vals<ValT<MapT>> turned_vals(const Chan<LAYOUT>& ch, const MapRef& m, long long p,
                                                        double c2, double s2) {
  using R = ValT<MapT>;
  Vals<R> o = raw_vals<MapT, LAYOUT>(ch, m, p);
  const R q = pick4(o.v, ch.q), u = pick4(o.v, ch.u);
  const R tq = turn_q(q, u, c2, s2), tu = turn_u(q, u, c2, s2);
#pragma unroll
  for (int c = 0; c < 4; ++c) {
    if (c == ch.q) o.v[c] = tq;
    if (c == ch.u) o.v[c] = tu;
  }
  return o;
}

template <int PM, bool HAS_QU, typename MapT, int LAYOUT>
__device__ __forceinline__ Vals<ValT<MapT>> pixel_vals(const Chan<LAYOUT>& ch, const MapRef& m, const Bore& bo,
                                                       double z, double sth, double dphi, long long p) {
  if constexpr (HAS_QU) {
    double c2, s2;
    if (!spin2_small<PM>(z, sth, dphi, bo, c2, s2)) {
      const double2 r = spin2_far(z, sth, dphi, bo.z, bo.sth);
      c2 = r.x;
      s2 = r.y;
    }
    return turned_vals<MapT, LAYOUT>(ch, m, p, c2, s2);
  } else {
    return raw_vals<MapT, LAYOUT>(ch, m, p);
  }
}

// The sample's value table in shared memory: slot i holds the values of one
// footprint pixel -- packed maps components 0 and 1 as a pair, then component
// 2 and component 3 arrays; float64 values components 0 and 1
// as a pair (a single for C = 1), then component 2 and component 3 arrays.
__host__ __device__ constexpr int slot_bytes(bool packed, int C) {
  return packed ? (C <= 3 ? 12 : 16) : (C == 1 ? 8 : (C == 2 ? 16 : (C == 3 ? 24 : 32)));
}

template <typename MapT, int LAYOUT>
struct ValTable {
  using R = ValT<MapT>;
  unsigned base;  // shared address
  int cap;
  __device__ __forceinline__ void store(const Chan<LAYOUT>& ch, int i, const Vals<R>& o) const {
    if constexpr (MapTraits<MapT>::packed) {
      asm volatile("st.shared.v2.f32 [%0], {%1, %2};" ::"r"(base + 8u * i), "f"(o.v[0]), "f"(o.v[1]) : "memory");
      asm volatile("st.shared.f32 [%0], %1;" ::"r"(base + 8u * cap + 4u * i), "f"(o.v[2]) : "memory");
      if (ch.C > 3) asm volatile("st.shared.f32 [%0], %1;" ::"r"(base + 12u * cap + 4u * i), "f"(o.v[3]) : "memory");
    } else {
      if (ch.C == 1) {
        asm volatile("st.shared.f64 [%0], %1;" ::"r"(base + 8u * i), "d"(o.v[0]) : "memory");
        return;
      }
      asm volatile("st.shared.v2.f64 [%0], {%1, %2};" ::"r"(base + 16u * i), "d"(o.v[0]), "d"(o.v[1]) : "memory");
      if (ch.C > 2) asm volatile("st.shared.f64 [%0], %1;" ::"r"(base + 16u * cap + 8u * i), "d"(o.v[2]) : "memory");
      if (ch.C > 3) asm volatile("st.shared.f64 [%0], %1;" ::"r"(base + 24u * cap + 8u * i), "d"(o.v[3]) : "memory");
    }
  }
  __device__ __forceinline__ Vals<R> load(const Chan<LAYOUT>& ch, int i) const {
    Vals<R> o{{0, 0, 0, 0}};
    if constexpr (MapTraits<MapT>::packed) {
      asm volatile("ld.shared.v2.f32 {%0, %1}, [%2];" : "=f"(o.v[0]), "=f"(o.v[1]) : "r"(base + 8u * i));
      o.v[2] = __uint_as_float(lds_u1(base + 8u * cap + 4u * i));
      if (ch.C > 3) o.v[3] = __uint_as_float(lds_u1(base + 12u * cap + 4u * i));
    } else {
      if (ch.C == 1) {
        o.v[0] = lds_d1(base + 8u * i);
        return o;
      }
      const double2 p = lds_d2(base + 16u * i);
      o.v[0] = p.x;
      o.v[1] = p.y;
      if (ch.C > 2) o.v[2] = lds_d1(base + 16u * cap + 8u * i);
      if (ch.C > 3) o.v[3] = lds_d1(base + 24u * cap + 8u * i);
    }
    return o;
  }
};

// Weighted sum of the four neighbours per component, in the reference's order
// k = 0..3; float32 (with the reference form's separate Q/U products) for
// packed maps.
template <typename MapT, int LAYOUT, bool HAS_QU>
struct Mix {
  using R = ValT<MapT>;
  R t[4];
  __device__ __forceinline__ void add(const Chan<LAYOUT>& ch, bool start, double wk, const Vals<R>& o) {
    const R w = (R)wk;
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      if (c >= ch.C) break;
      if constexpr (MapTraits<MapT>::packed) {
        if (HAS_QU && (c == ch.q || c == ch.u)) {
          const float x = w * o.v[c];
          t[c] = start ? x : t[c] + x;
          continue;
        }
      }
      t[c] = start ? w * o.v[c] : fma(w, o.v[c], t[c]);
    }
  }
};

// What one beam pixel adds per component; err = 1: nothing (non-finite or
// outside the map).
struct Contrib {
  double v[4];
  int err;
};

template <typename MapT>
__device__ __forceinline__ void accumulate(Acc64& acc, int c, double t, float bv) {
  acc.v[c] = fma(t, (double)bv, acc.v[c]);
}
template <typename MapT>
__device__ __forceinline__ void accumulate(AccKahan& acc, int c, float t, float bv) {
  acc.add(c, t * bv);
}

// ---------------------------------------------------------------------------
// Bilinear stencil.
// ---------------------------------------------------------------------------

// hp_ring_above for |z| <= 1, with the table path's square root and one fused
// multiply-add (the weights are continuous across a ring).
__device__ __forceinline__ long long ring_above(long long nside, double z) {
  const double az = fabs(z);
  if (az > kTwoThirds) {
    const double s = 3.0 * (1.0 - az);
    const long long ir = s > 0.0 ? (long long)((double)nside * sqrt_near(s)) : 0;
    return z < 0.0 ? 4 * nside - ir - 1 : ir;
  }
  return (long long)((double)nside * fma(-1.5, z, 2.0));
}

// theta_q - theta_u of a query z from sin(theta_q - theta_u) = cos(theta_u)
// sin(theta_q) - z sin(theta_u) and the arcsine series for angles under
// kNearSin (the first term left out, 231/13312 d^13, is below 4e-18 there).
__device__ __forceinline__ double colat_near(double z, double cu, double su, double& d) {
  d = fma(cu, sqrt_near((1.0 - z) * (1.0 + z)), -z * su);
  const double d2 = d * d;
  double p = fma(d2, 63.0 / 2816.0, 35.0 / 1152.0);
  p = fma(d2, p, 5.0 / 112.0);
  p = fma(d2, p, 3.0 / 40.0);
  p = fma(d2, p, 1.0 / 6.0);
  return fma(d * d2, p, d);
}
__device__ __forceinline__ bool sin_is_near(double d) { return (__double2hiint(d) & 0x7fffffff) < 0x3fb00000; }

__device__ __forceinline__ RingRec ring_at(const KArgs& a, long long ir) {
  if (a.ring_table != nullptr) {
    const RingRec* r = static_cast<const RingRec*>(a.ring_table) + ir;
    RingRec o;
    o.z = __ldg(&r->z);
    o.sth = __ldg(&r->sth);
    o.phi0 = __ldg(&r->phi0);
    o.dphi = __ldg(&r->dphi);
    o.ta = __ldg(&r->ta);
    o.inv_dta = __ldg(&r->inv_dta);
    o.n = __ldg(&r->n);
    o.inv_dphi = __ldg(&r->inv_dphi);
    o.first = __ldg(&r->first);
    return o;
  }
  return make_ring(a.nside, ir);
}

// One beam pixel without the sample's table: any position (poles, ring ends, longitudes far from the frame's
// origin), every ring and pixel value evaluated here.  Out of line; the same
// operations on the same values as the table path.
template <int PM, bool HAS_QU, typename MapT, int LAYOUT, typename VecT>
__device__ __noinline__ Contrib bilinear_direct(const KArgs& a, const SampleBlock* sb, const VecT* v) {
  Contrib out{{0.0, 0.0, 0.0, 0.0}, 0};
  double x, y, vz;
  const VecT* const vec[3] = {v, v + a.vec_si, v + 2 * a.vec_si};
  rotate_frame<1>(smem_u32(sb), vec, {0}, &x, &y, &vz);
  if (PM == kParamsRef32 && is_polar(vz)) vz = polar_z(smem_u32(sb), vec, 0);
  if (!(isfinite(x) && isfinite(y) && isfinite(vz))) {
    out.err = 1;
    return out;
  }
  const Chan<LAYOUT> ch(a);
  const Bore bo{sb->bz, sb->bsth};
  const double z = clamp1(vz);
  // a vector on the axis has longitude 0, as atan2(0, 0)
  const double rel = x == 0.0 && y == 0.0 ? -sb->phi_u : frame_lon(x, y);
  Mix<MapT, LAYOUT, HAS_QU> mix;
  int k0;
  double f0;
  // ring pixel j relative to the frame's origin
  auto visit = [&](bool start, const RingRec& r, int j, double wk) {
    const int ip = (int)py_imod((long long)k0 + j, r.n);
    mix.add(ch, start, wk,
            pixel_vals<PM, HAS_QU, MapT, LAYOUT>(ch, MapRef{a.map, a.map_stride}, bo, r.z, r.sth,
                                                 pixel_dphi(sb->bdl, f0, j, r.dphi), r.first + ip));
  };
  // the pixel left of the query and the fraction past it
  auto locate = [&](const RingRec& r, double& frac) {
    ring_origin(sb->phi_u, r.phi0, r.dphi, r.inv_dphi, k0, f0);
    const double u = fma(rel, r.inv_dphi, f0);
    const int j = __double2int_rd(u);
    frac = u - (double)j;
    return j;
  };
  const long long ir = ring_above(a.nside, z), last = 4 * a.nside - 1;
  double frac, d = 0.0;
  if (ir == 0 || ir == last) {
    // beyond the first or last ring: its pair and the opposite pair
    const RingRec r = ring_at(a, ir == 0 ? 1 : last);
    const int j = locate(r, frac);
    const double theta = acos(z);
    if (ir == 0) {
      const double wt = theta / r.ta;
      const double nf = (1.0 - wt) * 0.25;
      visit(true, r, j + 2, nf);
      visit(false, r, j + 3, nf);
      visit(false, r, j, (1.0 - frac) * wt + nf);
      visit(false, r, j + 1, frac * wt + nf);
    } else {
      const double ws = (theta - r.ta) / (kPi - r.ta);
      const double sf = ws * 0.25;
      visit(true, r, j, (1.0 - frac) * (1.0 - ws) + sf);
      visit(false, r, j + 1, frac * (1.0 - ws) + sf);
      visit(false, r, j + 2, sf);
      visit(false, r, j + 3, sf);
    }
  } else {
    double wb;
    {
      const RingRec r = ring_at(a, ir);
      double rel_th = colat_near(z, sb->cu, sb->su, d);
      if (!sin_is_near(d)) rel_th = acos(z) - sb->theta_u;
      wb = (rel_th - (r.ta - sb->theta_u)) * r.inv_dta;
      const int j = locate(r, frac);
      const double wa = 1.0 - wb;
      visit(true, r, j, wa * (1.0 - frac));
      visit(false, r, j + 1, wa * frac);
    }
    const RingRec r = ring_at(a, ir + 1);
    const int j = locate(r, frac);
    visit(false, r, j, wb * (1.0 - frac));
    visit(false, r, j + 1, wb * frac);
  }
#pragma unroll
  for (int c = 0; c < 4; ++c) {
    if (c >= ch.C) break;
    out.v[c] = (double)mix.t[c];
  }
  return out;
}

// Where a beam pixel falls: its left neighbours on the ring above and the ring
// below -- their slots in the sample's table, or (without a table) the pixels
// relative to the frame's origin --, the ring above's record and the four weights.
struct Place {
  int ia, ib;
  unsigned ra;
  double w[4];
};

// Forms of the pixel loops, by where a sample's window lies.
constexpr int kBelt = 0;      // all rings within the belt |z| <= 2/3 (and of one length)
constexpr int kAnywhere = 1;
// Footprints whose pixels are mostly beyond the short series -- wider than 3.6
// degrees in colatitude or 7 in longitude, so near the poles too --, and for the
// nearest rule rings of fewer than 157 pixels: the same with atan2 and acos where the
// series end.  Without it these went through the direct evaluation after a table had
// been filled for them: 2000 pixels of a 10 degree disc, nside 64, 10,000 samples
// 1976 -> 518 us; nearest at nside 16, 1560 -> 427; a 30' beam within 6 degrees of the
// pole, nside 1024, 20,000 samples 1823 -> 1010, nearest 1927 -> 1230 (calls, with
// their host part).
constexpr int kWide = 2;

// Place of a beam pixel: false when the query is not near the frame's origin
// in longitude, not between two rings of the window or (TABLE) not among their
// slots.
// Straight-line code, so that two pixels' chains interleave.
template <int REGION>
__device__ __forceinline__ bool frame_position(double x, double y, double& rel) {
  const double t = div_near(y, x);
  if constexpr (REGION == kWide) {
    rel = lon_is_near(x, t) ? atan_near(t) : atan2(y, x);
    // not finite, or on the axis: evaluated directly
    return fabs(x) < 1e300 && fabs(y) < 1e300 && (x != 0.0 || y != 0.0);
  } else {
    rel = atan_near(t);
    return lon_is_near(x, t);
  }
}
template <int REGION, bool TABLE>
__device__ __forceinline__ bool place_pixel(unsigned rings, int ir_lo, int nwin, int nside, double theta_u, double cu,
                                            double su, double belt_inv, double x, double y, double z, Place& o) {
  double rel;
  const bool near = frame_position<REGION>(x, y, rel);
  double rc = (double)nside * fma(-1.5, z, 2.0);
  int r;
  if constexpr (REGION == kBelt) {
    r = (int)rc;
  } else {
    const double az = fabs(z);
    const bool cap = az > kTwoThirds;
    const double rp = (double)nside * sqrt_near(3.0 * (1.0 - az));
    r = (int)(cap ? rp : rc);
    if (cap && z < 0.0) r = 4 * nside - r - 1;
  }
  r -= ir_lo;
  // (|z| >= 1 or NaN gives a ring outside every window)
  const bool in = near && (unsigned)r < (unsigned)nwin;
  const unsigned ra = rings + 80u * (in ? (unsigned)r : 0u);
  double2 f0, f1;
  if constexpr (REGION == kBelt) {
    f0 = make_double2(lds_d1(ra), belt_inv);
    f1 = make_double2(lds_d1(ra + 80), belt_inv);
  } else {
    f0 = lds_d2(ra);
    f1 = lds_d2(ra + 80);
  }
  const double ua = fma(rel, f0.y, f0.x), ub = fma(rel, f1.y, f1.x);
  const int ja = __double2int_rd(ua), jb = __double2int_rd(ub);
  int ia = ja, ib = jb;
  bool in_a = true, in_b = true;
  if constexpr (TABLE) {
    in_a = slot_of(lds_u1(ra + 64), ja, 2, ia);
    in_b = slot_of(lds_u1(ra + 144), jb, 2, ib);
  }
  const double xa = ua - (double)ja, xb = ub - (double)jb;
  double d;
  double rel_th = colat_near(z, cu, su, d);
  if (REGION == kWide && !sin_is_near(d)) rel_th = acos(z) - theta_u;
  const double2 ti = lds_d2(ra + 16);
  const double wb = (rel_th - ti.x) * ti.y;
  const double wa = 1.0 - wb;
  o.ia = ia;
  o.ib = ib;
  o.ra = ra;
  o.w[0] = wa * (1.0 - xa);
  o.w[1] = wa * xa;
  o.w[2] = wb * (1.0 - xb);
  o.w[3] = wb * xb;
  return in && in_a && in_b && (REGION == kWide || sin_is_near(d));
}

// A placed pixel's contribution from the table.
template <bool HAS_QU, typename MapT, int LAYOUT, class Acc>
__device__ __forceinline__ void add_placed(const Chan<LAYOUT>& ch, const ValTable<MapT, LAYOUT>& tab, const Place& o,
                                           float bvf, Acc& acc) {
  Mix<MapT, LAYOUT, HAS_QU> mix;
  mix.add(ch, true, o.w[0], tab.load(ch, o.ia));
  mix.add(ch, false, o.w[1], tab.load(ch, o.ia + 1));
  mix.add(ch, false, o.w[2], tab.load(ch, o.ib));
  mix.add(ch, false, o.w[3], tab.load(ch, o.ib + 1));
#pragma unroll
  for (int c = 0; c < 4; ++c) {
    if (c >= ch.C) break;
    accumulate<MapT>(acc, c, mix.t[c], bvf);
  }
}

// A placed pixel's contribution from the map; false when a neighbour is too far
// from the boresight in longitude for the form.
template <int REGION, int PM, bool HAS_QU, typename MapT, int LAYOUT, class Acc>
__device__ __forceinline__ bool add_from_map(const Chan<LAYOUT>& ch, const MapRef& map, const Bore& bo, double bdl,
                                             const Place& o, float bvf, Acc& acc) {
  Mix<MapT, LAYOUT, HAS_QU> mix;
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const unsigned r = o.ra + 80u * h;
    const uint4 g = lds_u4(r + 64);  // k0 in y, n in z
    const double2 fd = lds_d2(r + 48);
    const long long first = __double_as_longlong(fd.x);
    const int j = h == 0 ? o.ia : o.ib, n = (int)g.z;
    int ip = (int)g.y + j;  // (j up to half a turn and two pixels either way)
    ip += ip < 0 ? n : 0;
    ip -= ip >= n ? n : 0;
    ip -= ip >= n ? n : 0;
    const int in = ip + 1 == n ? 0 : ip + 1;
    double2 zs = make_double2(0.0, 0.0);
    double f0 = 0.0;
    if constexpr (HAS_QU) {
      zs = lds_d2(r + 32);
      f0 = lds_d1(r);
    }
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      const long long p = first + (k == 0 ? ip : in);
      Vals<ValT<MapT>> v;
      if constexpr (HAS_QU) {
        const double dphi = pixel_dphi(bdl, f0, j + k, fd.y);
        double c2, s2;
        if (!spin2_small<PM>(zs.x, zs.y, dphi, bo, c2, s2)) {
          if constexpr (REGION != kWide) return false;
          const double2 away = spin2_far(zs.x, zs.y, dphi, bo.z, bo.sth);
          c2 = away.x;
          s2 = away.y;
        }
        v = turned_vals<MapT, LAYOUT>(ch, map, p, c2, s2);
      } else {
        v = raw_vals<MapT, LAYOUT>(ch, map, p);
      }
      mix.add(ch, h + k == 0, o.w[2 * h + k], v);
    }
  }
#pragma unroll
  for (int c = 0; c < 4; ++c) {
    if (c >= ch.C) break;
    accumulate<MapT>(acc, c, mix.t[c], bvf);
  }
  return true;
}

// ---------------------------------------------------------------------------
// Nearest rule.
// ---------------------------------------------------------------------------

// cos(d) for |d| <= kCosSmallMax by its Taylor series through d^6 (the first
// term left out, d^8 / 8!, is below 7e-19 there), in Horner form in d^2.
constexpr double kCosSmallMax = 0.02;
__device__ __forceinline__ double cos_small(double d) {
  const double u = d * d;
  return fma(u, fma(u, fma(u, -1.0 / 720.0, 1.0 / 24.0), -0.5), 1.0);
}

// A component's term of the nearest mode: value x weight in float64, but a
// float32 map's own components as a float32 product (tod_nearest.py:146, :158).
template <bool HAS_QU, typename MapT, int LAYOUT>
__device__ __forceinline__ double nearest_term(const Chan<LAYOUT>& ch, int c, ValT<MapT> v, float bvf) {
  if constexpr (MapTraits<MapT>::packed) {
    return (double)(v * bvf);
  } else if constexpr (std::is_same<MapT, float>::value) {
    return (HAS_QU && (c == ch.q || c == ch.u)) ? v * (double)bvf : (double)((float)v * bvf);
  } else {
    return v * (double)bvf;
  }
}

// Pixel j of a ring of n as the one within half a turn of the frame's origin.
__device__ __forceinline__ int near_turn(int j, int n) {
  return j > n / 2 ? j - n : (j <= -(n / 2) ? j + n : j);
}

// The nearest rule as the reference evaluates it: its own rotation, atan2,
// four candidates ranked by cos().  Out of line.
template <int PM, bool HAS_QU, typename MapT, int LAYOUT, typename VecT>
__device__ __noinline__ Contrib nearest_exact(const KArgs& a, const SampleBlock* sb, const ExactBlock* eb, VecT v0,
                                              VecT v1, VecT v2, float bvf) {
  Contrib out{{0.0, 0.0, 0.0, 0.0}, 0};
  const Chan<LAYOUT> ch(a);
  double vx, vy, vz;
  rotate_exact(sb, eb, v0, v1, v2, vx, vy, vz);
  double phi_w = atan2(vy, vx);
  if (phi_w < 0.0) phi_w += kTwoPi;
  const double sin_th = sqrt(max0(vx * vx + vy * vy));
  const Nearest nb =
      a.ring_table != nullptr
          ? hp_nearest(a.nside, vz, sin_th, phi_w, TableRings{static_cast<const RingRec*>(a.ring_table)})
          : hp_nearest(a.nside, vz, sin_th, phi_w, DirectRingsNoAcos{a.nside, a.npix});
  if ((unsigned long long)nb.pix >= (unsigned long long)a.npix) {
    out.err = 1;
    return out;
  }
  const Bore bo{sb->bz, sb->bsth};
  // the boresight's longitude less the pixel's, as the window path forms it
  double dphi = sb->phi_u + sb->bdl - nb.phic;  // (ring 0: no candidate, a non-finite query)
  if (nb.ring > 0) {
    const RingRec r = ring_at(a, nb.ring);
    int k0;
    double f0;
    ring_origin(sb->phi_u, r.phi0, r.dphi, r.inv_dphi, k0, f0);
    dphi = pixel_dphi(sb->bdl, f0, near_turn((int)nb.ip - k0, r.n), r.dphi);
  }
  const Vals<ValT<MapT>> o = pixel_vals<PM, HAS_QU, MapT, LAYOUT>(ch, MapRef{a.map, a.map_stride}, bo, nb.zc,
                                                                  sqrt(max0(1.0 - nb.zc * nb.zc)), dphi, nb.pix);
#pragma unroll
  for (int c = 0; c < 4; ++c) {
    if (c >= ch.C) break;
    out.v[c] = nearest_term<HAS_QU, MapT, LAYOUT>(ch, c, o.v[c], bvf);
  }
  return out;
}

// Where a beam pixel of the nearest mode falls: window ring (its shared
// address) and pixel relative to the ring's origin.
//
// On each of the two rings that bracket z, the reference's two candidates are
// the pixels either side of the query, so the closer one is the rounded
// position; the two rings' winners are ranked by the cosine of their angular
// distance (cos_small).  The frame's positions differ from the reference's
// own (rounded) ones by under 1e-14 rad and the cosines by under 1e-15, so
// the reference picks the same pixel unless the query lies within 1e-9 of a
// candidate boundary (of a ring's or a pixel's width) or the lead is under
// 1e-13: then, and when anything is out of the window, false is returned and
// the caller takes the reference's evaluation.  Straight-line code; a false
// result still holds a valid ring.
struct NearPlace {
  unsigned ring;
  int j;
};
template <int REGION>
__device__ __forceinline__ bool place_nearest(unsigned rings, int ir_lo, int nwin, int nside, double x, double y,
                                              double z, NearPlace& o) {
  constexpr double kEdge = 1e-9;
  double rel;
  const bool near = frame_position<REGION>(x, y, rel);
  double rc = (double)nside * (2.0 - 1.5 * z);
  bool south = false;
  if constexpr (REGION != kBelt) {
    const double az = fabs(z);
    const double rp = (double)nside * sqrt_near(3.0 * (1.0 - az));
    const bool cap = az > kTwoThirds;
    rc = cap ? rp : rc;
    south = cap && z < 0.0;
  }
  int r = (int)rc;
  const double rf = rc - (double)r;
  if (south) r = 4 * nside - r - 1;
  r -= ir_lo;
  // (|z| >= 1 or NaN gives a ring outside every window)
  const bool in = near && (unsigned)r < (unsigned)nwin;
  const unsigned ra = rings + 80u * (in ? (unsigned)r : 0u);
  const double2 fa = lds_d2(ra), fb = lds_d2(ra + 80);
  const double ua = fma(rel, fa.y, fa.x), ub = fma(rel, fb.y, fb.x);
  const int ja = __double2int_rn(ua), jb = __double2int_rn(ub);
  const double ea = ua - (double)ja, eb = ub - (double)jb;
  const double la = ea * lds_d1(ra + 56), lb = eb * lds_d1(ra + 136);
  const double2 za = lds_d2(ra + 32), zb = lds_d2(ra + 112);
  const double sin_th = sqrt_near(fma(x, x, y * y));
  double cla, clb;
  if constexpr (REGION == kWide) {
    double sine;
    sincos_near(la, sine, cla);
    sincos_near(lb, sine, clb);
  } else {
    cla = cos_small(la);
    clb = cos_small(lb);
  }
  const double ca = fma(sin_th * za.y, cla, z * za.x);
  const double cb = fma(sin_th * zb.y, clb, z * zb.x);
  const bool b = cb > ca;
  o.ring = ra + (b ? 80u : 0u);
  o.j = b ? jb : ja;
  return in && fabs(rf - 0.5) < 0.5 - kEdge && fmax(fabs(ea), fabs(eb)) < 0.5 - kEdge &&
         fmax(fabs(la), fabs(lb)) <= (REGION == kWide ? kNearTan : kCosSmallMax) && fabs(ca - cb) > 1e-13;
}

// A placed pixel's contribution: from the table, or from the map where the
// launch has no table; false when the table does not hold the pixel.
template <int REGION, int PM, bool HAS_QU, typename MapT, int LAYOUT, class Acc>
__device__ __forceinline__ bool add_nearest(const Chan<LAYOUT>& ch, const MapRef& map, const Bore& bo, double bdl,
                                            const ValTable<MapT, LAYOUT>& tab, bool table, const NearPlace& o,
                                            const float* bv, Acc& acc) {
  Vals<ValT<MapT>> v;
  if (HAS_QU && table) {
    int slot;
    if (!slot_of(lds_u1(o.ring + 64), o.j, 1, slot)) return false;
    v = tab.load(ch, slot);
  } else {
    const int n = (int)lds_u1(o.ring + 72);
    int ip = (int)lds_u1(o.ring + 68) + o.j;
    ip += ip < 0 ? n : 0;
    ip -= ip >= n ? n : 0;
    const long long p = __double_as_longlong(lds_d1(o.ring + 48)) + ip;
    if constexpr (HAS_QU) {
      const double2 zs = lds_d2(o.ring + 32);
      double c2, s2;
      const int j = REGION == kWide ? near_turn(o.j, n) : o.j;
      const double dphi = pixel_dphi(bdl, lds_d1(o.ring), j, lds_d1(o.ring + 56));
      if (!spin2_small<PM>(zs.x, zs.y, dphi, bo, c2, s2)) {
        if constexpr (REGION != kWide) return false;
        const double2 far = spin2_far(zs.x, zs.y, dphi, bo.z, bo.sth);
        c2 = far.x;
        s2 = far.y;
      }
      v = turned_vals<MapT, LAYOUT>(ch, map, p, c2, s2);
    } else {
      v = raw_vals<MapT, LAYOUT>(ch, map, p);
    }
  }
  const float bvf = __ldg(bv);
#pragma unroll
  for (int c = 0; c < 4; ++c) {
    if (c >= ch.C) break;
    acc.add(c, nearest_term<HAS_QU, MapT, LAYOUT>(ch, c, v.v[c], bvf));
  }
  return true;
}

// ---------------------------------------------------------------------------
// One sample's window and table.
// ---------------------------------------------------------------------------

__device__ __forceinline__ void copy_ring(const RingRec* r, double theta_u, RingWin& w) {
  w.inv_dphi = __ldg(&r->inv_dphi);
  w.rta = __ldg(&r->ta) - theta_u;
  w.z = __ldg(&r->z);
  w.sth = __ldg(&r->sth);
  w.inv_dta = __ldg(&r->inv_dta);
  w.first = __ldg(&r->first);
  w.dphi = __ldg(&r->dphi);
  w.n = __ldg(&r->n);
}

// Window of one sample without a table, by the whole CTA.
static __device__ __noinline__ void plain_window(const RingRec* rt0, const SampleBlock* sb, RingWin* rings,
                                                 int4* s_hdr) {
  const int nr = sb->nr;
  for (int t = threadIdx.x; t < nr; t += blockDim.x) {
    const RingRec* r = rt0 + sb->ir_lo + t;
    int k0;
    double f0;
    ring_origin(sb->phi_u, __ldg(&r->phi0), __ldg(&r->dphi), __ldg(&r->inv_dphi), k0, f0);
    rings[t].f0 = f0;
    rings[t].k0 = k0;
    copy_ring(r, sb->theta_u, rings[t]);
  }
  if (threadIdx.x == 0) *s_hdr = make_int4(sb->ir_lo, nr > 0 ? nr - 1 : 0, 0, 0);
}

// Window of one sample, by the whole CTA: warp 0 places each ring in the
// sample's frame, counts its slots and lays them out, the other warps copy the
// rings' geometry.  ring_end[t] is the first slot past ring t, ring_of[i] the
// ring that holds slot 32 i (where the fill starts its search).
//
// Slots per ring: pixel j of ring r is a neighbour of queries between rings r
// - 1 and r + 1, so within d = max(0, |theta_r - theta_u| - spacing) of the
// disc's centre at the nearest; at that colatitude theta_q the beam disc
// (radius rbeam) reaches 2 asin(sqrt((sin^2(rbeam / 2) - sin^2(d / 2)) /
// (sin theta_u sin theta_q))) in longitude (2% margin), H pixels, and the
// query's two neighbours lie between -floor(f0 + H) - 1 and floor(f0 + H) + 1.
// (A ring that the disc holds whole comes out whole.)  The first rings about a pole
// take the ring table's reservation for any footprint of its reach.  (A pixel
// outside its ring's slots is still evaluated, directly; only the cost changes.)
template <int MODE>
__device__ __noinline__ void footprint_window(const RingRec* rt0, const SampleBlock* sb, int nside, int tab_cap,
                                              float rbeam, RingWin* rings, int* ring_end, unsigned short* ring_of,
                                              int4* s_hdr) {  // x first ring, y rings with a next one (0: no window),
                                                              // z table slots (0: no table)
  const int nr = sb->nr, ir_lo = sb->ir_lo;
  const RingRec* rt = rt0 + ir_lo;
  const double theta_u = sb->theta_u, phi_u = sb->phi_u;
  if (threadIdx.x >= 32) {
    for (int t = threadIdx.x - 32; t < nr; t += blockDim.x - 32) copy_ring(rt + t, theta_u, rings[t]);
    return;
  }
  const int lane = threadIdx.x;
  const float spacing = 0.9f / (float)nside;  // the widest step between rings
  const float hr = __sinf(0.5f * rbeam), inv_su = 1.f / (float)sb->su;
  int carry = 0;
  for (int b0 = 0; b0 < nr; b0 += 32) {
    const int t = b0 + lane;
    int own = 0;
    if (t < nr) {
      const RingRec* r = rt + t;
      const double inv = __ldg(&r->inv_dphi);
      int k0;
      double f0;
      ring_origin(phi_u, __ldg(&r->phi0), __ldg(&r->dphi), inv, k0, f0);
      rings[t].f0 = f0;
      rings[t].k0 = k0;
      own = __ldg(&r->cap);
      const float sq = (float)__ldg(&r->sth) - spacing;
      if (sq > 2.f * spacing) {
        const float d = fmaxf(0.f, fabsf((float)(__ldg(&r->ta) - theta_u)) - spacing);
        const float hd = __sinf(0.5f * d);
        const float q = fmaxf(0.f, hr * hr - hd * hd) * inv_su / sq;
        const float H = 2.04f * asinf(fminf(1.f, sqrtf(q))) * (float)inv;
        own = min(own, 2 * (int)((float)f0 + H) + 3);
      }
    }
    int v = own;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(0xffffffffu, v, o);
      if (lane >= o) v += y;
    }
    v += carry;
    if (t < nr) {
      const int off = v - own;
      rings[t].slots = (unsigned)(off + (own - 1) / 2) << 16 | (unsigned)((own - 1) & 0xffff);
      ring_end[t] = v;
      for (int i = (off + 31) >> 5; 32 * i < v && 32 * i < tab_cap; ++i) ring_of[i] = (unsigned short)t;
    }
    carry = __shfl_sync(0xffffffffu, v, 31);
  }
  const bool fits = carry <= tab_cap;
  if (lane == 0)
    *s_hdr = make_int4(ir_lo, (fits || MODE == TODGPU_NEAREST) && nr > 0 ? nr - 1 : 0, fits ? carry : 0, 0);
}

// Fill of the sample's value table, by the whole CTA.
template <int PM, bool HAS_QU, typename MapT, int LAYOUT>
__device__ __noinline__ void fill_table(const Chan<LAYOUT> ch, const MapRef map, const SampleBlock* sb,
                                        const RingWin* rings, const int* ring_end, const unsigned short* ring_of,
                                        int slots, const ValTable<MapT, LAYOUT> tab) {
  const Bore bo{sb->bz, sb->bsth};
  const double bdl = sb->bdl;
#pragma unroll 1
  for (int e = threadIdx.x; e < slots; e += blockDim.x) {
    int t = ring_of[e >> 5];
    while (e >= ring_end[t]) ++t;
    const RingWin& w = rings[t];
    const int j = e - (int)(w.slots >> 16), n = w.n;
    int ip = w.k0 + j;
    ip += ip < 0 ? n : 0;
    ip -= ip >= n ? n : 0;
    tab.store(ch, e, pixel_vals<PM, HAS_QU, MapT, LAYOUT>(ch, map, bo, w.z, w.sth,
                                                          HAS_QU ? pixel_dphi(bdl, w.f0, j, w.dphi) : 0.0,
                                                          w.first + ip));
  }
}

// What the pixel loops of a pass over the beam read, in shared memory: as a
// parameter it went through every thread's local memory once a sample.
template <typename MapT, int LAYOUT, typename VecT>
struct PixelLoop {
  const VecT* vec[3];  // component i of beam pixel s at vec[i][s ss]
  const float* vals;
  MapRef map;          // where there is no table
  unsigned rings;      // shared addresses of the window's rings and the table
  ValTable<MapT, LAYOUT> tab;
  int ss, n, nside;
  Chan<LAYOUT> ch;
};

template <class Acc>
struct LoopState {
  Acc acc;
  int s;
};

// Beam pixels s, s + kSumLanes, ... < n of one summation lane, as long as the
// window and table hold them: returns the sums and the first pixel that they
// do not hold (or one past the last).  Without calls: a call inside would
// spill the loop's registers.  Two pixels at a time: each is a chain of some 60
// dependent float64 operations, and two side by side hide what the warps of an
// SM alone do not.
//
// Bound (30' beam, S = 1512, nside 1024, 120k samples, float64 records): 5.30 ms
// with the map gathered and the spin-2 angle looked up per neighbour (677
// thread instructions an evaluation, L1 at 79%), 2.52 ms now, of which the
// table fill is 0.4 and the window 0.1; 294 instructions an evaluation, all parts of a
// sample counted, 66 float64 ones in this loop, issue slots 57% and the shared-memory data path 60-70% busy:
// leaving out 12 of 16 shared loads saved 5%, 22 of 66 float64 operations 13%.
// TABLE false: the same from the map (bound there: its loads, 12 a pixel with I, Q and
// U, and L1, see choose_shape).  It stands in for the direct evaluation, one pixel at a
// time out of line: 1000 pixels of a 45' beam at nside 4096, packed float32, 5000
// samples 362 us direct, 291 now; 16,000 pixels, I alone, nside 8192, 30' 5090, 1920.
template <int REGION, bool TABLE, bool HAS_QU, typename MapT, int PM, int LAYOUT, class Acc, typename VecT>
__device__ __forceinline__ LoopState<Acc> bilinear_loop(const PixelLoop<MapT, LAYOUT, VecT>* sp, const SampleBlock* blk,
                                                     int ir_lo, int nwin, LoopState<Acc> st) {
  const PixelLoop<MapT, LAYOUT, VecT> p = *sp;
  const unsigned sb = smem_u32(blk);
  const double theta_u = blk->theta_u, cu = blk->cu, su = blk->su, belt_inv = lds_d1(p.rings + 8);
  int s = st.s;
  Acc acc = st.acc;
#pragma unroll 1
  for (; s + kSumLanes < p.n; s += 2 * kSumLanes) {
    double x[2], y[2], z[2];
    rotate_frame<2>(sb, p.vec, {s * p.ss, (s + kSumLanes) * p.ss}, x, y, z);
    if (REGION != kBelt && PM == kParamsRef32 && (is_polar(z[0]) || is_polar(z[1]))) {
#pragma unroll
      for (int k = 0; k < 2; ++k)
        if (is_polar(z[k])) z[k] = polar_z(sb, p.vec, (s + k * kSumLanes) * p.ss);
    }
    Place o[2];
    bool ok = true;
#pragma unroll
    for (int k = 0; k < 2; ++k)
      ok = place_pixel<REGION, TABLE>(p.rings, ir_lo, nwin, p.nside, theta_u, cu, su, belt_inv, x[k], y[k], z[k], o[k]) && ok;
    if (!ok) break;
    if constexpr (TABLE) {
      add_placed<HAS_QU, MapT, LAYOUT>(p.ch, p.tab, o[0], __ldg(p.vals + s), acc);
      add_placed<HAS_QU, MapT, LAYOUT>(p.ch, p.tab, o[1], __ldg(p.vals + s + kSumLanes), acc);
    } else {
      const Bore bo{blk->bz, blk->bsth};
      if (!add_from_map<REGION, PM, HAS_QU, MapT, LAYOUT>(p.ch, p.map, bo, blk->bdl, o[0], __ldg(p.vals + s), acc))
        break;
      if (!add_from_map<REGION, PM, HAS_QU, MapT, LAYOUT>(p.ch, p.map, bo, blk->bdl, o[1],
                                                          __ldg(p.vals + s + kSumLanes), acc)) {
        s += kSumLanes;
        break;
      }
    }
  }
  if (s < p.n) {
    double x, y, z;
    rotate_frame<1>(sb, p.vec, {s * p.ss}, &x, &y, &z);
    if (REGION != kBelt && PM == kParamsRef32 && is_polar(z)) z = polar_z(sb, p.vec, s * p.ss);
    Place o;
    if (place_pixel<REGION, TABLE>(p.rings, ir_lo, nwin, p.nside, theta_u, cu, su, belt_inv, x, y, z, o)) {
      if constexpr (TABLE) {
        add_placed<HAS_QU, MapT, LAYOUT>(p.ch, p.tab, o, __ldg(p.vals + s), acc);
        s += kSumLanes;
      } else if (add_from_map<REGION, PM, HAS_QU, MapT, LAYOUT>(p.ch, p.map, Bore{blk->bz, blk->bsth}, blk->bdl, o,
                                                                __ldg(p.vals + s), acc)) {
        s += kSumLanes;
      }
    }
  }
  st.acc = acc;
  st.s = s;
  return st;
}

template <int REGION, bool HAS_QU, typename MapT, int PM, int LAYOUT, class Acc, typename VecT>
__device__ __forceinline__ LoopState<Acc> nearest_loop(const PixelLoop<MapT, LAYOUT, VecT>* sp, const SampleBlock* blk,
                                                    int ir_lo, int nwin, bool table, LoopState<Acc> st) {
  const PixelLoop<MapT, LAYOUT, VecT> p = *sp;
  const unsigned sb = smem_u32(blk);
  const Bore bo{blk->bz, blk->bsth};
  const double bdl = blk->bdl;
  int s = st.s;
  Acc acc = st.acc;
#pragma unroll 1
  for (; s + kSumLanes < p.n; s += 2 * kSumLanes) {
    double x[2], y[2], z[2];
    rotate_frame<2>(sb, p.vec, {s * p.ss, (s + kSumLanes) * p.ss}, x, y, z);
    NearPlace o[2];
    bool ok = true;
#pragma unroll
    for (int k = 0; k < 2; ++k)
      ok = place_nearest<REGION>(p.rings, ir_lo, nwin, p.nside, x[k], y[k], z[k], o[k]) && ok;
    if (!ok) break;
    if (!add_nearest<REGION, PM, HAS_QU, MapT, LAYOUT>(p.ch, p.map, bo, bdl, p.tab, table, o[0], p.vals + s, acc)) break;
    if (!add_nearest<REGION, PM, HAS_QU, MapT, LAYOUT>(p.ch, p.map, bo, bdl, p.tab, table, o[1], p.vals + s + kSumLanes,
                                               acc)) {
      s += kSumLanes;
      break;
    }
  }
  if (s < p.n) {
    double x, y, z;
    rotate_frame<1>(sb, p.vec, {s * p.ss}, &x, &y, &z);
    NearPlace o;
    if (place_nearest<REGION>(p.rings, ir_lo, nwin, p.nside, x, y, z, o) &&
        add_nearest<REGION, PM, HAS_QU, MapT, LAYOUT>(p.ch, p.map, bo, bdl, p.tab, table, o, p.vals + s, acc))
      s += kSumLanes;
  }
  st.acc = acc;
  st.s = s;
  return st;
}

// Out of line: the calls inside would spill the other forms' registers.
template <int MODE, bool TABLE, bool HAS_QU, typename MapT, int PM, int LAYOUT, class Acc, typename VecT>
__device__ __noinline__ LoopState<Acc> wide_loop(const PixelLoop<MapT, LAYOUT, VecT>* p, const SampleBlock* sb,
                                                 int ir_lo, int nwin, bool table, LoopState<Acc> st) {
  if constexpr (MODE == TODGPU_NEAREST) {
    if (TABLE && !sb->wide)
      return nearest_loop<kAnywhere, HAS_QU, MapT, PM, LAYOUT, Acc, VecT>(p, sb, ir_lo, nwin, false, st);
    return nearest_loop<kWide, HAS_QU, MapT, PM, LAYOUT, Acc, VecT>(p, sb, ir_lo, nwin, table, st);
  } else
    return bilinear_loop<kWide, TABLE, HAS_QU, MapT, PM, LAYOUT, Acc, VecT>(p, sb, ir_lo, nwin, st);
}

template <int MODE, bool TABLE, bool HAS_QU, typename MapT, int PM, int LAYOUT, class Acc, typename VecT>
__device__ __forceinline__ LoopState<Acc> pixel_loop(const PixelLoop<MapT, LAYOUT, VecT>* p, const SampleBlock* sb,
                                                     const int4& hdr, int nside, const LoopState<Acc>& st) {
  const bool table = TABLE && hdr.z > 0;
  // (nearest: a sample whose footprint the launch's table does not hold reads the map
  // there too, so that the loops below have one source of values: 1% of a nearest call)
  if (TABLE ? sb->wide || (MODE == TODGPU_NEAREST && !table) : sb->far)
    return wide_loop<MODE, TABLE, HAS_QU, MapT, PM, LAYOUT, Acc, VecT>(p, sb, hdr.x, hdr.y, table, st);
  // the window's rings all in the belt (rings nside to 3 nside)?
  const bool belt = hdr.x >= nside && hdr.x + hdr.y <= 3 * nside;
  if constexpr (MODE == TODGPU_NEAREST) {
    if (belt) return nearest_loop<kBelt, HAS_QU, MapT, PM, LAYOUT, Acc, VecT>(p, sb, hdr.x, hdr.y, TABLE, st);
    return nearest_loop<kAnywhere, HAS_QU, MapT, PM, LAYOUT, Acc, VecT>(p, sb, hdr.x, hdr.y, TABLE, st);
  } else {
    if (belt) return bilinear_loop<kBelt, TABLE, HAS_QU, MapT, PM, LAYOUT, Acc, VecT>(p, sb, hdr.x, hdr.y, st);
    return bilinear_loop<kAnywhere, TABLE, HAS_QU, MapT, PM, LAYOUT, Acc, VecT>(p, sb, hdr.x, hdr.y, st);
  }
}

// ---------------------------------------------------------------------------
// The sample loop.
// ---------------------------------------------------------------------------

// Beams of more than kBeamChunkMin pixels run in chunks of beam_chunk consecutive
// pixels, each with its own centre, frame and window: a far-sidelobe beam's whole
// footprint holds 1e5 to 1e6 map pixels, a chunk of a beam in kernels.beam_order a
// patch that fits a table.  (Float64 sums only: the order of the float32 Kahan sums is
// part of their result.)  Without Q and U there is no table to fit, and longer chunks
// prepare each sample less often (nearest, 100,000 pixels of 1 degree, nside 1024,
// float32 parameters, 1000 samples: 1024 pixels 2285 us, 4096 1840; with Q and U 2797
// and 1963, but 3430 and 5230 for an annulus of 3 to 10 degrees, whose map pixels then
// leave L1).
constexpr int kBeamChunkMin = 16384;
template <bool HAS_QU>
constexpr int beam_chunk() { return HAS_QU ? 1024 : 4096; }

// What a CTA keeps from sample to sample of a run besides the pixel loop's
// state, in shared memory: in registers it was spilled, and an L1 that the tables
// leave little of sent the reloads to L2.  The batched kernel, with its tiles
// and jobs to keep as well, gains most: six detectors over a float32 map 4330 ->
// 3845 us, far sidelobes in pieces 4710 -> 4480; nearest 1872 -> 1827, packed
// float32 records 1925 -> 1905, the 30' float64 beam 2478 -> 2486.
struct RunState {
  long long t_begin, t_step, tile, total;  // tiles t_begin, t_begin + t_step, ...; samples in all of them
  double cx, cy, cz, rbeam;
  unsigned long long nerr;
  long long b[kPrep];                      // the samples being prepared or summed
  // sample q of the run
  __device__ __forceinline__ long long sample(long long q) const volatile {
    const long long n = tile, ti = n == 1 ? q : q / n;
    return (t_begin + ti * t_step) * n + (q - ti * n);
  }
};

// Samples of tiles t = t_begin, t_begin + t_step, ... < t_end of one job (one
// beam entry over one batch of samples; tile t holds samples [t tile,
// min(B, (t + 1) tile))), by the whole CTA.  All threads of the CTA must call
// it together.
template <int MODE, bool TABLE, bool HAS_QU, typename MapT, int PM, int LAYOUT, bool TILES>
__device__ void run_samples(const KArgs& a, long long t_begin, long long t_end, long long t_step, long long tile,
                            unsigned char* smem_raw, double* s_red, SampleBlock* s_blk, ExactBlock* s_exact,
                            int4* s_hdr) {
  using Acc = typename std::conditional<MapTraits<MapT>::packed, AccKahan, Acc64>::type;
  using VecT = typename std::conditional<PM == kParamsRef32, float, double>::type;
  const Chan<LAYOUT> ch(a);
  const int NT = blockDim.x, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  RingWin* rings = reinterpret_cast<RingWin*>(smem_raw);
  int* ring_end = reinterpret_cast<int*>(smem_raw + sizeof(RingWin) * (size_t)a.ring_cap);
  unsigned short* ring_of = reinterpret_cast<unsigned short*>(smem_raw + window_bytes(a.ring_cap));
  unsigned char* tab_mem = smem_raw + window_bytes(a.ring_cap) + ring_of_bytes(a.tab_cap);
  const ValTable<MapT, LAYOUT> tab{smem_u32(tab_mem), a.tab_cap};
  double* xchg = reinterpret_cast<double*>(tab_mem);  // lane sums of 256-thread CTAs, after the table's last use
  using Loop = PixelLoop<MapT, LAYOUT, VecT>;
  __shared__ __align__(16) unsigned char loop_mem[sizeof(Loop)];
  Loop* loop = reinterpret_cast<Loop*>(loop_mem);
  const int nside = (int)a.nside;
  // samples of this CTA: whole tiles, but the job's last tile may be short
  if (t_begin >= t_end) return;
  const long long ntile = (t_end - t_begin + t_step - 1) / t_step;
  const long long t_last = t_begin + (ntile - 1) * t_step;
  const long long total = (ntile - 1) * tile + min(tile, a.B - t_last * tile);
  __shared__ RunState run_mem;
  volatile RunState* run = &run_mem;
  if (tid == 0) run->nerr = 0;
  const int S = (int)a.S;
  const int step = S > kBeamChunkMin && !MapTraits<MapT>::packed ? beam_chunk<HAS_QU>() : S;
  for (int s0 = 0; s0 < S; s0 += step) {
    const int s1 = min(S, s0 + step);
    double cx, cy, cz, rbeam;
    beam_extent<PM>(a, s0, s1, s_red, cx, cy, cz, rbeam);
    rbeam += 1e-5;  // slack for the float32 parameter rounding
    // the ring table reserves per-ring slots for footprints up to its reach:
    // a stencil neighbour's centre lies within 1.7/nside rad of its query (one
    // ring spacing plus one pixel width; the opposite pair around a pole
    // within twice the colatitude of ring 1)
    const bool window = a.ring_table != nullptr &&
                        rbeam + 2.0 / (double)a.nside <= __ldg(&static_cast<const RingRec*>(a.ring_table)[0].ta);
    const int n = s1 - s0;
    if (tid == 0) {
      const VecT* vec = static_cast<const VecT*>(a.vec) + (long long)s0 * a.vec_ss;
      if (TILES) {
        run->t_begin = t_begin;
        run->t_step = t_step;
        run->tile = tile;
        run->total = total;
      }
      run->cx = cx;
      run->cy = cy;
      run->cz = cz;
      run->rbeam = rbeam;
      for (int k = 0; k < 3; ++k) loop->vec[k] = vec + k * a.vec_si;
      loop->vals = a.beam + s0;
      loop->map = MapRef{a.map, a.map_stride};
      loop->rings = smem_u32(rings);
      loop->tab = tab;
      loop->ss = a.vec_ss;
      loop->n = n;
      loop->nside = nside;
      loop->ch = ch;
    }
    // the nearest rule's margin on ring boundaries (place_nearest) holds away
    // from the poles, where a ring's width in z vanishes
    const float reach = (float)rbeam;
    const double polar = MODE == TODGPU_NEAREST ? 0.01 : -4.0;
    for (long long q0 = 0;; q0 += kPrep) {
      __syncthreads();  // the previous samples' blocks are no longer read; the run's state is written
      const int nq = (int)min((long long)kPrep, (TILES ? run->total : total) - q0);
      if (nq <= 0) break;
      if (tid < nq) {
        const long long b = TILES ? run->sample(q0 + tid) : t_begin + (q0 + tid) * t_step;
        if (TILES) run->b[tid] = b;
        prepare_sample<PM, TABLE>(a, b, HAS_QU, run->cx, run->cy, run->cz, run->rbeam, window, polar, s_blk[tid],
                           s_exact != nullptr ? s_exact + tid : nullptr);
      }
      __syncthreads();
#pragma unroll 1
      for (int i = 0; i < nq; ++i) {
        const SampleBlock* sb = s_blk + i;
        // the warps' sums alternate between two sets: one sample's are read
        // while the next sample's may already be written
        double* red = s_red + 16 * (i & 1);
        int4 hdr = make_int4(0, 0, 0, 0);
        if (window) {
          const RingRec* rt = static_cast<const RingRec*>(a.ring_table);
          if constexpr (TABLE)
            footprint_window<MODE>(rt, sb, nside, a.tab_cap, reach, rings, ring_end, ring_of, s_hdr);
          else
            plain_window(rt, sb, rings, s_hdr);
          __syncthreads();
          hdr = *s_hdr;
          if (TABLE && hdr.z > 0) {
            fill_table<PM, HAS_QU, MapT, LAYOUT>(ch, MapRef{a.map, a.map_stride}, sb, rings, ring_end, ring_of,
                                                 hdr.z, tab);
            __syncthreads();
          }
        }
        // Summation lane l (of kSumLanes) takes the beam pixels l, l +
        // kSumLanes, ... of the pass; thread t holds lanes t and (128-thread
        // CTAs) t + 128.  Lane sums l and l + 128 are added, then the 128
        // sums per warp, then the four warps': the TOD does not depend on
        // the CTA's thread count.
        double keep[4] = {0.0, 0.0, 0.0, 0.0};
        Acc acc;
#pragma unroll 1
        for (int l = tid; l < kSumLanes; l += NT) {
          LoopState<Acc> st{Acc(), l};
          // pixels that the window and table do not hold are evaluated here,
          // each in its place in the sum
          while (st.s < n) {
            if (hdr.y > 0) st = pixel_loop<MODE, TABLE, HAS_QU, MapT, PM, LAYOUT, Acc, VecT>(loop, sb, hdr, nside, st);
            if (st.s < n) {
              const VecT* v = static_cast<const VecT*>(a.vec) + (s0 + (long long)st.s) * a.vec_ss;
              const float bvf = a.beam[s0 + st.s];
              Contrib r;
              if constexpr (MODE == TODGPU_BILINEAR)
                r = bilinear_direct<PM, HAS_QU, MapT, LAYOUT, VecT>(a, sb, v);
              else
                r = nearest_exact<PM, HAS_QU, MapT, LAYOUT, VecT>(a, sb, s_exact + i, v[0], v[a.vec_si], v[2 * a.vec_si], bvf);
              if (r.err) {
                atomicAdd(&run_mem.nerr, (unsigned long long)r.err);
              } else {
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                  if (c >= ch.C) break;
                  if constexpr (MODE == TODGPU_BILINEAR)
                    accumulate<MapT>(st.acc, c, (ValT<MapT>)r.v[c], bvf);
                  else
                    st.acc.add(c, r.v[c]);
                }
              }
              st.s += kSumLanes;
            }
          }
          acc = st.acc;
          if (NT < kSumLanes) {
#pragma unroll
            for (int c = 0; c < 4; ++c) keep[c] = l == tid ? acc.total(c) : keep[c] + acc.total(c);
          }
        }
        if (NT == kSumLanes) {
          __syncthreads();  // the table is no longer read
          if (tid >= kMeanLanes) {
#pragma unroll
            for (int c = 0; c < 4; ++c)
              if (c < ch.C) xchg[c * kMeanLanes + tid - kMeanLanes] = acc.total(c);
          }
          __syncthreads();
          if (tid < kMeanLanes) {
#pragma unroll
            for (int c = 0; c < 4; ++c)
              if (c < ch.C) keep[c] = acc.total(c) + xchg[c * kMeanLanes + tid];
          }
        }
        if (tid < kMeanLanes) {
#pragma unroll
          for (int c = 0; c < 4; ++c) {
            if (c >= ch.C) break;
            const double v = warp_sum(keep[c]);
            if (lane == 0) red[warp * 4 + c] = v;
          }
        }
        __syncthreads();  // the sums are written and the table, window and header free
        if (tid < a.C) {
          const long long b = TILES ? run->b[i] : t_begin + (q0 + i) * t_step;
          double v = 0.0;
          for (int k = 0; k < kMeanLanes / 32; ++k) v += red[k * 4 + tid];
          a.tod[(long long)tid * a.tod_stride + b] += v;
        }
      }
    }
  }
  __syncthreads();  // every count is in; shared memory may be reused by the next job
  if (tid == 0 && a.err != nullptr && run->nerr) atomicAdd(a.err, run->nerr);
}

template <int MODE, bool TABLE, bool HAS_QU, typename MapT, int PM, int LAYOUT>
__global__ void __maxnreg__(kRegs) gather_accum_kernel(const __grid_constant__ KArgs a) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ double s_red[(kSumLanes / 32) * 4];
  __shared__ SampleBlock s_blk[kPrep];
  __shared__ ExactBlock s_exact[MODE == TODGPU_NEAREST ? kPrep : 1];
  __shared__ int4 s_hdr;
  run_samples<MODE, TABLE, HAS_QU, MapT, PM, LAYOUT, false>(a, blockIdx.x, a.B, gridDim.x, 1, smem_raw, s_red, s_blk,
                                                     MODE == TODGPU_NEAREST ? s_exact : nullptr, &s_hdr);
}

// Many jobs (detectors: each its own beam, pointing, output and length) in
// one persistent launch.  Job j's samples form tiles of `tile` samples; the
// tiles of all jobs are numbered job by job (tiles_before[j] = tiles of jobs
// 0..j-1) and CTA k takes tiles k, k + G, k + 2G, ... (G = grid size), as one
// launch per job with its samples interleaved over the CTAs would, without a
// launch boundary between jobs.  CTAs running at the same time then work on
// neighbouring samples of one job (the same sky region, shared in L2), and
// every CTA gets an equal share of every job whatever its beam size.  `tile`
// sets how many consecutive samples a CTA takes at a time.  The descriptors
// travel in the kernel parameters; each CTA copies the current job's into
// shared memory, so that the sample loop reads its fields with plain shared
// loads rather than parameter loads at a job index known only at run time
// (5% of the batched launch).
constexpr int kMaxBatchJobs = 96;
struct BatchParams {
  int njobs;
  long long tile;
  long long tiles_before[kMaxBatchJobs + 1];
  KArgs job[kMaxBatchJobs];
};

template <int MODE, bool TABLE, bool HAS_QU, typename MapT, int PM, int LAYOUT>
__global__ void __maxnreg__(kRegs) gather_batched_kernel(const __grid_constant__ BatchParams p) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ double s_red[(kSumLanes / 32) * 4];
  __shared__ SampleBlock s_blk[kPrep];
  __shared__ ExactBlock s_exact[MODE == TODGPU_NEAREST ? kPrep : 1];
  __shared__ int4 s_hdr;
  __shared__ __align__(16) KArgs s_job;
  const long long G = gridDim.x, k = blockIdx.x;
  for (int j = 0; j < p.njobs; ++j) {
    const long long ntiles = p.tiles_before[j + 1] - p.tiles_before[j];
    // first tile of job j that falls to this CTA: global index = k (mod G)
    const long long t0 = ((k - p.tiles_before[j]) % G + G) % G;
    if (t0 < ntiles) {
      __syncthreads();
      if (threadIdx.x < (int)(sizeof(KArgs) / 8))
        reinterpret_cast<unsigned long long*>(&s_job)[threadIdx.x] =
            reinterpret_cast<const unsigned long long*>(&p.job[j])[threadIdx.x];
      __syncthreads();
      run_samples<MODE, TABLE, HAS_QU, MapT, PM, LAYOUT, true>(s_job, t0, ntiles, G, p.tile, smem_raw, s_red, s_blk,
                                                        MODE == TODGPU_NEAREST ? s_exact : nullptr, &s_hdr);
    }
  }
}

// ---------------------------------------------------------------------------
// Host-side launch templates.
// ---------------------------------------------------------------------------

inline int sm_count() {
  static int count = 0;
  static std::once_flag once;
  std::call_once(once, [] {
    int dev = 0;
    if (cudaGetDevice(&dev) == cudaSuccess) cudaDeviceGetAttribute(&count, cudaDevAttrMultiProcessorCount, dev);
    if (count <= 0) count = 148;
  });
  return count;
}

// Shared memory per SM on B200, what the driver keeps per CTA, and a bound of
// the kernels' static shared memory (sample blocks, partial sums, the batched
// job descriptor).
constexpr size_t kSmemPerSM = 228 * 1024;
constexpr size_t kSmemPerCTAMax = 227 * 1024;
constexpr size_t kSmemPerCTAReserved = 1024;
template <int MODE>
constexpr size_t static_smem() {
  return kPrep * (sizeof(SampleBlock) + (MODE == TODGPU_NEAREST ? sizeof(ExactBlock) : 0)) + 1024;
}

// Window rings a launch reserves for a call.  A request of N slots is a beam disc of
// radius r with at least 3.15 (r nside)^2 slots (kernels.footprint_slots), so r
// nside <= sqrt(N / 3.15), and such a disc crosses at most 3 r nside + 4 rings
// of the RING scheme (ring spacing at least 2 / (3 nside) in colatitude, plus
// the rings either side); the default table reserves kRingCap.  A request is the
// whole beam's: a chunk's window has fewer rings (kRingCap with its default table).
inline int ring_cap_for(int requested, bool chunked, int slots) {
  if (chunked ? slots > 0 : requested <= 0) return kRingCap;
  if (requested <= 0) return kRingChunk;
  return std::min(chunked ? kRingChunk : kRingMax, (int)std::ceil(3.0 * std::sqrt(requested / 3.15)) + 6);
}
constexpr size_t align16(size_t x) { return (x + 15) & ~size_t(15); }

// (Nearest: only for turned Q and U values.)
template <int MODE, bool HAS_QU>
constexpr bool may_have_table() { return MODE == TODGPU_BILINEAR || HAS_QU; }

// Whether a value table of `slots` (`bytes` in all) pays for a pass over `pixels`
// beam pixels.  Filling a slot costs a map read and a turned (Q, U), more as fewer
// CTAs share an SM; a pixel read from the table saves four of them.  Bilinear, I, Q
// and U, 5000 samples unless said, microseconds with the table / without:
//   nside 2048, 30', 1263 slots (30 KB), 20,000 samples: 200 pixels 479 / 344,
//     400 pixels 515 / 516, 1600 pixels 673 / 1022;
//   nside 4096, 30', 4500 slots (108 KB): 1000 pixels 608 / 300, 4000 pixels
//     802 / 642, 16,000 pixels 1548 / 2072;
//   packed float32, nside 4096, 45', 9500 slots (114 KB): 4000 pixels 1057 / 668,
//     16,000 pixels 1685 / 2201;
//   I alone, nside 4096, 45', 80 KB: 4000 pixels 691 / 544, 16,000 pixels 1315 /
//     1681; nside 8192, 30', 136 KB: 16,000 pixels 2323 / 1778.
// So: as many slots a pixel as CTAs with such a table fit an SM, four at most.
template <int MODE, bool HAS_QU>
bool table_pays(long long slots, long long pixels, size_t bytes) {
  if (!may_have_table<MODE, HAS_QU>()) return false;
  // nearest reads one value per beam pixel: a table pays when the footprint
  // has fewer pixels than the beam
  if (MODE == TODGPU_NEAREST) return slots <= pixels;
  return slots <= (long long)std::min<size_t>(4, kSmemPerSM / (bytes + 8 * 1024)) * pixels;
}

// Shape of a launch: threads per CTA, window rings, table slots, dynamic
// shared memory.
struct Shape {
  int nt = 128, ring_cap = 1, tab_cap = 0;
  size_t smem = 0;
};

inline int ctas_per_sm(int nt, size_t smem) {  // smem: static and dynamic
  const size_t per = smem + kSmemPerCTAReserved;
  return (int)std::min<size_t>(kThreadsSM / nt, kSmemPerSM / per);
}

// What a launch asks for: the window's rings and the table's slots, slot bytes,
// components, samples, beam pixels per pass, the fewest threads per CTA.
struct Wants {
  int rings = 1, slots = 0, slot = 0, C = 1;
  long long samples = 0, pixels = 0;
  int min_nt = 128;
  size_t fixed = 0;  // static shared memory
  bool map_reads = false;  // bilinear with a window
};

// Shared memory left for a table, and whether one of `slots` fits it.
inline bool table_fits(int slots, int slot, size_t fixed, int rings) {
  const size_t used = fixed + window_bytes(rings) + 1024;
  return used < kSmemPerCTAMax && (size_t)slots <= (kSmemPerCTAMax - used) / (slot + 1);
}

inline Shape choose_shape(const Wants& w) {
  Shape best;
  int best_threads = 0;
  for (int nt = w.min_nt; nt <= kSumLanes; nt *= 2) {
    Shape s;
    s.nt = nt;
    s.ring_cap = w.rings;
    const size_t xchg = nt > kMeanLanes ? sizeof(double) * kMeanLanes * (size_t)w.C : 0;
    const size_t head = window_bytes(s.ring_cap);
    s.tab_cap = table_fits(w.slots, w.slot, w.fixed, w.rings) ? (w.slots + 1) & ~1 : 0;
    s.smem = align16(head + ring_of_bytes(s.tab_cap) + std::max(xchg, (size_t)w.slot * s.tab_cap));
    const int threads = nt * ctas_per_sm(nt, s.smem + w.fixed);
    // without a table bilinear reads the map itself: 256-thread CTAs have fewer
    // samples in flight on an SM, whose footprints then stay in L1 (16,000 pixels of a
    // 30' beam at nside 8192, 5000 samples: 5020 us in 128-thread CTAs, 2290; 1000
    // pixels 297 and 316 at nside 4096)
    if (w.map_reads && s.tab_cap == 0 && w.pixels >= 2048 && nt < kSumLanes) continue;
    const bool idle = w.samples * nt <= (long long)kThreadsSM * sm_count() && w.pixels >= nt;
    if (threads > best_threads || (threads == best_threads && idle)) {
      best = s;
      best_threads = threads;
    }
  }
  return best;
}

// A job's part in its launch: window rings, table slots (0: no value table).  The
// request is the caller's, else 32 KiB of the float64 or float32 pairs earlier
// versions kept.  A table that no CTA can hold is not made (no sample would fit it).
struct JobWants {
  int rings = 1, slots = 0;
};
template <int MODE, bool HAS_QU, typename MapT>
JobWants job_wants(const KArgs& k) {
  JobWants j;
  if (k.ring_table == nullptr) return j;
  constexpr bool packed = MapTraits<MapT>::packed;
  const bool chunked = k.S > kBeamChunkMin && !packed;
  const long long pixels = chunked ? beam_chunk<HAS_QU>() : k.S;
  const int slot = slot_bytes(packed, k.C);
  const int req = k.tab_req > 0 && !chunked ? k.tab_req : (packed ? 2 * kTabCapDefault : kTabCapDefault);
  const bool holds = !chunked || (HAS_QU && (long long)k.tab_req * pixels <= req * (long long)k.S);
  if (holds && table_pays<MODE, HAS_QU>(req, pixels, (size_t)req * slot)) j.slots = req;
  j.rings = ring_cap_for(k.tab_req, chunked, j.slots);
  if (!table_fits(j.slots, slot, static_smem<MODE>(), j.rings)) {
    j.slots = 0;
    j.rings = ring_cap_for(k.tab_req, chunked, 0);
  }
  return j;
}

// One job's part in what its launch asks for (the most any job does).  `tables`: the
// launch has tables, and only the jobs with one decide on its window.
template <int MODE, bool HAS_QU, typename MapT>
void add_wants(Wants& w, const KArgs& k, bool tables) {
  const JobWants j = job_wants<MODE, HAS_QU, MapT>(k);
  if (!tables || j.slots > 0) w.rings = std::max(w.rings, j.rings);
  w.slots = std::max(w.slots, j.slots);
  w.slot = slot_bytes(MapTraits<MapT>::packed, k.C);
  w.C = k.C;
  w.fixed = static_smem<MODE>();
  w.map_reads = MODE == TODGPU_BILINEAR && k.ring_table != nullptr;
  w.samples += k.B;
  w.pixels = std::max(w.pixels, k.S > kBeamChunkMin && !MapTraits<MapT>::packed
                                    ? (long long)beam_chunk<HAS_QU>() : (long long)k.S);
  w.min_nt = std::max(w.min_nt, k.flags_wide ? 256 : 128);
}

// A kernel's opt-in to more than 48 KB of dynamic shared memory, once per device: the
// attribute belongs to the current device's copy of the kernel, so a process-wide
// flag would leave a second GPU's launches failing.
class SmemOptIn {
 public:
  template <typename Bytes>
  cudaError_t operator()(const void* kern, Bytes bytes) {  // bytes(): asked once per device
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    const unsigned long long bit = dev < 64 ? 1ull << dev : 0;
    if (e != cudaSuccess || (done_.load() & bit)) return e;
    e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes());
    if (e == cudaSuccess) done_.fetch_or(bit);
    return e;
  }

 private:
  std::atomic<unsigned long long> done_{0};
};

// All that the kernel's static shared memory leaves of a CTA's.
template <typename Kern>
int allow_smem(Kern kern, SmemOptIn& opt_in) {
  const cudaError_t e = opt_in(reinterpret_cast<const void*>(kern), [kern] {
    cudaFuncAttributes fa;
    return cudaFuncGetAttributes(&fa, kern) == cudaSuccess ? (int)(kSmemPerCTAMax - fa.sharedSizeBytes) : -1;
  });
  return e == cudaSuccess ? TODGPU_OK : cuda_fail(e, "kernel shared-memory attributes");
}

template <int MODE, bool TABLE, bool HAS_QU, typename MapT, int PM, int LAYOUT>
int launch_gather(KArgs k, const Wants& w, const Shape& s, cudaStream_t stream) {
  auto kern = gather_accum_kernel<MODE, TABLE, HAS_QU, MapT, PM, LAYOUT>;
  static SmemOptIn opt_in;
  const int rc = allow_smem(kern, opt_in);
  if (rc != TODGPU_OK) return rc;
  k.ring_cap = s.ring_cap;
  k.tab_cap = s.tab_cap;
  const long long max_blocks = (long long)sm_count() * ctas_per_sm(s.nt, s.smem + w.fixed);
  const int grid = (int)std::max(1LL, std::min(k.B, max_blocks));
  kern<<<grid, s.nt, s.smem, stream>>>(k);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return cuda_fail(e, "gather_accum_kernel launch");
  return TODGPU_OK;
}

static_assert(sizeof(BatchParams) <= 32000, "batched descriptors must fit the kernel parameter space");
static_assert(sizeof(KArgs) % 8 == 0 && sizeof(KArgs) / 8 <= 128, "KArgs copied as 8-byte words, one per thread");

// Batched launch: descriptors of up to kMaxBatchJobs jobs per launch, in one
// CTA shape, sized for the largest table any job asks for.
template <int MODE, bool TABLE, bool HAS_QU, typename MapT, int PM, int LAYOUT>
int launch_shape(BatchParams& bp, const Wants& w, const Shape& s, cudaStream_t stream) {
  auto kern = gather_batched_kernel<MODE, TABLE, HAS_QU, MapT, PM, LAYOUT>;
  static SmemOptIn opt_in;
  const int rc = allow_smem(kern, opt_in);
  if (rc != TODGPU_OK) return rc;
  for (int j = 0; j < bp.njobs; ++j) {
    bp.job[j].tab_cap = s.tab_cap;
    bp.job[j].ring_cap = s.ring_cap;
  }
  const long long max_blocks = (long long)sm_count() * ctas_per_sm(s.nt, s.smem + w.fixed);
  const int grid = (int)std::max(1LL, std::min(bp.tiles_before[bp.njobs], max_blocks));
  kern<<<grid, s.nt, s.smem, stream>>>(bp);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return cuda_fail(e, "gather_batched_kernel launch");
  return TODGPU_OK;
}
template <int MODE, bool HAS_QU, typename MapT, int PM, int LAYOUT>
int launch_batched(BatchParams& bp, cudaStream_t stream) {
  if (bp.tiles_before[bp.njobs] == 0) return TODGPU_OK;
  Wants w;
  bool tables = false;
  for (int j = 0; j < bp.njobs; ++j) tables = tables || job_wants<MODE, HAS_QU, MapT>(bp.job[j]).slots > 0;
  for (int j = 0; j < bp.njobs; ++j) add_wants<MODE, HAS_QU, MapT>(w, bp.job[j], tables);
  const Shape s = choose_shape(w);
  if constexpr (may_have_table<MODE, HAS_QU>())
    if (s.tab_cap > 0) return launch_shape<MODE, true, HAS_QU, MapT, PM, LAYOUT>(bp, w, s, stream);
  return launch_shape<MODE, false, HAS_QU, MapT, PM, LAYOUT>(bp, w, s, stream);
}

// A batch in launches of jobs whose own shapes keep equally many threads on an
// SM: in one launch the widest footprint's table sets every job's shape (six
// detectors, 25' to 35' beams over packed float32 records at nside 2048, 1.4 M
// samples: 34.4 ms in one launch, 29.6 as one launch per detector, 30.2 in two
// groups).  A group gets a launch of its own only where it has kSplitWaves tiles per resident
// CTA, so that the ends of the launches, half a tile each on average, stay a few
// percent of it (the same detectors with 0.14 M samples in tiles of 16 stay in one
// launch); smaller groups join the next narrower shape's.
constexpr int kSplitWaves = 16;
template <int MODE, bool HAS_QU, typename MapT, int PM, int LAYOUT>
int launch_alike(BatchParams& bp, cudaStream_t stream) {
  int threads[kMaxBatchJobs], ctas[kMaxBatchJobs];  // threads and CTAs per SM of a job's own shape
  bool alike = true;
  for (int j = 0; j < bp.njobs; ++j) {
    Wants w;
    add_wants<MODE, HAS_QU, MapT>(w, bp.job[j], false);
    w.samples = 1LL << 40;
    const Shape s = choose_shape(w);
    ctas[j] = ctas_per_sm(s.nt, s.smem + w.fixed);
    threads[j] = s.nt * ctas[j];
    alike = alike && threads[j] == threads[0];
  }
  if (alike) return launch_batched<MODE, HAS_QU, MapT, PM, LAYOUT>(bp, stream);
  // groups from the most threads down; group[j] counts up
  int group[kMaxBatchJobs], groups = 0;
  long long tiles = 0, enough = 0;
  for (int below = INT_MAX;;) {
    int t = 0, fewest = INT_MAX;  // CTAs: the group's widest job sets its shape
    for (int j = 0; j < bp.njobs; ++j)
      if (threads[j] < below) t = std::max(t, threads[j]);
    if (t == 0) break;
    for (int j = 0; j < bp.njobs; ++j)
      if (threads[j] == t) {
        group[j] = groups;
        fewest = std::min(fewest, ctas[j]);
        tiles += bp.tiles_before[j + 1] - bp.tiles_before[j];
      }
    below = t;
    enough = (long long)kSplitWaves * sm_count() * fewest;
    if (tiles >= enough) {
      ++groups;
      tiles = 0;
    }
  }
  // what is left over at the end joins the last full group
  const int last = std::max(0, groups - 1);
  BatchParams part;
  for (int g = 0; g <= last; ++g) {
    part.njobs = 0;
    part.tile = bp.tile;
    part.tiles_before[0] = 0;
    for (int j = 0; j < bp.njobs; ++j)
      if (std::min(group[j], last) == g) {
        part.job[part.njobs] = bp.job[j];
        part.tiles_before[part.njobs + 1] =
            part.tiles_before[part.njobs] + bp.tiles_before[j + 1] - bp.tiles_before[j];
        ++part.njobs;
      }
    const int rc = launch_batched<MODE, HAS_QU, MapT, PM, LAYOUT>(part, stream);
    if (rc != TODGPU_OK) return rc;
  }
  return TODGPU_OK;
}

// The jobs of bp that have a table (or have none), in order.
template <int MODE, bool HAS_QU, typename MapT>
void pick_jobs(const BatchParams& bp, bool table, BatchParams& out) {
  out.njobs = 0;
  out.tile = bp.tile;
  out.tiles_before[0] = 0;
  for (int j = 0; j < bp.njobs; ++j) {
    if ((job_wants<MODE, HAS_QU, MapT>(bp.job[j]).slots > 0) != table) continue;
    out.job[out.njobs] = bp.job[j];
    out.tiles_before[out.njobs + 1] = out.tiles_before[out.njobs] + bp.tiles_before[j + 1] - bp.tiles_before[j];
    ++out.njobs;
  }
}

// Jobs without a table -- sparse beams, footprints beyond one CTA's memory -- have a
// launch of their own where they are enough work for it, and never decide on the
// others' table and window: one footprint too large for a table took it from every job
// of its launch (six beams of 1500 pixels, 30', nside 2048, 20,000 samples each, alone
// 3.29 ms; with a seventh of 8000 pixels and 2 degrees and 400 samples 9.91, now 4.98,
// and 20,000 samples 17.7, now 11.0).
template <int MODE, bool HAS_QU, typename MapT, int PM, int LAYOUT>
int launch_grouped(BatchParams& bp, cudaStream_t stream) {
  int with = 0;
  long long without = 0;  // tiles of the jobs without a table
  for (int j = 0; j < bp.njobs; ++j) {
    const bool table = job_wants<MODE, HAS_QU, MapT>(bp.job[j]).slots > 0;
    with += table;
    if (!table) without += bp.tiles_before[j + 1] - bp.tiles_before[j];
  }
  if (with == 0 || without < (long long)kSplitWaves * sm_count())
    return launch_alike<MODE, HAS_QU, MapT, PM, LAYOUT>(bp, stream);
  static thread_local BatchParams part;
  for (const bool table : {true, false}) {
    pick_jobs<MODE, HAS_QU, MapT>(bp, table, part);
    const int rc = launch_alike<MODE, HAS_QU, MapT, PM, LAYOUT>(part, stream);
    if (rc != TODGPU_OK) return rc;
  }
  return TODGPU_OK;
}

template <int MODE, typename MapT, int PM>
int dispatch_batched_qu(BatchParams& bp, bool has_qu, bool iqu, cudaStream_t s) {
  if (has_qu && iqu) return launch_grouped<MODE, true, MapT, PM, kLayoutIQU>(bp, s);
  return has_qu ? launch_grouped<MODE, true, MapT, PM, kLayoutGeneric>(bp, s)
                : launch_grouped<MODE, false, MapT, PM, kLayoutGeneric>(bp, s);
}

template <int MODE, bool HAS_QU, typename MapT, int PM, int LAYOUT>
int launch_single(const KArgs& k, cudaStream_t stream) {
  Wants w;
  add_wants<MODE, HAS_QU, MapT>(w, k, false);
  const Shape s = choose_shape(w);
  if constexpr (may_have_table<MODE, HAS_QU>())
    if (s.tab_cap > 0) return launch_gather<MODE, true, HAS_QU, MapT, PM, LAYOUT>(k, w, s, stream);
  return launch_gather<MODE, false, HAS_QU, MapT, PM, LAYOUT>(k, w, s, stream);
}
template <int MODE, typename MapT, int PM>
int dispatch_qu(const KArgs& k, bool has_qu, cudaStream_t s) {
  if (has_qu && k.C == 3 && k.c_q == 1 && k.c_u == 2) return launch_single<MODE, true, MapT, PM, kLayoutIQU>(k, s);
  return has_qu ? launch_single<MODE, true, MapT, PM, kLayoutGeneric>(k, s)
                : launch_single<MODE, false, MapT, PM, kLayoutGeneric>(k, s);
}


// Pointing-mode switch of one map element type (instantiated by gather_map_*.cu).
template <int MODE, typename MapT>
int dispatch_single_pm(const KArgs& k, bool has_qu, int params_dtype, cudaStream_t s) {
  if (params_dtype == TODGPU_F32) return dispatch_qu<MODE, MapT, kParamsRef32>(k, has_qu, s);
  if (params_dtype == TODGPU_F64) return dispatch_qu<MODE, MapT, kParamsF64>(k, has_qu, s);
  return dispatch_qu<MODE, MapT, kAngles>(k, has_qu, s);
}

template <int MODE, typename MapT>
int dispatch_batched_pm(BatchParams& bp, bool has_qu, bool iqu, int params_dtype, cudaStream_t s) {
  if (params_dtype == TODGPU_F32) return dispatch_batched_qu<MODE, MapT, kParamsRef32>(bp, has_qu, iqu, s);
  if (params_dtype == TODGPU_F64) return dispatch_batched_qu<MODE, MapT, kParamsF64>(bp, has_qu, iqu, s);
  return dispatch_batched_qu<MODE, MapT, kAngles>(bp, has_qu, iqu, s);
}

// Entry points of the per-map-type translation units.
#define TODGPU_DECLARE_MAP_DISPATCH(NAME)                                                                   \
  int dispatch_single_##NAME(const KArgs& k, int interp, bool has_qu, int params_dtype, cudaStream_t s);   \
  int dispatch_batched_##NAME(BatchParams& bp, int interp, bool has_qu, bool iqu, int params_dtype,        \
                              cudaStream_t s);
TODGPU_DECLARE_MAP_DISPATCH(f64)
TODGPU_DECLARE_MAP_DISPATCH(f32)
TODGPU_DECLARE_MAP_DISPATCH(pf32)
TODGPU_DECLARE_MAP_DISPATCH(pbf16)
TODGPU_DECLARE_MAP_DISPATCH(pf64)
#undef TODGPU_DECLARE_MAP_DISPATCH

#define TODGPU_DEFINE_MAP_DISPATCH(NAME, MAPT)                                                             \
  int dispatch_single_##NAME(const KArgs& k, int interp, bool has_qu, int params_dtype, cudaStream_t s) {  \
    return interp == TODGPU_BILINEAR ? dispatch_single_pm<TODGPU_BILINEAR, MAPT>(k, has_qu, params_dtype, s) \
                                     : dispatch_single_pm<TODGPU_NEAREST, MAPT>(k, has_qu, params_dtype, s);  \
  }                                                                                                        \
  int dispatch_batched_##NAME(BatchParams& bp, int interp, bool has_qu, bool iqu, int params_dtype,        \
                              cudaStream_t s) {                                                            \
    return interp == TODGPU_BILINEAR                                                                       \
               ? dispatch_batched_pm<TODGPU_BILINEAR, MAPT>(bp, has_qu, iqu, params_dtype, s)              \
               : dispatch_batched_pm<TODGPU_NEAREST, MAPT>(bp, has_qu, iqu, params_dtype, s);              \
  }

}  // namespace todgpu
