// kmeans.cu -- weighted spherical k-means of beam pixels on the GPU, the
// clustering behind beam_cluster.cluster_beam_pixels (beam_cluster.py:70-188):
// k-means++ seeding and the assignment / weighted-centroid iterations.
//
// * Similarities are v . c with the products accumulated as
//   fma(v2, c2, fma(v1, c1, v0 c0)), the order a BLAS matrix product with
//   fused multiply-adds uses; argmax keeps the first maximum, like numpy.
// * The per-cluster sums (weights, weighted vectors) are taken in pixel order
//   for every cluster, as numpy's bincount does, by one warp per cluster: it
//   reads 32 pixels at a time and adds them one after another.  Small
//   problems find a cluster's pixels by reading all labels; large ones sort the
//   pixels by label first (a stable counting sort: per-chunk histograms, a
//   per-cluster scan over the chunks, a warp-sequential stable scatter).
//   Deterministic and equal to the sequential sums bit for bit.
// * k-means++ seeding draws index i with probability p_i / sum p (p_i =
//   w_i max(1 - nearest_cos_i, 0)^2) as the first i with
//   cumsum(p)_i / sum(p) > u for a uniform u supplied by the caller (so the
//   caller's random stream decides); the cumulative sums are taken per warp
//   of pixels and then across them.  Up to kSeedPixels pixels one CTA draws
//   all centroids without leaving the GPU; beyond, two launches per centroid.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>

#include "gather_impl.cuh"

namespace todgpu {
namespace km {

constexpr int kThreads = 256;
constexpr int kChunk = 2048;         // pixels per histogram/scatter chunk
constexpr int kMaxClusters = 8192;   // shared-memory counters of one chunk
constexpr int kCentTile = 2048;      // centroids staged in shared memory at a time
constexpr int kSumWarps = 4;         // clusters per CTA of the sums

__device__ __forceinline__ double dot3(const double* v, double c0, double c1, double c2) {
  return fma(v[2], c2, fma(v[1], c1, v[0] * c0));
}

// labels[i] = argmax_k v_i . c_k (first maximum), best[i] = that maximum.  G
// neighbouring lanes share a pixel, each taking a contiguous part of the
// centroids: 8 up to 16384 pixels, where one lane per pixel leaves SMs idle (200 and
// 1000 centroids, us, one lane / eight: 5414 pixels 8.3 / 5.2, 26.7 / 12.3; 12,288
// 8.3 / 6.2, 26.7 / 14.7; 30,000 8.3 / 8.3, 26.7 / 28.7; 65,536 10.3 / 14.4, 36.9 /
// 51.3).
template <int G>
__global__ void assign_kernel(const double* vec, long long S, const double* cent, int K, int* labels, double* best) {
  __shared__ double sc[kCentTile * 3];
  const long long i = (blockIdx.x * (long long)blockDim.x + threadIdx.x) / G;
  const int g = threadIdx.x % G;
  double v[3] = {0.0, 0.0, 0.0};
  if (i < S) {
    v[0] = vec[3 * i];
    v[1] = vec[3 * i + 1];
    v[2] = vec[3 * i + 2];
  }
  double bs = -INFINITY;
  int bl = 0;
  for (int k0 = 0; k0 < K; k0 += kCentTile) {
    const int nk = min(kCentTile, K - k0);
    __syncthreads();
    for (int t = threadIdx.x; t < 3 * nk; t += blockDim.x) sc[t] = cent[3LL * k0 + t];
    __syncthreads();
    const int part = (nk + G - 1) / G, k1 = min(nk, (g + 1) * part);
    double ts = -INFINITY;
    int tl = 0x7fffffff;
#pragma unroll 4
    for (int k = g * part; k < k1; ++k) {
      const double s = dot3(v, sc[3 * k], sc[3 * k + 1], sc[3 * k + 2]);
      if (s > ts) {
        ts = s;
        tl = k0 + k;
      }
    }
    // the tile's first maximum over the lanes, then over the tiles so far
#pragma unroll
    for (int o = 1; o < G; o <<= 1) {
      const double os = __shfl_xor_sync(0xffffffffu, ts, o);
      const int ol = __shfl_xor_sync(0xffffffffu, tl, o);
      if (os > ts || (os == ts && ol < tl)) {
        ts = os;
        tl = ol;
      }
    }
    if (ts > bs) {
      bs = ts;
      bl = tl;
    }
  }
  if (i < S && g == 0) {
    labels[i] = bl;
    best[i] = bs;
  }
}

// counts[c * K + k] = pixels of chunk c with label k
__global__ void chunk_hist_kernel(const int* labels, long long S, int K, int* counts) {
  __shared__ int h[kMaxClusters];
  for (int k = threadIdx.x; k < K; k += blockDim.x) h[k] = 0;
  __syncthreads();
  const long long c0 = (long long)blockIdx.x * kChunk;
  for (long long i = c0 + threadIdx.x; i < min(S, c0 + kChunk); i += blockDim.x) atomicAdd(&h[labels[i]], 1);
  __syncthreads();
  for (int k = threadIdx.x; k < K; k += blockDim.x) counts[(long long)blockIdx.x * K + k] = h[k];
}

// per cluster: base[c * K + k] = pixels of label k in chunks before c; total[k]
__global__ void chunk_scan_kernel(int* counts, int nchunks, int K, int* total) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= K) return;
  int run = 0;
  for (int c = 0; c < nchunks; ++c) {
    const int n = counts[(long long)c * K + k];
    counts[(long long)c * K + k] = run;
    run += n;
  }
  total[k] = run;
}

// offsets[k] = sum of total[0..k) (one block, K <= kMaxClusters)
__global__ void offsets_kernel(const int* total, int K, int* offsets) {
  __shared__ int part[kThreads];
  const int per = (K + blockDim.x - 1) / blockDim.x;
  const int k0 = threadIdx.x * per, k1 = min(K, k0 + per);
  int s = 0;
  for (int k = k0; k < k1; ++k) s += total[k];
  part[threadIdx.x] = s;
  __syncthreads();
  if (threadIdx.x == 0) {
    int run = 0;
    for (int t = 0; t < (int)blockDim.x; ++t) {
      const int n = part[t];
      part[t] = run;
      run += n;
    }
    offsets[K] = run;
  }
  __syncthreads();
  int run = part[threadIdx.x];
  for (int k = k0; k < k1; ++k) {
    offsets[k] = run;
    run += total[k];
  }
}

// Stable scatter of chunk c: one warp walks the chunk in index order, 32 pixels
// at a time; pixels of one label in a step take consecutive slots in lane order.
__global__ void scatter_kernel(const int* labels, long long S, int K, const int* base, const int* offsets,
                               int* order) {
  __shared__ int next[kMaxClusters];
  for (int k = threadIdx.x; k < K; k += blockDim.x) next[k] = offsets[k] + base[(long long)blockIdx.x * K + k];
  __syncthreads();
  if (threadIdx.x >= 32) return;
  const int lane = threadIdx.x;
  const long long c0 = (long long)blockIdx.x * kChunk, c1 = min(S, c0 + kChunk);
  for (long long i0 = c0; i0 < c1; i0 += 32) {
    const long long i = i0 + lane;
    const bool valid = i < c1;
    const int lab = valid ? labels[i] : -1;
    const unsigned peers = __match_any_sync(0xffffffffu, lab);
    const int rank = __popc(peers & ((1u << lane) - 1u));
    const int slot = valid ? next[lab] + rank : 0;
    __syncwarp();
    if (valid) order[slot] = (int)i;
    const int leader = __ffs(peers) - 1;
    if (valid && lane == leader) next[lab] += __popc(peers);
    __syncwarp();
  }
}

// Adds the weighted vectors of up to 32 pixels (lane l's is idx, n of them) to
// the warp's four sums -- lane c holds sum c of (w x, w y, w z, w) -- one pixel
// after another in lane order (products w * v rounded first, then added).
__device__ __forceinline__ void add_in_order(const double* vec, const double* w, long long idx, int n, int lane,
                                             double (*buf)[33], double& acc) {
  if (lane < n) {
    const double wi = w[idx];
    buf[0][lane] = wi * vec[3 * idx];
    buf[1][lane] = wi * vec[3 * idx + 1];
    buf[2][lane] = wi * vec[3 * idx + 2];
    buf[3][lane] = wi;
  }
  __syncwarp();
  if (lane < 4) {
#pragma unroll 4
    for (int q = 0; q < n; ++q) acc += buf[lane][q];
  }
  __syncwarp();
}

// sums[4 k ..] = (sum w x, sum w y, sum w z, sum w) over cluster k's pixels in
// increasing pixel order; one warp per cluster, the pixels sorted by label.  (One
// thread per cluster waited for memory at every pixel.)
__global__ void cluster_sums_kernel(const double* vec, const double* w, const int* order, const int* offsets, int K,
                                    double* sums) {
  __shared__ double buf[kSumWarps][4][33];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, k = blockIdx.x * kSumWarps + warp;
  if (k >= K) return;
  double acc = 0.0;
  const int end = offsets[k + 1];
  for (int j = offsets[k]; j < end; j += 32) {
    const int n = min(32, end - j);
    add_in_order(vec, w, lane < n ? order[j + lane] : 0, n, lane, buf[warp], acc);
  }
  if (lane < 4) sums[4 * k + lane] = acc;
}

// The same sums from the labels themselves: each cluster's warp reads all of them
// (S K / 32 reads of 128 bytes: one launch in place of five for S K up to
// kScanLimit).
constexpr long long kScanLimit = 1LL << 23;
__global__ void cluster_scan_kernel(const double* vec, const double* w, const int* labels, long long S, int K,
                                    double* sums) {
  __shared__ double buf[kSumWarps][4][33];
  __shared__ int found[kSumWarps][64];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, k = blockIdx.x * kSumWarps + warp;
  if (k >= K) return;
  double acc = 0.0;
  int n = 0;  // pixels found and not yet added
  for (long long i0 = 0; i0 < S; i0 += 128) {
    int lab[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) lab[u] = i0 + 32 * u + lane < S ? labels[i0 + 32 * u + lane] : -1;
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const unsigned hit = __ballot_sync(0xffffffffu, lab[u] == k);
      if (hit == 0) continue;
      if (lab[u] == k) found[warp][n + __popc(hit & ((1u << lane) - 1u))] = (int)(i0 + 32 * u + lane);
      n += __popc(hit);
      __syncwarp();
      if (n >= 32) {
        add_in_order(vec, w, found[warp][lane], 32, lane, buf[warp], acc);
        n -= 32;
        const int rest = found[warp][32 + lane];
        __syncwarp();
        if (lane < n) found[warp][lane] = rest;
        __syncwarp();
      }
    }
  }
  if (n > 0) add_in_order(vec, w, lane < n ? found[warp][lane] : 0, n, lane, buf[warp], acc);
  if (lane < 4) sums[4 * k + lane] = acc;
}

// First index of the minimum of best[0..S) (one block).
__global__ void argmin_kernel(const double* best, long long S, long long* out) {
  __shared__ double sv[kThreads];
  __shared__ long long si[kThreads];
  double bv = INFINITY;
  long long bi = S;
  for (long long i = threadIdx.x; i < S; i += blockDim.x) {
    const double v = best[i];
    if (v < bv) {
      bv = v;
      bi = i;
    }
  }
  sv[threadIdx.x] = bv;
  si[threadIdx.x] = bi;
  __syncthreads();
  for (int d = blockDim.x / 2; d > 0; d >>= 1) {
    if ((int)threadIdx.x < d) {
      const double v = sv[threadIdx.x + d];
      const long long j = si[threadIdx.x + d];
      if (v < sv[threadIdx.x] || (v == sv[threadIdx.x] && j < si[threadIdx.x])) {
        sv[threadIdx.x] = v;
        si[threadIdx.x] = j;
      }
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) *out = si[0] < S ? si[0] : 0;
}

// ---- k-means++ seeding ------------------------------------------------------
__device__ __forceinline__ double warp_total(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
__device__ __forceinline__ double warp_inclusive(double v, int lane) {
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const double y = __shfl_up_sync(0xffffffffu, v, o);
    if (lane >= o) v += y;
  }
  return v;
}

// Step k: nearest[i] = max(nearest[i], v_i . c_{k-1}) (k >= 1), p_i as above
// (p_i = w_i at k = 0), block sums of p.
__global__ void seed_weights_kernel(const double* vec, const double* w, long long S, double* nearest,
                                    const double* cent, int k, double* p, double* block_sums) {
  __shared__ double red[kThreads / 32];
  const long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  double pi = 0.0;
  if (i < S) {
    if (k == 0) {
      pi = w[i];
    } else {
      const double* c = cent + 3LL * (k - 1);
      const double s = dot3(vec + 3 * i, c[0], c[1], c[2]);
      double nc = (k == 1) ? s : nearest[i];
      if (k > 1 && s > nc) nc = s;
      nearest[i] = nc;
      const double d = max(1.0 - nc, 0.0);
      pi = w[i] * (d * d);
    }
    p[i] = pi;
  }
  // sum of the block's warps, in a fixed order
  const double ws = warp_total(pi);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = ws;
  __syncthreads();
  if (threadIdx.x == 0) {
    double s = 0.0;
    for (int t = 0; t < kThreads / 32; ++t) s += red[t];
    block_sums[blockIdx.x] = s;
  }
}

// First index i < n with (before + cumsum(x)_i) / total > u, by one warp, or -1;
// `before` becomes the sum before it (or of everything).
__device__ __forceinline__ long long first_above(const double* x, long long n, double total, double u, int lane,
                                                 double& before) {
  double run = before;
  for (long long i0 = 0; i0 < n; i0 += 32) {
    const double v = i0 + lane < n ? x[i0 + lane] : 0.0;
    const double incl = run + warp_inclusive(v, lane);
    const unsigned hit = __ballot_sync(0xffffffffu, i0 + lane < n && incl / total > u);
    if (hit != 0) {
      const int l = __ffs(hit) - 1;
      before = __shfl_sync(0xffffffffu, incl - v, l);
      return i0 + l;
    }
    run = __shfl_sync(0xffffffffu, incl, 31);
  }
  before = run;
  return -1;
}

// The drawn index for uniform u by one warp -- the first i with cumsum(p)_i /
// total > u, from the sums of `nb` runs of `len` pixels each.  When every p_i is
// 0 the weights w are used instead (the caller's fallback to the initial
// probabilities).
__device__ long long draw_index(const double* p, const double* sums, int nb, int len, const double* w, long long S,
                                double u, int lane) {
  double total = 0.0;
  for (int b = lane; b < nb; b += 32) total += sums[b];
  total = warp_total(total);
  double before = 0.0;
  if (!(total > 0.0)) {
    double t = 0.0;
    for (long long i = lane; i < S; i += 32) t += w[i];
    const long long i = first_above(w, S, warp_total(t), u, lane, before);
    return i < 0 ? S - 1 : i;
  }
  long long b = first_above(sums, nb, total, u, lane, before);
  if (b < 0) {  // u at or above the rounded total: the last run with weight
    int last = 0;
    for (int q = lane; q < nb; q += 32)
      if (sums[q] > 0.0) last = q;
    for (int o = 16; o > 0; o >>= 1) last = max(last, __shfl_xor_sync(0xffffffffu, last, o));
    return min(S, (long long)(last + 1) * len) - 1;
  }
  const long long i0 = b * len, n = min(S - i0, (long long)len);
  const long long i = first_above(p + i0, n, total, u, lane, before);
  return i0 + (i < 0 ? n - 1 : i);
}

// One warp: the drawn index, then c_k = v_i.
__global__ void seed_pick_kernel(const double* vec, const double* w, long long S, const double* p,
                                 const double* block_sums, int nblocks, double u, int k, double* cent,
                                 long long* chosen) {
  const int lane = threadIdx.x;
  const long long pick = draw_index(p, block_sums, nblocks, kThreads, w, S, u, lane);
  if (lane < 3) cent[3LL * k + lane] = vec[3 * pick + lane];
  if (lane == 0) chosen[k] = pick;
}

// All steps k0 .. k0 + nk of the seeding in one CTA, S <= kSeedPixels: pixel t
// + 1024 j belongs to thread t, which keeps its nearest similarity in a
// register; p and the sums of the runs of 32 pixels are in shared memory, and
// warp 0 draws.  What the two launches per centroid with a one-thread scan
// each took (5,414 pixels, 200 centroids: 5.6 ms) is now one kernel (0.9 ms with
// its host calls).
constexpr int kSeedThreads = 1024;
constexpr int kSeedPer = 12;
constexpr int kSeedPixels = kSeedThreads * kSeedPer;
constexpr int kSeedBatch = 1024;  // draws per launch (they travel in the kernel parameters)
struct SeedDraws {
  double u[kSeedBatch];
};
__global__ void __launch_bounds__(kSeedThreads) seed_all_kernel(const double* vec, const double* w, int S,
                                                                double* nearest, double* cent, long long* chosen,
                                                                int k0, int nk, const __grid_constant__ SeedDraws d) {
  extern __shared__ double s_p[];  // p of kSeedThreads * per pixels
  __shared__ double s_sums[kSeedPer * 32];
  __shared__ double s_c[3];
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
  const int per = (S + kSeedThreads - 1) / kSeedThreads;
  double near[kSeedPer];
#pragma unroll
  for (int j = 0; j < kSeedPer; ++j) {
    const int i = j * kSeedThreads + t;
    near[j] = k0 > 0 && i < S ? nearest[i] : 0.0;
  }
  if (t < 3) s_c[t] = k0 > 0 ? cent[3LL * (k0 - 1) + t] : 0.0;
  __syncthreads();
  for (int k = k0; k < k0 + nk; ++k) {
    const double c0 = s_c[0], c1 = s_c[1], c2 = s_c[2];
#pragma unroll
    for (int j = 0; j < kSeedPer; ++j) {
      if (j >= per) break;
      const int i = j * kSeedThreads + t;
      double pi = 0.0;
      if (i < S) {
        pi = w[i];
        if (k > 0) {
          const double s = dot3(vec + 3LL * i, c0, c1, c2);
          if (k == 1 || s > near[j]) near[j] = s;
          const double e = max(1.0 - near[j], 0.0);
          pi *= e * e;
        }
      }
      s_p[i] = pi;
      const double ws = warp_total(pi);
      if (lane == 0) s_sums[j * 32 + warp] = ws;
    }
    __syncthreads();
    if (warp == 0) {
      const long long pick = draw_index(s_p, s_sums, 32 * per, 32, w, S, d.u[k - k0], lane);
      if (lane < 3) cent[3LL * k + lane] = s_c[lane] = vec[3 * pick + lane];
      if (lane == 0) chosen[k] = pick;
    }
    __syncthreads();
  }
#pragma unroll
  for (int j = 0; j < kSeedPer; ++j) {
    const int i = j * kSeedThreads + t;
    if (i < S) nearest[i] = near[j];
  }
}

inline unsigned blocks_for(long long n, int t) { return (unsigned)std::max(1LL, (n + t - 1) / t); }

}  // namespace km
}  // namespace todgpu

using namespace todgpu;
using namespace todgpu::km;

namespace {

int check_sk(long long S, int K) {
  if (S < 1 || S > (1LL << 31) - 1) return fail(TODGPU_ESHAPE, "pixel count must be in [1, 2^31)");
  if (K < 1 || K > kMaxClusters) return fail(TODGPU_ESHAPE, "cluster count must be in [1, 8192]");
  return TODGPU_OK;
}

int done(const char* what) {
  const cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? TODGPU_OK : cuda_fail(e, what);
}

}  // namespace

extern "C" size_t todgpu_kmeans_workspace_bytes(int64_t S, int32_t K) {
  if (S < 1 || K < 1 || K > kMaxClusters) return 0;
  const long long nchunks = (S + kChunk - 1) / kChunk;
  const long long nblk = (S + kThreads - 1) / kThreads;
  const long long ints = nchunks * K + K + (K + 1) + S;  // base/counts, total, offsets, order
  const long long dbl = S + S + nblk;                     // nearest, p, block sums
  return (size_t)(ints * 4 + 64 + dbl * 8 + 64);
}

extern "C" int todgpu_kmeans_seed(const double* vec, const double* w, int64_t S, int32_t K, const double* uniforms,
                                  double* centroids, int64_t* chosen, void* ws, size_t ws_bytes, void* stream) {
  int rc = check_sk(S, K);
  if (rc) return rc;
  if (!vec || !w || !uniforms || !centroids || !chosen || !ws) return fail(TODGPU_EINVAL, "NULL pointer");
  if (ws_bytes < todgpu_kmeans_workspace_bytes(S, K)) return fail(TODGPU_ESHAPE, "workspace too small");
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const long long nchunks = (S + kChunk - 1) / kChunk;
  const long long nblk = (S + kThreads - 1) / kThreads;
  char* b = static_cast<char*>(ws);
  double* dws = reinterpret_cast<double*>(b + ((nchunks * K + K + (K + 1) + S) * 4 + 64) / 8 * 8);
  double* nearest = dws;
  double* p = dws + S;
  double* bsum = dws + 2 * S;
  if (S <= kSeedPixels) {
    const size_t smem = sizeof(double) * kSeedThreads * ((S + kSeedThreads - 1) / kSeedThreads);
    static SmemOptIn opt_in;
    const cudaError_t attr = opt_in(reinterpret_cast<const void*>(seed_all_kernel),
                                    [] { return (int)(sizeof(double) * kSeedPixels); });
    if (attr != cudaSuccess) return cuda_fail(attr, "kmeans seeding attributes");
    for (int k0 = 0; k0 < K; k0 += kSeedBatch) {
      SeedDraws d;
      const int nk = std::min(kSeedBatch, K - k0);
      std::copy(uniforms + k0, uniforms + k0 + nk, d.u);
      seed_all_kernel<<<1, kSeedThreads, smem, s>>>(vec, w, (int)S, nearest, centroids,
                                                    reinterpret_cast<long long*>(chosen), k0, nk, d);
    }
    return done("kmeans seeding");
  }
  for (int k = 0; k < K; ++k) {
    seed_weights_kernel<<<(unsigned)nblk, kThreads, 0, s>>>(vec, w, S, nearest, centroids, k, p, bsum);
    seed_pick_kernel<<<1, 32, 0, s>>>(vec, w, S, p, bsum, (int)nblk, uniforms[k], k, centroids,
                                      reinterpret_cast<long long*>(chosen));
  }
  return done("kmeans seeding");
}

extern "C" int todgpu_kmeans_assign(const double* vec, int64_t S, const double* centroids, int32_t K, int32_t* labels,
                                    double* best, void* stream) {
  int rc = check_sk(S, K);
  if (rc) return rc;
  if (!vec || !centroids || !labels || !best) return fail(TODGPU_EINVAL, "NULL pointer");
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  int* lab = reinterpret_cast<int*>(labels);
  if (S <= (1 << 14))
    assign_kernel<8><<<blocks_for(8 * S, kThreads), kThreads, 0, s>>>(vec, S, centroids, K, lab, best);
  else
    assign_kernel<1><<<blocks_for(S, kThreads), kThreads, 0, s>>>(vec, S, centroids, K, lab, best);
  return done("kmeans assign");
}

extern "C" int todgpu_kmeans_sums(const double* vec, const double* w, const int32_t* labels, int64_t S, int32_t K,
                                  double* sums, void* ws, size_t ws_bytes, void* stream) {
  int rc = check_sk(S, K);
  if (rc) return rc;
  if (!vec || !w || !labels || !sums || !ws) return fail(TODGPU_EINVAL, "NULL pointer");
  if (ws_bytes < todgpu_kmeans_workspace_bytes(S, K)) return fail(TODGPU_ESHAPE, "workspace too small");
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  if (S * K <= kScanLimit) {
    cluster_scan_kernel<<<blocks_for(K, kSumWarps), 32 * kSumWarps, 0, s>>>(
        vec, w, reinterpret_cast<const int*>(labels), S, K, sums);
    return done("kmeans sums");
  }
  const long long nchunks = (S + kChunk - 1) / kChunk;
  int* counts = static_cast<int*>(ws);
  int* total = counts + nchunks * K;
  int* offsets = total + K;
  int* order = offsets + (K + 1);
  const int* lab = reinterpret_cast<const int*>(labels);
  chunk_hist_kernel<<<(unsigned)nchunks, kThreads, 0, s>>>(lab, S, K, counts);
  chunk_scan_kernel<<<blocks_for(K, kThreads), kThreads, 0, s>>>(counts, (int)nchunks, K, total);
  offsets_kernel<<<1, kThreads, 0, s>>>(total, K, offsets);
  scatter_kernel<<<(unsigned)nchunks, kThreads, 0, s>>>(lab, S, K, counts, offsets, order);
  cluster_sums_kernel<<<blocks_for(K, kSumWarps), 32 * kSumWarps, 0, s>>>(vec, w, order, offsets, K, sums);
  return done("kmeans sums");
}

extern "C" int todgpu_kmeans_argmin(const double* best, int64_t S, int64_t* index, void* stream) {
  if (S < 1) return fail(TODGPU_ESHAPE, "S must be >= 1");
  if (!best || !index) return fail(TODGPU_EINVAL, "NULL pointer");
  argmin_kernel<<<1, kThreads, 0, static_cast<cudaStream_t>(stream)>>>(best, S,
                                                                        reinterpret_cast<long long*>(index));
  return done("kmeans argmin");
}
