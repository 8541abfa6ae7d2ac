// kmeans.cu -- the k-means assignment step as a consumer of the skinny SGEMM.
//
// HiperML's assignment kernel (hmlKmeansAssignCtrdSmem,
// include/hml_kmeans_kernel_template.h:19-90) gives each point the index of
// its nearest centroid: dist_k = sum_d (x_d - c_kd)^2 accumulated in FP32 in
// dimension order (nvcc contracts `dist += delta * delta` into one fused
// multiply-add per dimension), the first k with the smallest dist winning
// (strict `<` from FLT_MAX).  Points are row-major [points][dims], centroids
// row-major [clusters][dims].
//
// Here, with ||x||^2 constant per point, argmin_k dist_k = argmin_k
// (||c_k||^2 - 2 x . c_k), and the dot products of every point with every
// centroid are one skinny GEMM S = X C^T (points x clusters), in one of three
// forms:
//   * tensor-core (method 3, the default wherever its kernel can run: at most
//     256 centroids that fit in shared memory as FP16 planes): FP16X3 products
//     on tcgen05 into TMEM, the argmin read back from the accumulator by the
//     thread that owns the point;
//   * tiled (method 1, the default otherwise up to 256 dimensions): a
//     register-tiled FP32 SIMT GEMM with the argmin in its epilogue;
//   * SGEMM (method 2, wider points): the library's SGEMM in an FP32-accurate
//     configuration (BF16X6 or SIMT; never the fast BF16X3 mode), S in HBM,
//     and a pick kernel.
// The products carry rounding errors that the reference's direct sums do
// not, so the pick is made exact: with g_k = ||c_k||^2 - 2 S_k, every
// centroid whose g_k lies within a bound of the smallest (16 gamma_{dims+4}
// (||x||^2 + max_k ||c_k||^2) for the FP32 forms, 2^-19 of it more for the
// FP16X3 products: more than twice the sum of the worst-case errors of g and
// of the reference's dist) is a candidate, and the reference's choice is
// always among them.  A point with more than one candidate (or non-finite
// values) goes to a close-call list that is settled with the reference's own
// arithmetic over the candidates, the first smallest in increasing k.  So
// every point gets the reference kernel's index, exact ties included.
#include <cuda_fp16.h>

#include <algorithm>
#include <cfloat>
#include <cstring>
#include <type_traits>

#include "hml_device.cuh"
#include "hml_internal.h"
#include "hml_lines.h"
#include "hml_select.h"
#include "hml_tune.h"
#include "hml_tcgen05.cuh"
#include "simt_tile.cuh"

namespace hml {
namespace {

constexpr int kNormWarps = 8;
// Widest points the automatic choice gives the tiled form (method 1); wider
// ones go through the SGEMM (method 2).
constexpr int kKmeansTiledMaxDims = 256;

// ||c_k||^2 for every centroid, one warp per centroid (FP32; used only to
// screen candidates).  It also empties the close-call list of the call.
__global__ void centroid_norms_kernel(const float *cent, int k, int d, float *cnorm,
                                      unsigned *ccount) {
  const int lane = threadIdx.x & 31;
  if (blockIdx.x == 0 && threadIdx.x == 0) *ccount = 0u;
  for (int c = blockIdx.x * kNormWarps + (threadIdx.x >> 5); c < k; c += gridDim.x * kNormWarps) {
    const float *row = cent + static_cast<int64_t>(c) * d;
    float s = 0.0f;
    for (int j = lane; j < d; j += 32) s = fmaf(row[j], row[j], s);
    cnorm[c] = warp_sum(s);
  }
}

// The reference's distance of point x to centroid c (the fused form nvcc
// gives `dist += delta * delta`).
__device__ __forceinline__ float ref_dist(const float *x, const float *c, int d) {
  float dist = 0.0f;
  for (int j = 0; j < d; ++j) {
    const float delta = __fsub_rn(x[j], c[j]);
    dist = __fmaf_rn(delta, delta, dist);
  }
  return dist;
}

// The reference's pick for point x among the candidates -- the centroids
// whose g_k, recomputed, is at most lim -- by one warp (every lane calls
// this with the same arguments).  For 16 centroids at a time, in increasing
// k, the lanes form x . c_k together (lane r takes dimensions r, r + 32,
// ...: coalesced loads of the rows; the partial sums added by xor shuffles,
// so every lane holds the same dot product: any FP32 evaluation of g stays
// within the bound the screen allowed for); for a candidate every lane forms
// the reference's own distance (sequential, subtract then FMA) and keeps the
// first smallest below FLT_MAX (strict <), which is the reference's pick.
// 0 when no candidate's distance is below FLT_MAX (the reference leaves that
// case unset).  A limit that is not finite (norms or products beyond FP32,
// where g says nothing) makes every centroid a candidate.
__device__ __noinline__ uint32_t exact_pick(const float *x, int d, const float *cent, int k,
                                            const float *cnorm, float lim) {
  constexpr int U = 16;  // centroids in flight: their loads and shuffle trees interleave
  const int lane = threadIdx.x & 31;
  float bd = FLT_MAX;
  uint32_t bk = 0;
  for (int c0 = 0; c0 < k; c0 += U) {
    float part[U], cnv[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      part[u] = 0.0f;
      cnv[u] = c0 + u < k ? cnorm[c0 + u] : 0.0f;  // loaded ahead of the tests below
    }
    for (int j = lane; j < d; j += 32) {
      const float xj = x[j];
#pragma unroll
      for (int u = 0; u < U; ++u)
        if (c0 + u < k) part[u] = fmaf(xj, cent[static_cast<int64_t>(c0 + u) * d + j], part[u]);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
#pragma unroll
      for (int u = 0; u < U; ++u) part[u] += __shfl_xor_sync(0xffffffffu, part[u], o);
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int c = c0 + u;
      if (c >= k || !(fmaf(-2.0f, part[u], cnv[u]) <= lim || !(lim < INFINITY))) continue;
      const float dist = ref_dist(x, cent + static_cast<int64_t>(c) * d, d);
      if (dist < bd) {
        bd = dist;
        bk = static_cast<uint32_t>(c);
      }
    }
  }
  return bk;
}

// Close calls (a second smallest g within the bound of the smallest, or
// non-finite values) are not settled where they are found: the screening
// kernels append (point, bound) to a list, every lane of a warp calling this
// together (one atomic per warp), and kmeans_settle_kernel settles the list
// afterwards, a warp per point -- so a rare long settling never holds up the
// screening of the other points.
__device__ __forceinline__ void push_close(unsigned *ccount, uint2 *citems, int64_t p, float lim,
                                           bool close) {
  const unsigned m = __ballot_sync(0xffffffffu, close);
  if (!m) return;
  const int lane = threadIdx.x & 31, leader = __ffs(m) - 1;
  unsigned base = 0;
  if (lane == leader) base = atomicAdd(ccount, static_cast<unsigned>(__popc(m)));
  base = __shfl_sync(0xffffffffu, base, leader);
  if (close)
    citems[base + __popc(m & ((1u << lane) - 1u))] =
        make_uint2(static_cast<uint32_t>(p), __float_as_uint(lim));
}

// The same pick with the centroids staged in shared memory (rows padded to
// cs = d + 1 floats, so that lane r reading element j of centroid r + 32 i
// hits bank (r + j) % 32: no conflicts), their norms beside them and the
// point's row in `xs`: lane r takes whole centroids r, r + 32, ... (its dot
// products in dimension order, any FP32 order being within the bound), forms
// the reference's distance of its candidates and keeps the first smallest
// below FLT_MAX; the warp then keeps the smallest distance, the lowest index
// among equal ones -- the first minimum in k order, the reference's pick.
// xs lies on a 16-byte boundary: the warp reads it four elements a load.  The
// loads bound the settling: 1M x 32 points, k = 64, all of them close calls
// 1363 us, 1558 one element a load.  Points below 16 dimensions keep that, as the
// loop over the rest (1M x 7, k = 64 1179 us, 1237 so).
__device__ __forceinline__ uint32_t exact_pick_smem(const float *xs, int d, const float *cs,
                                                    int k, const float *cn, float lim) {
  const int lane = threadIdx.x & 31, st = d + 1, dv = d >= 16 ? d : 0;
  float bd = FLT_MAX;
  int bk = -1;
  for (int c = lane; c < k; c += 32) {
    const float *cp = cs + c * st;
    if (lim < INFINITY) {
      float dot = 0.0f;
      int j = 0;
      for (; j + 4 <= dv; j += 4) {
        const float4 v = *reinterpret_cast<const float4 *>(xs + j);
        dot = fmaf(v.x, cp[j], dot);
        dot = fmaf(v.y, cp[j + 1], dot);
        dot = fmaf(v.z, cp[j + 2], dot);
        dot = fmaf(v.w, cp[j + 3], dot);
      }
      for (; j < d; ++j) dot = fmaf(xs[j], cp[j], dot);
      if (!(fmaf(-2.0f, dot, cn[c]) <= lim)) continue;
    }  // else: every centroid is a candidate (see exact_pick)
    float dist = 0.0f;  // ref_dist
    auto add = [&](float x, float y) {
      const float delta = __fsub_rn(x, y);
      dist = __fmaf_rn(delta, delta, dist);
    };
    int j = 0;
    for (; j + 4 <= dv; j += 4) {
      const float4 v = *reinterpret_cast<const float4 *>(xs + j);
      add(v.x, cp[j]);
      add(v.y, cp[j + 1]);
      add(v.z, cp[j + 2]);
      add(v.w, cp[j + 3]);
    }
    for (; j < d; ++j) add(xs[j], cp[j]);
    if (dist < bd) {
      bd = dist;
      bk = c;
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const float od = __shfl_xor_sync(0xffffffffu, bd, o);
    const int ok = __shfl_xor_sync(0xffffffffu, bk, o);
    if (ok >= 0 && (bk < 0 || od < bd || (od == bd && ok < bk))) {
      bd = od;
      bk = ok;
    }
  }
  return bk < 0 ? 0u : static_cast<uint32_t>(bk);
}

// Shared-memory floats the settle kernel stages (0: the centroids do not fit
// in 96 KB and are read from global memory): centroids with rows of d + 1,
// their norms, one point row per warp (8 warps), each on a 16-byte boundary.
__host__ __device__ constexpr int64_t up4(int64_t n) { return (n + 3) / 4 * 4; }
__host__ __device__ constexpr int64_t settle_smem_floats(int k, int d) {
  return up4(static_cast<int64_t>(k) * (d + 1) + k) + 8 * up4(d);
}
constexpr int64_t kSettleSmemFloats = 96 * 1024 / 4 + 27;  // (27: all that the rounding adds)

__global__ void __launch_bounds__(256) kmeans_settle_kernel(
    const float *points, int d, const float *cent, int k, const float *cnorm,
    const unsigned *ccount, const uint2 *citems, uint32_t *out, unsigned *exact, int staged) {
  extern __shared__ __align__(16) float s_set[];
  const unsigned n = *ccount;
  if (exact && n && blockIdx.x == 0 && threadIdx.x == 0) atomicAdd(exact, n);
  const unsigned wpb = blockDim.x >> 5, warps = gridDim.x * wpb;
  if (blockIdx.x * wpb >= n) return;  // no entry for this block's warps
  const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
  float *cs = s_set, *cn = s_set + static_cast<int64_t>(k) * (d + 1);
  float *xs = s_set + up4(static_cast<int64_t>(k) * (d + 1) + k) + wib * up4(d);
  if (staged) {
    for (int e = threadIdx.x; e < k * d; e += blockDim.x) {
      const int c = e / d, j = e - c * d;
      cs[c * (d + 1) + j] = cent[e];
    }
    for (int c = threadIdx.x; c < k; c += blockDim.x) cn[c] = cnorm[c];
    __syncthreads();
  }
  for (unsigned w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; w < n; w += warps) {
    const uint2 it = citems[w];
    const float *x = points + static_cast<int64_t>(it.x) * d;
    uint32_t pick;
    if (staged) {
      for (int j = lane; j < d; j += 32) xs[j] = x[j];
      __syncwarp();
      pick = exact_pick_smem(xs, d, cs, k, cn, __uint_as_float(it.y));
      __syncwarp();  // xs is rewritten for the warp's next entry
    } else {
      pick = exact_pick(x, d, cent, k, cnorm, __uint_as_float(it.y));
    }
    if (lane == 0) out[it.x] = pick;
  }
}

// One thread per point: g_k = ||c_k||^2 - 2 S(p, k) (S column-major, ld lds),
// the candidates within `margin` of the smallest; a point with more than
// one goes to the close-call list.
__global__ void kmeans_pick_kernel(const float *points, int64_t np, int d, int k, const float *S,
                                   int64_t lds, const float *cnorm, uint32_t *out,
                                   unsigned *ccount, uint2 *citems) {
  extern __shared__ float s_cnorm[];  // [k], then the block's max
  float cmax = 0.0f;
  for (int c = threadIdx.x; c < k; c += blockDim.x) {
    const float v = cnorm[c];
    s_cnorm[c] = v;
    cmax = fmaxf(cmax, v);
  }
  cmax = fmaxf(cmax, __shfl_xor_sync(0xffffffffu, cmax, 16));
  cmax = fmaxf(cmax, __shfl_xor_sync(0xffffffffu, cmax, 8));
  cmax = fmaxf(cmax, __shfl_xor_sync(0xffffffffu, cmax, 4));
  cmax = fmaxf(cmax, __shfl_xor_sync(0xffffffffu, cmax, 2));
  cmax = fmaxf(cmax, __shfl_xor_sync(0xffffffffu, cmax, 1));
  __shared__ float s_wmax[32];
  if ((threadIdx.x & 31) == 0) s_wmax[threadIdx.x >> 5] = cmax;
  __syncthreads();
  cmax = 0.0f;
  for (int w = 0; w < static_cast<int>(blockDim.x >> 5); ++w) cmax = fmaxf(cmax, s_wmax[w]);
  // 16 gamma_{d+4}, rounded up (gamma_n = n u / (1 - n u), u = 2^-24)
  const double nu = (d + 4) * 0x1p-24;
  const float bound = static_cast<float>(16.0 * nu / (1.0 - nu) * 1.001);
  const int lane = threadIdx.x & 31;
  // the warp walks 32 consecutive points at a time (every lane takes every
  // step, so the warp can list its close calls together)
  const int64_t wstride = static_cast<int64_t>(gridDim.x) * blockDim.x;
  for (int64_t p0 = blockIdx.x * static_cast<int64_t>(blockDim.x) + (threadIdx.x & ~31); p0 < np;
       p0 += wstride) {
    const int64_t p = p0 + lane;
    const bool live = p < np;
    float lim = 0.0f;
    bool close = false;
    if (live) {
      const float *x = points + p * d;
      float xn = 0.0f;
      for (int j = 0; j < d; ++j) xn = fmaf(x[j], x[j], xn);
      const float *sp = S + p;
      float gmin = INFINITY;
      int kmin = 0;
      for (int c = 0; c < k; ++c) {
        const float g = fmaf(-2.0f, sp[c * lds], s_cnorm[c]);
        if (g < gmin) {
          gmin = g;
          kmin = c;
        }
      }
      lim = gmin + bound * (xn + cmax) + 1e-37f;
      int cand = 0;
      for (int c = 0; c < k; ++c) cand += fmaf(-2.0f, sp[c * lds], s_cnorm[c]) <= lim;
      close = cand != 1 || !(lim < INFINITY);
      if (!close) out[p] = static_cast<uint32_t>(kmin);
    }
    push_close(ccount, citems, p, lim, close);
  }
}

// The tiled form: the dot products of 128 points with 64 centroids at a
// time as a register-tiled FP32 SIMT GEMM with the argmin in its epilogue.
// A block of 256 threads takes 128 points; thread (tx, ty) of the 16 x 16
// grid owns points ty*4 .. ty*4+3 and 64+ty*4 .. 64+ty*4+3 and centroids
// tx*4 .. tx*4+3 of each 64-centroid pass.  Points and centroids are staged
// dimension-major in shared memory, 32 dimensions at a time (read from HBM
// with whole-row, coalesced loads), so each dimension step is three 16-byte
// shared-memory loads feeding 32 fused multiply-adds.  After a pass, g_k =
// ||c_k||^2 - 2 x.c_k updates the thread's smallest g, its index and the
// second smallest for each of its 8 points, in increasing k; at the end the
// 16 threads that share a point merge theirs (the smaller g, the lower index
// on equal g) with shuffles.  A point whose second smallest lies within the
// bound of the smallest goes to the close-call list.  The products never
// leave the SM.
constexpr int kTP = 128;         // points per block
constexpr int kTC = 64;          // centroids per pass
constexpr int kTD = 32;          // dimensions per shared-memory stage
constexpr int kTThreads = 256;
constexpr int kXS = kTP + 4;     // row stride of the staged points (a 16-byte multiple)
constexpr int kCS = kTC + 4;     // row stride of the staged centroids

// Smallest g, its centroid and the second smallest g seen (values of g that
// compare false, i.e. NaN, are never taken).
struct Best {
  float g1;
  int k1;
  float g2;
};

__device__ __forceinline__ void best_add(Best &b, float g, int k) {
  if (g < b.g1) {
    b.g2 = b.g1;
    b.g1 = g;
    b.k1 = k;
  } else if (g < b.g2) {
    b.g2 = g;
  }
}

// Union of two disjoint centroid sets' states: (g1, k1) ordered by g, then
// k, so the merge is commutative and associative and keeps the first index.
__device__ __forceinline__ Best best_merge(const Best &a, const Best &b) {
  if (b.g1 < a.g1 || (b.g1 == a.g1 && b.k1 < a.k1)) return {b.g1, b.k1, fminf(b.g2, a.g1)};
  return {a.g1, a.k1, fminf(a.g2, b.g1)};
}

__device__ __forceinline__ Best shfl_best(unsigned mask, const Best &b, int o) {
  return {__shfl_xor_sync(mask, b.g1, o), __shfl_xor_sync(mask, b.k1, o),
          __shfl_xor_sync(mask, b.g2, o)};
}

// End of a tile for the 16 lanes of a point group (one half-warp, lane tx):
// their states for the group's 8 points (thread-local point i = tile row
// ty*4+i for i < 4, 64+ty*4+i-4 otherwise) are merged by a reduce-scatter --
// at offsets 8, 4 and 2 a lane keeps half of the points it carries, merged
// with its partner's half, and at offset 1 the pair merges its one point --
// so lanes tx and tx^1 end with point 4*bit3 + 2*bit2 + bit1 of tx merged
// over all 16.  The even lane writes a settled point or lists a close call
// (all 32 lanes of the warp call this together).
__device__ __forceinline__ void settle_group(Best (&best)[8], int64_t p0, int nb, int ty, int tx,
                                             const float *s_xn, float cmax, float bound,
                                             uint32_t *out, unsigned *ccount, uint2 *citems) {
  const unsigned hmask = 0xFFFFu << (threadIdx.x & 16);
  Best b4[4];
  {
    const bool up = tx & 8;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const Best keep = up ? best[4 + i] : best[i];
      const Best send = up ? best[i] : best[4 + i];
      b4[i] = best_merge(keep, shfl_best(hmask, send, 8));
    }
  }
  Best b2[2];
  {
    const bool up = tx & 4;
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const Best keep = up ? b4[2 + i] : b4[i];
      const Best send = up ? b4[i] : b4[2 + i];
      b2[i] = best_merge(keep, shfl_best(hmask, send, 4));
    }
  }
  Best b;
  {
    const bool up = tx & 2;
    const Best keep = up ? b2[1] : b2[0];
    const Best send = up ? b2[0] : b2[1];
    b = best_merge(keep, shfl_best(hmask, send, 2));
  }
  b = best_merge(b, shfl_best(hmask, b, 1));
  const int i = ((tx >> 3) & 1) * 4 + ((tx >> 2) & 1) * 2 + ((tx >> 1) & 1);
  const int pt = i < 4 ? ty * 4 + i : 64 + ty * 4 + (i - 4);
  const bool mine = (tx & 1) == 0 && pt < nb;
  float lim = 0.0f;
  bool close = false;
  if (mine) {
    lim = b.g1 + bound * (s_xn[pt] + cmax) + 1e-37f;
    close = !(b.g2 > lim);
    if (!close) out[p0 + pt] = static_cast<uint32_t>(b.k1);
  }
  push_close(ccount, citems, p0 + pt, lim, close);
}

__global__ void __launch_bounds__(kTThreads, 2) kmeans_tile_kernel(
    const float *__restrict__ points, int np, int d, const float *__restrict__ cent, int k,
    const float *__restrict__ cnorm, uint32_t *__restrict__ out, unsigned *ccount,
    uint2 *citems) {
  __shared__ __align__(16) float xs[kTD][kXS];
  __shared__ __align__(16) float cs[kTD][kCS];
  __shared__ float s_cn[kTC];
  __shared__ float s_xn[kTP];
  __shared__ float s_wmax[kTThreads / 32];
  const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
  const int64_t p0 = static_cast<int64_t>(blockIdx.x) * kTP;
  const int nb = static_cast<int>(min(static_cast<int64_t>(kTP), np - p0));

  // max_k ||c_k||^2 (for the bound)
  float cmax = 0.0f;
  for (int c = tid; c < k; c += kTThreads) cmax = fmaxf(cmax, cnorm[c]);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) cmax = fmaxf(cmax, __shfl_xor_sync(0xffffffffu, cmax, o));
  if ((tid & 31) == 0) s_wmax[tid >> 5] = cmax;

  Best best[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) best[i] = {INFINITY, 0, INFINITY};
  float xn = 0.0f;  // thread t < 128: ||x||^2 of point t, from the staged values
  const int dchunks = (d + kTD - 1) / kTD;
  const bool x_once = dchunks <= 1;

  // stage dimensions [d0, d0 + kTD) of the block's points, zero padded
  auto stage_points = [&](int d0, bool norms) {
    const int dn = min(kTD, d - d0);
    for (int e = tid; e < kTP * kTD; e += kTThreads) {
      const int pt = e / kTD, j = e % kTD;
      xs[j][pt] = (pt < nb && j < dn) ? points[(p0 + pt) * d + d0 + j] : 0.0f;
    }
    __syncthreads();
    if (norms && tid < kTP)
      for (int j = 0; j < dn; ++j) xn = fmaf(xs[j][tid], xs[j][tid], xn);
  };
  if (x_once && d > 0) stage_points(0, true);

  for (int c0 = 0; c0 < k; c0 += kTC) {
    __syncthreads();  // the previous pass is done with s_cn and the stages
    // ||c||^2 of the pass's centroids; NaN past the last (never taken)
    if (tid < kTC) s_cn[tid] = c0 + tid < k ? cnorm[c0 + tid] : __int_as_float(0x7fc00000);
    float acc[8][4];
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
      for (int q = 0; q < 4; ++q) acc[i][q] = 0.0f;
    for (int dc = 0; dc < dchunks; ++dc) {
      const int d0 = dc * kTD, dn = min(kTD, d - d0);
      if (dc > 0) __syncthreads();  // the previous stage's readers are done
      if (!x_once) stage_points(d0, c0 == 0);
      for (int e = tid; e < kTC * kTD; e += kTThreads) {
        const int c = e / kTD, j = e % kTD;
        cs[j][c] = (c0 + c < k && j < dn) ? cent[static_cast<int64_t>(c0 + c) * d + d0 + j] : 0.0f;
      }
      __syncthreads();
      const int jn = (dn + 3) & ~3;  // zero padded up to a multiple of 4
      for (int j0 = 0; j0 < jn; j0 += 4) {
#pragma unroll
        for (int jj = 0; jj < 4; ++jj) {
          const int j = j0 + jj;
          const float4 xa = *reinterpret_cast<const float4 *>(&xs[j][ty * 4]);
          const float4 xb = *reinterpret_cast<const float4 *>(&xs[j][64 + ty * 4]);
          const float4 cv = *reinterpret_cast<const float4 *>(&cs[j][tx * 4]);
          const float xv[8] = {xa.x, xa.y, xa.z, xa.w, xb.x, xb.y, xb.z, xb.w};
          const float cw[4] = {cv.x, cv.y, cv.z, cv.w};
#pragma unroll
          for (int i = 0; i < 8; ++i)
#pragma unroll
            for (int q = 0; q < 4; ++q) acc[i][q] = fmaf(xv[i], cw[q], acc[i][q]);
        }
      }
    }
    if (dchunks == 0) __syncthreads();  // s_cn, written above, had no barrier after it
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int c = tx * 4 + q;
      const float cn = s_cn[c];
#pragma unroll
      for (int i = 0; i < 8; ++i) best_add(best[i], fmaf(-2.0f, acc[i][q], cn), c0 + c);
    }
  }
  if (tid < kTP) s_xn[tid] = xn;
  __syncthreads();
  cmax = 0.0f;
#pragma unroll
  for (int w = 0; w < kTThreads / 32; ++w) cmax = fmaxf(cmax, s_wmax[w]);
  const double nu = (d + 4) * 0x1p-24;
  const float bound = static_cast<float>(16.0 * nu / (1.0 - nu) * 1.001);

  settle_group(best, p0, nb, ty, tx, s_xn, cmax, bound, out, ccount, citems);
}

// The resident form of the tiled kernel, for centroids that fit in shared
// memory (k and dims padded to kp = 64-multiple and dp = 4-multiple, dp <= 64
// and kp * dp <= kResidentFloats, so two blocks fit on an SM): each block
// stages the transposed centroids and their norms once and then walks
// 128-point tiles (a persistent grid), the next tile's rows copied by
// cp.async into the other of two row-major buffers while the current tile
// is computed, so the loads' latency hides behind the arithmetic.  A
// thread's 8 points are read as 16-byte row pieces (4 dimensions each), the
// centroids as 16-byte pieces of a dimension row; the products, the running
// argmin, the merge and the close-call list are the tiled kernel's.
constexpr int kResidentFloats = 8192;

__global__ void __launch_bounds__(kTThreads, 2) kmeans_resident_kernel(
    const float *__restrict__ points, int np, int d, int dp, bool vec,
    const float *__restrict__ cent, int k, int kp, const float *__restrict__ cnorm,
    uint32_t *__restrict__ out, unsigned *ccount, uint2 *citems) {
  extern __shared__ __align__(16) float sm[];
  const int cst = kp + 4;                   // row stride of the transposed centroids
  float *ct = sm;                           // [dp][cst]
  float *cn = ct + dp * cst;                // [kp]
  float *xr = cn + kp;                      // [2][kTP][dp]
  float *s_xn = xr + 2 * kTP * dp;          // [kTP]
  __shared__ float s_wmax[kTThreads / 32];
  const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
  const int64_t tiles = (static_cast<int64_t>(np) + kTP - 1) / kTP;

  // the next tile's rows into buffer `buf` (zero past d and past np when
  // copied element-wise)
  auto issue = [&](int64_t t, int buf) {
    const int64_t p0 = t * kTP;
    const int nbt = static_cast<int>(min(static_cast<int64_t>(kTP), np - p0));
    float *dst = xr + buf * kTP * dp;
    if (vec) {
      const int q = dp / 4;
      for (int e = tid; e < nbt * q; e += kTThreads) {
        const int pt = e / q, c4 = e - pt * q;
        cp_async16(smem_u32(dst + pt * dp + c4 * 4), points + (p0 + pt) * d + c4 * 4, 16);
      }
    } else {
      for (int e = tid; e < kTP * dp; e += kTThreads) {
        const int pt = e / dp, j = e - pt * dp;
        const bool v = pt < nbt && j < d;
        cp_async4(smem_u32(dst + e), v ? points + (p0 + pt) * d + j : points, v);
      }
    }
    cp_async_commit();
  };
  int64_t t = blockIdx.x;
  if (t < tiles) issue(t, 0);

  // centroids (transposed, zero padded) and norms (NaN past k: never taken)
  for (int e = tid; e < dp * kp; e += kTThreads) {
    const int j = e / kp, c = e - j * kp;
    ct[j * cst + c] = (c < k && j < d) ? cent[static_cast<int64_t>(c) * d + j] : 0.0f;
  }
  float cmax = 0.0f;
  for (int c = tid; c < kp; c += kTThreads) {
    const float v = c < k ? cnorm[c] : __int_as_float(0x7fc00000);
    cn[c] = v;
    if (c < k) cmax = fmaxf(cmax, v);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) cmax = fmaxf(cmax, __shfl_xor_sync(0xffffffffu, cmax, o));
  if ((tid & 31) == 0) s_wmax[tid >> 5] = cmax;
  __syncthreads();
  cmax = 0.0f;
#pragma unroll
  for (int w = 0; w < kTThreads / 32; ++w) cmax = fmaxf(cmax, s_wmax[w]);
  const double nu = (d + 4) * 0x1p-24;
  const float bound = static_cast<float>(16.0 * nu / (1.0 - nu) * 1.001);

  for (int buf = 0; t < tiles; t += gridDim.x, buf ^= 1) {
    const int64_t tn = t + gridDim.x;
    if (tn < tiles) {
      issue(tn, buf ^ 1);
      asm volatile("cp.async.wait_group 1;" ::: "memory");
    } else {
      asm volatile("cp.async.wait_group 0;" ::: "memory");
    }
    __syncthreads();  // this tile's rows are in place
    const float *x = xr + buf * kTP * dp;
    const int64_t p0 = t * kTP;
    const int nb = static_cast<int>(min(static_cast<int64_t>(kTP), np - p0));
    if (tid < kTP) {
      // ||x||^2 for the bound (the row's 16-byte pieces in a rotated order,
      // so that the lanes of a warp read different banks)
      const int q = dp / 4;
      float xn = 0.0f;
      for (int i = 0; i < q; ++i) {
        const float4 v = lds128(x + tid * dp + ((i + tid) % q) * 4);
        xn = fmaf(v.x, v.x, xn);
        xn = fmaf(v.y, v.y, xn);
        xn = fmaf(v.z, v.z, xn);
        xn = fmaf(v.w, v.w, xn);
      }
      s_xn[tid] = xn;
    }
    Best best[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) best[i] = {INFINITY, 0, INFINITY};
    const float *xa = x + (ty * 4) * dp, *xb = x + (64 + ty * 4) * dp;
    for (int c0 = 0; c0 < kp; c0 += kTC) {
      float acc[8][4];
#pragma unroll
      for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int q = 0; q < 4; ++q) acc[i][q] = 0.0f;
      const float *cc = ct + c0 + tx * 4;
      for (int j0 = 0; j0 < dp; j0 += 4) {
        float4 xv[8];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          xv[i] = lds128(xa + i * dp + j0);
          xv[4 + i] = lds128(xb + i * dp + j0);
        }
#pragma unroll
        for (int jj = 0; jj < 4; ++jj) {
          const float4 cv = lds128(cc + (j0 + jj) * cst);
          const float cw[4] = {cv.x, cv.y, cv.z, cv.w};
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            const float xi = jj == 0 ? xv[i].x : jj == 1 ? xv[i].y : jj == 2 ? xv[i].z : xv[i].w;
#pragma unroll
            for (int q = 0; q < 4; ++q) acc[i][q] = fmaf(xi, cw[q], acc[i][q]);
          }
        }
      }
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const int c = tx * 4 + q;
        const float cnv = cn[c0 + c];
#pragma unroll
        for (int i = 0; i < 8; ++i) best_add(best[i], fmaf(-2.0f, acc[i][q], cnv), c0 + c);
      }
    }
    __syncthreads();  // s_xn is complete
    settle_group(best, p0, nb, ty, tx, s_xn, cmax, bound, out, ccount, citems);
    __syncthreads();  // the buffer and s_xn are free for the tile after next
  }
}

// ------------------------------------------------ the tensor-core form
// (method 3, and the automatic choice wherever the centroids fit in shared
// memory)  One persistent CTA per SM screens 128-point tiles on tcgen05 and
// settles its own close calls; nothing runs before or after it.
//
// Products.  Points and centroids are scaled by one power of two s (exact)
// that brings the largest coordinate of the centroids into [2^5, 2^6); then
// x = x0 + x1 and -2c = c0 + c1 in FP16, 22 significant bits, and
// -2 x.c ~ x0.c0 + x0.c1 + x1.c0 accumulated in FP32 in TMEM.  This only
// screens.  The split leaves out at most 3.02 2^-22 |x_j 2 c_j| and, where a
// half is subnormal, 1.01 2^-25 (|x_j| + |2 c_j|) of a product; with
// max ||c|| >= 2^5 and dims <= 2048 that is at most 3.42 2^-22 (||x||^2 +
// max ||c||^2) of a g_k, and a point is settled from the screen only when its
// second smallest g lies further from the smallest than twice that and the
// FP32 margin together, (2^-19 + 16 gamma_{dims+4}) (||x||^2 + max ||c||^2).
// Every other point gets the reference's own FP32 arithmetic, and so does one
// with ||x|| s >= 2^15.5, whose halves could overflow.
// (BF16 halves need no scale and 16 packed instructions less a block, but a
// margin of 2^-15: points far from the origin became close calls, 200k x 30,
// k = 200 at an offset of 100 spreads 671 us.)
//
// Roles of a CTA (W = 4 or 2 groups, each with 512 / W TMEM columns: an
// accumulator of NC columns, then S stages of 32 columns of A):
//   * controller warp g (one lane): streams group g's tiles, 32 dimensions a
//     block, into the group's ring of shared-memory slots by TMA (rows that
//     are not 16-byte aligned through four maps, one per row index modulo 4,
//     with boxes 4 floats wider, as the SGEMM's unaligned form does), and
//     issues the group's tcgen05.mma (A in TMEM, the centroid planes resident
//     in shared memory, N = NC).  A block's slot is refilled when its stage
//     is written, so the ring needs no barrier of its own for that.
//   * the 4 warps of group g take the CTA's tiles g, g + W, ...  Thread m owns
//     point m, which is a TMEM lane: it splits the point's row block by block
//     into TMEM (tcgen05.st), then -- while the tensor core works on the
//     tile -- the first blocks of its next tile, then reads the accumulator
//     row and takes the argmin.
// With more than 64 centroids (NC columns a pass, P passes) the tile's stages
// stay in TMEM for all passes.
//
// The argmin over a row costs 3 issue slots a centroid (it was 7, and the
// limit): g in packed FP32x2 adds, the smallest by 3-input minima (half an
// instruction a value), then the sign bits of g - lim shifted into a mask, in
// which the first smallest is alone unless the point is a close call.
// Measured on B200 (whole calls): 1M x 32, k = 64 43 us (65 us with TF32X3
// products, the per-value argmin and separate prep and settle kernels; 21 us
// of HBM time), k = 256 106 us (162); 1M x 128, k = 64 87 us (709 us on the
// tiled form; 84 us of HBM time), 1M x 256, k = 64 163 us (1560; 167); 1M x
// 11, k = 192 94 us (300).  Wide points are bound by HBM, narrow ones by the
// groups' own instructions and the latencies between them.
constexpr int kTcMaxK = 256;                     // centroids (padded to 16)
constexpr int kTcMaxPlanes = 128 * 1024;         // bytes of the centroids' planes
constexpr int kTcStageCols = 32;                 // TMEM columns of a 32-dimension block
__host__ __device__ constexpr int km_slot_bytes(bool au) {
  return au ? 4 * 36 * 32 * 4 : kTP * 32 * 4;  // 18 KB or 16 KB: a block of a tile
}

template <bool AU>
struct KmMaps {
  CUtensorMap m[AU ? 4 : 1];  // unaligned rows: class r = rows r, r + 4, ...
};

struct KmTcArgs {
  const float *points, *cent;
  int np, d, k;
  int nb;       // 32-dimension blocks
  int kp;       // centroids padded to passes x nc
  int passes, stages, sa;
  int e[4];     // floats before the data in class r's boxes
  uint32_t *out;
  uint2 *citems;  // [grid][list]: the CTA's close calls
  int list;       // points a CTA can have
  unsigned *exact;
  int *err;
};

__host__ __device__ constexpr int km_tc_threads(int w) { return (4 + 4 * w) * 32; }

__device__ __forceinline__ uint32_t km_f16x2(float lo, float hi) {
  uint32_t r;
  asm("cvt.rn.f16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(hi), "f"(lo));
  return r;
}

// The values a packed FP16 pair holds.
__device__ __forceinline__ float2 km_f16_pair(uint32_t w) {
  return __half22float2(*reinterpret_cast<const __half2 *>(&w));
}

// x less the pair's values.
__device__ __forceinline__ float2 km_residual(uint32_t w, float2 x) {
  float2 r;
  asm("{\n\t.reg .b16 h0, h1, m;\n\t"
      "mov.b32 {h0, h1}, %2;\n\t"
      "mov.b16 m, 0xBC00;\n\t"
      "fma.rn.f32.f16 %0, h0, m, %3;\n\t"
      "fma.rn.f32.f16 %1, h1, m, %4;\n\t}"
      : "=f"(r.x), "=f"(r.y)
      : "r"(w), "f"(x.x), "f"(x.y));
  return r;
}

// The power of two that brings magnitudes up to `top` (not NaN) below 2^6: at
// most 2^105, so that 1 / s is normal (g of centroids that small all lie within
// the margin's 1e-37), and 1 when there is nothing to scale.
__device__ __forceinline__ float km_scale(float top) {
  const int e = __float_as_int(top) >> 23;  // biased
  if (top == 0.0f || e == 255) return 1.0f;
  return __int_as_float(min(259 - e, 232) << 23);  // 2^(5 - (e - 127))
}

__device__ __forceinline__ float min3(float a, float b, float c) {
  float r;
  asm("min.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
  return r;
}

// g of 16 consecutive centroids: accumulator columns plus ||c||^2 (at the
// shared address cn).
__device__ __forceinline__ void km_g16(const uint32_t (&r)[16], uint32_t cn, float2 *g) {
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float4 c = lds128(cn + 16 * i);
    g[2 * i] = __fadd2_rn(make_float2(__uint_as_float(r[4 * i]), __uint_as_float(r[4 * i + 1])),
                          make_float2(c.x, c.y));
    g[2 * i + 1] =
        __fadd2_rn(make_float2(__uint_as_float(r[4 * i + 2]), __uint_as_float(r[4 * i + 3])),
                   make_float2(c.z, c.w));
  }
}

template <int W, int NC, bool AU>
__global__ void __launch_bounds__(km_tc_threads(W), 1)
    kmeans_tc_kernel(const __grid_constant__ KmMaps<AU> tm, const __grid_constant__ KmTcArgs a) {
  constexpr int SLOT = km_slot_bytes(AU);
  constexpr int kGroupWarps = 4 * W;
  extern __shared__ uint8_t smem_raw[];
  uint8_t *smem = align_shared(smem_raw, 1024);
  const int nb = a.nb, kp = a.kp, SA = a.sa, S = a.stages;
  const int bblock = kp * 64;  // bytes of one (plane, block) of the centroids
  uint8_t *xring = smem;                                       // [W][SA][SLOT]
  uint8_t *bsm = xring + W * SA * SLOT;                        // [2][nb][kp x 64 B]
  float *cn = reinterpret_cast<float *>(bsm + 2 * nb * bblock);  // [kp]
  uint64_t *xfull = reinterpret_cast<uint64_t *>(cn + kp);     // [W][SA] block landed
  uint64_t *sfull = xfull + W * SA;      // [W][S] stage written
  uint64_t *sempty = sfull + W * S;      // [W][S] the MMAs reading it are done
  uint64_t *accfull = sempty + W * S;    // [W] a pass's MMAs are done
  uint64_t *accempty = accfull + W;      // [W] the accumulator is read
  uint64_t *mmadone = accempty + W;      // every issued MMA has completed
  uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(mmadone + 1);
  float *s_cmax = reinterpret_cast<float *>(tmem_slot + 1);    // [kGroupWarps]
  float *s_top = s_cmax + kGroupWarps;                         // [kGroupWarps]
  unsigned *s_count = reinterpret_cast<unsigned *>(s_top + kGroupWarps);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int64_t tiles = (static_cast<int64_t>(a.np) + kTP - 1) / kTP;
  const int my_tiles = static_cast<int>((tiles - blockIdx.x + gridDim.x - 1) / gridDim.x);
  // tiles, and blocks, of group g
  auto group_tiles = [&](int g) { return my_tiles > g ? (my_tiles - g + W - 1) / W : 0; };

  if (threadIdx.x == 0) {
    for (int i = 0; i < W * SA; ++i) mbar_init(&xfull[i], 1);
    for (int i = 0; i < W * S; ++i) {
      mbar_init(&sfull[i], 4);
      mbar_init(&sempty[i], 1);
    }
    for (int g = 0; g < W; ++g) {
      mbar_init(&accfull[g], 1);
      mbar_init(&accempty[g], 4);
    }
    mbar_init(mmadone, W);
    *s_count = 0u;
    fence_mbar_init();
  }
  if (warp == 1) tmem_alloc(tmem_slot, 512);
  if (warp >= 4) {
    // the centroids' largest magnitude (an infinite one leaves no finite
    // margin, NaN is never taken)
    float top = 0.0f;
    const int t = static_cast<int>(threadIdx.x) - 128, kd = a.k * a.d;
    const int quads = (reinterpret_cast<uintptr_t>(a.cent) & 15u) == 0 ? kd / 4 : 0;
#pragma unroll 8
    for (int e = t; e < quads; e += 32 * kGroupWarps) {
      const float4 v = __ldg(reinterpret_cast<const float4 *>(a.cent) + e);
      top = fmaxf(top, fmaxf(fmaxf(fabsf(v.x), fabsf(v.y)), fmaxf(fabsf(v.z), fabsf(v.w))));
    }
#pragma unroll 8
    for (int e = 4 * quads + t; e < kd; e += 32 * kGroupWarps) top = fmaxf(top, fabsf(a.cent[e]));
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, o));
    if (lane == 0) s_top[warp - 4] = top;
  }
  __syncthreads();

  // Loads the next block of group g's sequence (its tiles one after another,
  // round the ring): tile it, block kb, slot `slot`.
  struct Next {
    int it = 0, kb = 0, slot = 0, phase = 0;
  } ld;
  auto load = [&](int g) {
    const int64_t t = blockIdx.x + (g + static_cast<int64_t>(ld.it) * W) * gridDim.x;
    uint64_t *bar = &xfull[g * SA + ld.slot];
    uint8_t *dst = xring + (g * SA + ld.slot) * SLOT;
    const int kb = ld.kb;
    if (++ld.kb == nb) { ld.kb = 0; ++ld.it; }
    if (++ld.slot == SA) { ld.slot = 0; ld.phase ^= 1; }
    mbar_arrive_expect_tx(bar, SLOT);
    if constexpr (AU) {
#pragma unroll
      for (int r = 0; r < 4; ++r)
        tma_load_2d(dst + r * (36 * 32 * 4), &tm.m[r], bar, kb * 32,
                    static_cast<int>(t * (kTP / 4)));
    } else {
      tma_load_2d(dst, &tm.m[0], bar, kb * 32, static_cast<int>(t * kTP));
    }
  };
  if (warp < W && lane == 0) {
    for (const CUtensorMap &m : tm.m) prefetch_tmap(&m);
    for (int c = 0; c < min(SA, group_tiles(warp) * nb); ++c) load(warp);
  }
  float scale = 1.0f;  // (the point groups')
  if (warp >= 4) {
    float top = s_top[0];
#pragma unroll
    for (int i = 0; i < kGroupWarps; ++i) top = fmaxf(top, s_top[i]);
    scale = km_scale(top);
    // the planes of -2c s (K-major, 64-byte swizzle), norms of c s (+inf past
    // k: never taken) and this warp's largest norm; eight lanes a centroid,
    // two dimensions each at a time
    const int sub = lane & 7;
    float cmax = 0.0f;
    for (int c = 4 * (warp - 4) + (lane >> 3); c < kp; c += 4 * kGroupWarps) {
      const float *row = a.cent + static_cast<int64_t>(c) * a.d;
      float sq = 0.0f;
#pragma unroll 4
      for (int j = 2 * sub; j < 32 * nb; j += 16) {
        const float v0 = c < a.k && j < a.d ? row[j] * scale : 0.0f;
        const float v1 = c < a.k && j + 1 < a.d ? row[j + 1] * scale : 0.0f;
        sq = fmaf(v0, v0, sq);
        sq = fmaf(v1, v1, sq);
        const uint32_t hi = km_f16x2(-2.0f * v0, -2.0f * v1);
        const float2 h = km_f16_pair(hi);
        const uint32_t lo = km_f16x2(__fsub_rn(-2.0f * v0, h.x), __fsub_rn(-2.0f * v1, h.y));
        const int w = (j & 31) >> 1;  // 32-bit word of the 64-byte row
        const int off = (j >> 5) * bblock + c * 64 + (((w >> 2) ^ ((c >> 1) & 3)) << 4) +
                        ((w & 3) << 2);
        *reinterpret_cast<uint32_t *>(bsm + off) = hi;
        *reinterpret_cast<uint32_t *>(bsm + nb * bblock + off) = lo;
      }
      // (kp is a multiple of 16: all lanes of a warp take the same steps)
#pragma unroll
      for (int o = 4; o > 0; o >>= 1) sq += __shfl_xor_sync(0xffffffffu, sq, o);
      if (sub == 0) cn[c] = c < a.k ? sq : INFINITY;
      if (c < a.k) cmax = fmaxf(cmax, sq);
    }
#pragma unroll
    for (int o = 16; o >= 8; o >>= 1) cmax = fmaxf(cmax, __shfl_xor_sync(0xffffffffu, cmax, o));
    if (lane == 0) s_cmax[warp - 4] = cmax;
    fence_proxy_async_smem();  // the MMAs read the planes
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;
  const int P = a.passes;

  if (warp < W) {
    // ---------------------------------------- controller of group `warp`
    if (lane == 0) {
      const int g = warp;
      const uint32_t tacc = tmem + static_cast<uint32_t>(g * (512 / W));
      const uint32_t tA = tacc + static_cast<uint32_t>(NC);
      const uint32_t idesc = idesc_f16(NC);
      const int ksteps = (a.d + 15) / 16;
      const int nt = group_tiles(g);
      int item = 0;          // passes issued
      int s = 0, sphase = 0; // the next block's stage
      // the products of a block against the centroids of pass q
      auto issue = [&](int stage, int kb, int q, bool fresh) {
        uint32_t acc = fresh ? 0u : 1u;
        const uint32_t at = tA + static_cast<uint32_t>(stage * kTcStageCols);
        const uint64_t b0 = sw64_desc(smem_u32(bsm + kb * bblock + q * NC * 64));
        const uint64_t b1 = b0 + static_cast<uint64_t>((nb * bblock) >> 4);
#pragma unroll
        for (int kk = 0; kk < 2; ++kk) {
          if (2 * kb + kk >= ksteps) break;  // dimensions past d are zero
          const uint32_t x0 = at + kk * 8, x1 = x0 + 16;
          mma_bf16_ts(tacc, x1, b0 + kk * 2, idesc, acc);
          mma_bf16_ts(tacc, x0, b1 + kk * 2, idesc, 1u);
          mma_bf16_ts(tacc, x0, b0 + kk * 2, idesc, 1u);
          acc = 1u;
        }
      };
      bool ok = true;
      for (int it = 0; it < nt && ok; ++it) {
        for (int kb = 0; kb < nb && ok; ++kb) {
          ok = mbar_wait(&sfull[g * S + s], sphase, a.err, kDevErrFullBarrier);
          if (!ok) break;
          // the stage is written, so its block's slot has been read
          if (ld.it < nt) load(g);
          if (kb == 0 && item > 0)
            ok = mbar_wait(&accempty[g], (item - 1) & 1, a.err, kDevErrEmptyBarrier);
          if (!ok) break;
          tc_fence_after();
          issue(s, kb, 0, kb == 0);
          if (P == 1) mma_commit(&sempty[g * S + s]);
          if (++s == S) { s = 0; sphase ^= 1; }
        }
        if (!ok) break;
        mma_commit(&accfull[g]);
        ++item;
        // the other passes, from the same stages (S == nb)
        for (int q = 1; q < P && ok; ++q, ++item) {
          ok = mbar_wait(&accempty[g], (item - 1) & 1, a.err, kDevErrEmptyBarrier);
          if (!ok) break;
          tc_fence_after();
          for (int b = 0; b < nb; ++b) issue(b, b, q, b == 0);
          if (q == P - 1)
            for (int b = 0; b < nb; ++b) mma_commit(&sempty[g * S + b]);
          mma_commit(&accfull[g]);
        }
      }
      mma_commit(mmadone);
      // every load issued has landed before the ring is reused: the slots
      // before ld.slot carry this lap's phase, the others the last lap's
      for (int i = 0; i < SA; ++i)
        if (i < ld.slot || ld.it * nb + ld.kb >= SA)
          mbar_wait(&xfull[g * SA + i], i < ld.slot ? ld.phase : ld.phase ^ 1, a.err,
                    kDevErrFullBarrier);
    }
  } else if (warp >= 4) {
    // ------------------------------------------------- point groups
    const int g = (warp - 4) >> 2, w4 = warp & 3;
    const int m = AU ? 4 * lane + w4 : w4 * 32 + lane;  // the point's row of the tile
    const uint32_t tacc = tmem + static_cast<uint32_t>(g * (512 / W)) +
                          (static_cast<uint32_t>(w4 * 32) << 16);  // this warp's lanes
    const uint32_t tA = tacc + static_cast<uint32_t>(NC);
    float cmax = 0.0f;
#pragma unroll
    for (int i = 0; i < kGroupWarps; ++i) cmax = fmaxf(cmax, s_cmax[i]);
    const double nu = (a.d + 4) * 0x1p-24;
    const float bound = static_cast<float>((16.0 * nu / (1.0 - nu) + 0x1p-19) * 1.001);
    // (in scaled units) sums of norms from which everything is a candidate --
    // near the end of FP32's range unscaled, or of FP16's -- and what the
    // margin is at least
    const float most = fminf(1e36f * scale * scale, 0x1p31f);
    const float least = 1e-37f * scale * scale;
    const float inv = 1.0f / scale;  // a power of two too
    const float2 scale2 = make_float2(scale, scale);
    [[maybe_unused]] const int e_w = AU ? a.e[w4] : 0;

    // Splits the next block of the group's sequence into its TMEM stage and
    // adds the block's part of ||x||^2; false when a wait expired.  (The first
    // lap's wait for a free stage passes: the phase before the first.)
    int slot = 0, xphase = 0, s = 0, sphase = 0;
    auto convert = [&](float2 &xn) -> bool {
      const bool ok = mbar_wait2(&xfull[g * SA + slot], xphase, &sempty[g * S + s], sphase ^ 1,
                                 a.err, kDevErrFullBarrier);
      if (!__all_sync(0xffffffffu, ok)) return false;
      tc_fence_after();
      const float *xs = reinterpret_cast<const float *>(xring + (g * SA + slot) * SLOT);
      float2 x[16];
      if constexpr (AU) {
        // 36 floats of the lane's row (rows 144 bytes apart), the block's 32
        // from e_w on
        const float *row = xs + w4 * (36 * 32) + lane * 36;
        float y[36];
#pragma unroll
        for (int i = 0; i < 9; ++i) {
          const float4 v = *reinterpret_cast<const float4 *>(row + 4 * i);
          y[4 * i] = v.x; y[4 * i + 1] = v.y; y[4 * i + 2] = v.z; y[4 * i + 3] = v.w;
        }
        auto shift = [&](auto e) {
#pragma unroll
          for (int i = 0; i < 16; ++i) x[i] = make_float2(y[2 * i + e.value], y[2 * i + 1 + e.value]);
        };
        switch (e_w) {  // uniform over the warp
          case 0: shift(std::integral_constant<int, 0>()); break;
          case 1: shift(std::integral_constant<int, 1>()); break;
          case 2: shift(std::integral_constant<int, 2>()); break;
          default: shift(std::integral_constant<int, 3>()); break;
        }
      } else {
        // row m: 32 floats in 128 bytes, 128-byte swizzle
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const float4 v = *reinterpret_cast<const float4 *>(xs + m * 32 + ((i ^ (m & 7)) * 4));
          x[2 * i] = make_float2(v.x, v.y);
          x[2 * i + 1] = make_float2(v.z, v.w);
        }
      }
      uint32_t hi[16], lo[16];
#pragma unroll
      for (int i = 0; i < 16; ++i) {
        x[i] = __fmul2_rn(x[i], scale2);
        xn = __ffma2_rn(x[i], x[i], xn);
        hi[i] = km_f16x2(x[i].x, x[i].y);
        const float2 r = km_residual(hi[i], x[i]);
        lo[i] = km_f16x2(r.x, r.y);
      }
      const uint32_t dst = tA + static_cast<uint32_t>(s * kTcStageCols);
      tmem_st16(dst, hi);
      tmem_st16(dst + 16u, lo);
      tmem_wait_st();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&sfull[g * S + s]);
      if (++slot == SA) { slot = 0; xphase ^= 1; }
      if (++s == S) { s = 0; sphase ^= 1; }
      return true;
    };

    const int nt = group_tiles(g);
    // blocks of the next tile split before this tile's argmin: at most what
    // leaves the stages and the ring a block short of full
    const int ahead = P > 1 ? 0 : min(nb, min(S - 1, SA));
    float2 xn = make_float2(0.0f, 0.0f);
    int done = 0, item = 0;
    bool ok = true;
    for (int it = 0; it < nt && ok; ++it) {
      for (; done < nb && ok; ++done) ok = convert(xn);
      float2 xnext = make_float2(0.0f, 0.0f);
      done = 0;
      if (it + 1 < nt)
        for (; done < ahead && ok; ++done) ok = convert(xnext);
      if (!ok) break;
      const float xsum = xn.x + xn.y + cmax;
      xn = xnext;
      const float margin = xsum < most ? bound * xsum + least : INFINITY;
      float g1 = INFINITY;  // the smallest g of the passes so far
      int k1 = 0;           // its centroid, when the only candidate
      bool close = true;
      for (int q = 0; q < P; ++q, ++item) {
        ok = mbar_wait(&accfull[g], item & 1, a.err, kDevErrMmaBarrier);
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) break;
        tc_fence_after();
        float2 gv[NC / 2];
        {
          uint32_t r[NC / 16][16];
#pragma unroll
          for (int h = 0; h < NC / 16; ++h) tmem_ld16(tacc + 16 * h, r[h]);
          tmem_wait_ld();
          const uint32_t cq = smem_u32(cn + q * NC);
#pragma unroll
          for (int h = 0; h < NC / 16; ++h) km_g16(r[h], cq + 64 * h, gv + 8 * h);
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&accempty[g]);
        // the pass's smallest (minima skip a NaN g, whose distance the
        // reference never takes either)
        float mc[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) mc[i] = fminf(gv[i].x, gv[i].y);
#pragma unroll
        for (int i = 4; i < NC / 2; ++i) mc[i & 3] = min3(mc[i & 3], gv[i].x, gv[i].y);
        const float m0 = fminf(min3(mc[0], mc[1], mc[2]), mc[3]);
        // the candidates, from the signs of g - lim: centroid i of the pass
        // is bit 31 - i % 32 of word i / 32
        const float nl = -(m0 + margin);
        uint32_t half[NC / 16] = {};
#pragma unroll
        for (int i = 0; i < 8; ++i)
#pragma unroll
          for (int h = 0; h < NC / 16; ++h) {
            const float2 t = __fadd2_rn(gv[8 * h + i], make_float2(nl, nl));
            half[h] = __funnelshift_l(__float_as_uint(t.x), half[h], 1);
            half[h] = __funnelshift_l(__float_as_uint(t.y), half[h], 1);
          }
        int cand = 0, kq = 0;
#pragma unroll
        for (int h = NC / 16 - 1; h >= 0; --h) {
          cand += __popc(half[h]);
          if (half[h]) kq = q * NC + 16 * h + __clz(half[h]) - 16;
        }
        // union with the passes before: alone only where the other side's
        // smallest lies beyond the margin
        if (m0 + margin < g1) {
          g1 = m0;
          k1 = kq;
          close = cand != 1;
        } else {
          close = close || !(g1 + margin < m0);
          g1 = fminf(g1, m0);
        }
      }
      if (!ok) break;
      const int64_t p = (blockIdx.x + (g + static_cast<int64_t>(it) * W) * gridDim.x) * kTP + m;
      const bool live = p < a.np;
      const float lim = margin < INFINITY ? (g1 + margin) * inv * inv : INFINITY;
      close = live && (close || !(lim < INFINITY));
      if (live && !close) a.out[p] = static_cast<uint32_t>(k1);
      const unsigned vote = __ballot_sync(0xffffffffu, close);
      if (vote) {
        unsigned base = 0;
        if (lane == 0) base = atomicAdd(s_count, static_cast<unsigned>(__popc(vote)));
        base = __shfl_sync(0xffffffffu, base, 0) + __popc(vote & ((1u << lane) - 1u));
        if (close)
          a.citems[static_cast<int64_t>(blockIdx.x) * a.list + base] =
              make_uint2(static_cast<uint32_t>(p), __float_as_uint(lim));
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    // the TMEM is freed only once every issued MMA has completed
    if (lane == 0) mbar_wait(mmadone, 0, a.err, kDevErrMmaBarrier);
    __syncwarp();
    tc_fence_after();
    tmem_dealloc(tmem, 512);
  }
  // ------------------------------------- the CTA's close calls
  const unsigned n = *s_count;
  if (n == 0) return;
  if (a.exact && threadIdx.x == 0) atomicAdd(a.exact, n);
  // the centroids in FP32 over the ring and the planes, padded rows of d + 1
  float *cs = reinterpret_cast<float *>(smem);
  for (int c = warp; c < a.k; c += km_tc_threads(W) / 32)
    for (int j = lane; j < a.d; j += 32) cs[c * (a.d + 1) + j] = a.cent[static_cast<int64_t>(c) * a.d + j];
  if (warp >= 4)
    for (int c = static_cast<int>(threadIdx.x) - 128; c < a.k; c += 32 * kGroupWarps)
      cn[c] = cn[c] / scale / scale;  // the norms unscaled
  __syncthreads();
  if (warp < 4) return;
  float *xs = cs + up4(a.k * (a.d + 1)) + (warp - 4) * up4(a.d);
  for (unsigned i = warp - 4; i < n; i += kGroupWarps) {
    const uint2 it = a.citems[static_cast<int64_t>(blockIdx.x) * a.list + i];
    const float *x = a.points + static_cast<int64_t>(it.x) * a.d;
    for (int j = lane; j < a.d; j += 32) xs[j] = x[j];
    __syncwarp();
    const uint32_t pick = exact_pick_smem(xs, a.d, cs, a.k, cn, __uint_as_float(it.y));
    if (lane == 0) a.out[it.x] = pick;
    __syncwarp();  // xs is rewritten for the warp's next entry
  }
}

// The call's workspace (the stream's second slot): `extra` bytes for the
// form (the products or the centroid planes), ||c||^2, and the close-call
// list (a count, then room for every point).
struct KmWs {
  uint8_t *extra;
  float *cnorm;
  unsigned *ccount;
  uint2 *citems;
};

hml_status km_workspace(size_t extra, int np, int k, cudaStream_t s, KmWs *w) {
  auto up = [](size_t b) { return (b + 255) & ~static_cast<size_t>(255); };
  const size_t o_norm = up(extra), o_cnt = o_norm + up(static_cast<size_t>(k) * sizeof(float));
  const size_t o_items = o_cnt + 256;
  void *ws = nullptr;
  hml_status st = workspace_slot(1, o_items + static_cast<size_t>(np) * sizeof(uint2), s, &ws);
  if (st != HML_STATUS_SUCCESS) return st;
  uint8_t *b = static_cast<uint8_t *>(ws);
  w->extra = b;
  w->cnorm = reinterpret_cast<float *>(b + o_norm);
  w->ccount = reinterpret_cast<unsigned *>(b + o_cnt);
  w->citems = reinterpret_cast<uint2 *>(b + o_items);
  return HML_STATUS_SUCCESS;
}

// ||c||^2 and an empty close-call list; first in the SIMT and SGEMM forms.
hml_status launch_norms(const float *cent, int k, int d, const KmWs &w, cudaStream_t s) {
  count_launch();
  const int nb = std::min((k + kNormWarps - 1) / kNormWarps, 4 * sm_count());
  centroid_norms_kernel<<<std::max(1, nb), 32 * kNormWarps, 0, s>>>(cent, k, d, w.cnorm,
                                                                     w.ccount);
  cudaError_t e = cudaGetLastError();
  note_cuda_error(e, "kmeans norms");
  return cuda_status(e);
}

// The close calls the screening kernel listed; last in the SIMT and SGEMM
// forms.
hml_status launch_settle(const float *points, int d, const float *cent, int k, const KmWs &w,
                         uint32_t *out, unsigned *exact, cudaStream_t s) {
  // the centroids, norms and point rows in shared memory when they fit
  const int staged = settle_smem_floats(k, d) <= kSettleSmemFloats ? 1 : 0;
  const size_t smem = staged ? static_cast<size_t>(settle_smem_floats(k, d)) * 4 : 0;
  cudaError_t e = cudaSuccess;
  if (smem > 48 * 1024)
    e = cudaFuncSetAttribute(kmeans_settle_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             static_cast<int>(smem));
  if (e == cudaSuccess)
    e = launch_k_ex(kmeans_settle_kernel, dim3(2 * sm_count()), dim3(256), smem, s, 1, false,
                    points, d, cent, k, static_cast<const float *>(w.cnorm),
                    static_cast<const unsigned *>(w.ccount),
                    static_cast<const uint2 *>(w.citems), out, exact, staged);
  note_cuda_error(e, "kmeans settle");
  return cuda_status(e);
}

// The tiled SIMT form (method 1).
hml_status assign_tiled(const float *points, int np, int d, const float *cent, int k,
                        uint32_t *out, unsigned *exact, cudaStream_t s) {
  KmWs w;
  hml_status st = km_workspace(0, np, k, s, &w);
  if (st == HML_STATUS_SUCCESS) st = launch_norms(cent, k, d, w, s);
  if (st != HML_STATUS_SUCCESS) return st;
  const int64_t blocks = (static_cast<int64_t>(np) + kTP - 1) / kTP;
  const int dp = (d + 3) & ~3, kp = (k + kTC - 1) / kTC * kTC;
  cudaError_t e = cudaSuccess;
  count_launch();
  if (d > 0 && dp <= 64 && static_cast<int64_t>(dp) * kp <= kResidentFloats) {
    const size_t smem =
        (static_cast<size_t>(dp) * (kp + 4) + kp + 2 * kTP * dp + kTP) * sizeof(float);
    e = cudaFuncSetAttribute(kmeans_resident_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             static_cast<int>(smem));
    // 16-byte row copies when every row starts on a 16-byte boundary
    const bool vec = d % 4 == 0 && (reinterpret_cast<uintptr_t>(points) & 15u) == 0;
    const int64_t grid = std::min<int64_t>(blocks, 2LL * sm_count());
    if (e == cudaSuccess)
      kmeans_resident_kernel<<<static_cast<unsigned>(grid), kTThreads, smem, s>>>(
          points, np, d, dp, vec, cent, k, kp, w.cnorm, out, w.ccount, w.citems);
  } else {
    kmeans_tile_kernel<<<static_cast<unsigned>(blocks), kTThreads, 0, s>>>(
        points, np, d, cent, k, w.cnorm, out, w.ccount, w.citems);
  }
  if (e == cudaSuccess) e = cudaGetLastError();
  note_cuda_error(e, "kmeans tiled");
  if (e != cudaSuccess) return cuda_status(e);
  return launch_settle(points, d, cent, k, w, out, exact, s);
}

// The GEMM form (method 2): S = X C^T through the library's SGEMM, then the
// pick kernel.
hml_status assign_gemm(const float *points, int np, int d, const float *cent, int k,
                       uint32_t *out, unsigned *exact, cudaStream_t s) {
  const size_t s_bytes = static_cast<size_t>(np) * k * sizeof(float);
  KmWs w;
  hml_status st = km_workspace(s_bytes, np, k, s, &w);
  if (st != HML_STATUS_SUCCESS) return st;
  float *S = reinterpret_cast<float *>(w.extra);
  // S (points x clusters, column-major) = X C^T: X is the row-major points
  // (column-major d x np, transposed), C^T the row-major centroids
  // (column-major d x k)
  if (d > 0) {
    GemmProblem p;
    st = gemm_from_blas(HML_COL_MAJOR, HML_OP_T, HML_OP_N, np, k, d, 1.0f, points, d, cent, d,
                        0.0f, S, np, &p);
    if (st != HML_STATUS_SUCCESS) return st;
    GemvProblem g;
    if (as_gemv(p, &g)) {
      st = launch_gemv(g, kGemvTuned, s);
    } else {
      hml_sgemm_config c;
      st = select_config(p, &c, s);
      // the candidate bound assumes FP32-level dot products
      if (st == HML_STATUS_SUCCESS && c.algo == HML_ALGO_BF16X3) {
        c = heuristic_config(p, HML_ALGO_BF16X6);
        if (!check_config_ok(p, c)) c = heuristic_config(p, HML_ALGO_SIMT);
      }
      if (st == HML_STATUS_SUCCESS) st = run_config(p, c, s);
    }
    if (st != HML_STATUS_SUCCESS) return st;
  } else {
    cudaError_t e = cudaMemsetAsync(S, 0, s_bytes, s);
    if (e != cudaSuccess) {
      note_cuda_error(e, "kmeans: zero products");
      return HML_STATUS_CUDA_ERROR;
    }
  }
  st = launch_norms(cent, k, d, w, s);
  if (st != HML_STATUS_SUCCESS) return st;
  count_launch();
  cudaError_t e = cudaSuccess;
  const size_t smem = static_cast<size_t>(k) * sizeof(float);
  if (smem > 48 * 1024) {
    e = cudaFuncSetAttribute(kmeans_pick_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             static_cast<int>(smem));
  }
  if (e == cudaSuccess) {
    const int64_t blocks = std::min<int64_t>((np + 255) / 256, 8LL * sm_count());
    kmeans_pick_kernel<<<static_cast<unsigned>(blocks), 256, smem, s>>>(
        points, np, d, k, S, np, w.cnorm, out, w.ccount, w.citems);
    e = cudaGetLastError();
  }
  note_cuda_error(e, "kmeans assign");
  if (e != cudaSuccess) return cuda_status(e);
  return launch_settle(points, d, cent, k, w, out, exact, s);
}

// Rows that TMA addresses as they stand: whole 16-byte granules.
bool km_rows_aligned(const float *points, int d) {
  return d % 4 == 0 && (reinterpret_cast<uintptr_t>(points) & 15u) == 0;
}

// What method 3 accepts: points with 4 <= dims <= 64 (a multiple of 4, rows
// 16-byte aligned) and at most 256 centroids.
bool tc_form_applies(const float *points, int d, int k) {
  return d >= 4 && km_rows_aligned(points, d) && d <= 64 && k <= kTcMaxK;
}

// How the tensor-core kernel runs a shape; false when it cannot.
struct KmTcPlan {
  int W, nb, kp, nc, passes, stages, sa;
  bool au;
  size_t smem;
};
bool km_tc_plan(const float *points, int np, int d, int k, KmTcPlan *out) {
  KmTcPlan p;
  p.au = !km_rows_aligned(points, d);
  // (four row classes; a smaller n leaves a class without a row to address)
  if (d < 1 || k < 1 || k > kTcMaxK || (p.au && np < 4) ||
      (reinterpret_cast<uintptr_t>(points) & 3u) != 0)
    return false;
  p.nb = (d + 31) / 32;
  const size_t slot = km_slot_bytes(p.au);
  const size_t budget = 220 * 1024;
  auto planes = [&](int kp) { return static_cast<size_t>(4) * kp * 32 * p.nb; };
  auto width = [](int n) { return n <= 16 ? 16 : n <= 32 ? 32 : n <= 64 ? 64 : 128; };
  p.passes = 1;
  // four groups while an accumulator of 64 columns and two stages serve the
  // shape (more centroids in passes over up to 64 resident dimensions) and
  // two slots a group fit beside the planes; else two groups, an accumulator
  // of 128 columns and four stages
  p.W = 4;
  p.nc = std::min(64, width(k));
  p.passes = (k + p.nc - 1) / p.nc;
  p.kp = p.passes * p.nc;
  if ((p.passes > 1 && p.nb > 2) || planes(p.kp) + 8 * slot > budget) {
    p.W = 2;
    p.nc = std::max(64, width(k));
    p.passes = (k + p.nc - 1) / p.nc;
    p.kp = p.passes * p.nc;
  }
  p.stages = std::min(4, (512 / p.W - p.nc) / kTcStageCols);
  if (p.passes > 1) {
    if (p.nb > p.stages) return false;
    p.stages = p.nb;
  }
  if (planes(p.kp) > kTcMaxPlanes) return false;
  p.sa = static_cast<int>(std::min<size_t>(4, (budget - planes(p.kp)) / (p.W * slot)));
  if (p.sa < 2) return false;
  const int bars = p.W * (p.sa + 2 * p.stages + 2) + 1;
  p.smem = 1024 + p.W * p.sa * slot + planes(p.kp) + static_cast<size_t>(p.kp) * 4 + bars * 8 +
           (1 + 8 * p.W + 1) * 4 + 16;
  // the close calls' centroids and point rows reuse the ring and the planes
  const size_t settle = static_cast<size_t>(up4(static_cast<int64_t>(k) * (d + 1)) + 4 * p.W * up4(d)) * 4;
  if (settle > p.W * p.sa * slot + planes(p.kp) || p.smem > 227 * 1024) return false;
  p.smem = std::max<size_t>(p.smem, 120 * 1024);  // one CTA per SM: all 512 TMEM columns
  *out = p;
  return true;
}

template <int W, int NC, bool AU>
hml_status launch_km_tc(const KmMaps<AU> &tm, const KmTcArgs &a, int grid, size_t smem,
                        cudaStream_t s) {
  auto kern = kmeans_tc_kernel<W, NC, AU>;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       static_cast<int>(smem));
  if (e == cudaSuccess) e = launch_k(kern, dim3(grid), dim3(km_tc_threads(W)), smem, s, 1, tm, a);
  note_cuda_error(e, "kmeans tensor-core");
  return cuda_status(e);
}

template <bool AU>
hml_status assign_tc_rows(const KmTcPlan &p, const float *points, int np, int d,
                          const float *cent, int k, uint32_t *out, unsigned *exact,
                          cudaStream_t s) {
  const int64_t tiles = (static_cast<int64_t>(np) + kTP - 1) / kTP;
  const int grid = static_cast<int>(std::min<int64_t>(tiles, sm_count()));
  KmTcArgs a = {};
  a.list = static_cast<int>((tiles + grid - 1) / grid) * kTP;
  void *ws = nullptr;
  hml_status st =
      workspace_slot(1, static_cast<size_t>(grid) * a.list * sizeof(uint2), s, &ws);
  if (st != HML_STATUS_SUCCESS) return st;
  a.points = points;
  a.cent = cent;
  a.np = np;
  a.d = d;
  a.k = k;
  a.nb = p.nb;
  a.kp = p.kp;
  a.passes = p.passes;
  a.stages = p.stages;
  a.sa = p.sa;
  a.out = out;
  a.citems = static_cast<uint2 *>(ws);
  a.exact = exact;
  a.err = device_error_word();
  KmMaps<AU> tm;
  memset(&tm, 0, sizeof tm);
  if constexpr (AU) {
    for (int r = 0; r < 4; ++r) {
      const LineClass c4 = line_class(points, d, np, d, r);
      a.e[r] = c4.skip;
      if (!tensor_map_2d(&tm.m[r], CU_TENSOR_MAP_DATA_TYPE_FLOAT32, c4.base, c4.len, c4.lines,
                         c4.stride, 36, 32, CU_TENSOR_MAP_SWIZZLE_NONE))
        return HML_STATUS_CUDA_ERROR;
    }
  } else if (!tensor_map_2d(&tm.m[0], CU_TENSOR_MAP_DATA_TYPE_FLOAT32, points, d, np,
                            static_cast<uint64_t>(d) * 4, 32, kTP, CU_TENSOR_MAP_SWIZZLE_128B)) {
    return HML_STATUS_CUDA_ERROR;
  }
  if (p.W == 2)
    return p.nc == 64 ? launch_km_tc<2, 64, AU>(tm, a, grid, p.smem, s)
                      : launch_km_tc<2, 128, AU>(tm, a, grid, p.smem, s);
  return p.nc == 16   ? launch_km_tc<4, 16, AU>(tm, a, grid, p.smem, s)
         : p.nc == 32 ? launch_km_tc<4, 32, AU>(tm, a, grid, p.smem, s)
                      : launch_km_tc<4, 64, AU>(tm, a, grid, p.smem, s);
}

// The tensor-core form (method 3).
hml_status assign_tc(const float *points, int np, int d, const float *cent, int k,
                     uint32_t *out, unsigned *exact, cudaStream_t s) {
  KmTcPlan p;
  if (!km_tc_plan(points, np, d, k, &p)) return HML_STATUS_NOT_SUPPORTED;
  return p.au ? assign_tc_rows<true>(p, points, np, d, cent, k, out, exact, s)
              : assign_tc_rows<false>(p, points, np, d, cent, k, out, exact, s);
}

}  // namespace

hml_status kmeans_assign(const float *points, int np, int d, const float *cent, int k,
                         uint32_t *out, int method, unsigned *exact, cudaStream_t s) {
  if (np < 0 || d < 0 || k < 1 || method < 0 || method > 3) return HML_STATUS_INVALID_VALUE;
  if (np == 0) return HML_STATUS_SUCCESS;
  if (!out || (d > 0 && (!points || !cent))) return HML_STATUS_INVALID_VALUE;
  // the pick kernel keeps ||c||^2 of every centroid in shared memory
  if (method == 2 && static_cast<size_t>(k) * sizeof(float) > 200 * 1024)
    return HML_STATUS_NOT_SUPPORTED;
  if (method == 3 && !tc_form_applies(points, d, k)) return HML_STATUS_NOT_SUPPORTED;
  if (method == 0) {
    // the tensor-core kernel wherever it can run the shape
    KmTcPlan plan;
    method = km_tc_plan(points, np, d, k, &plan) ? 3 : d <= kKmeansTiledMaxDims ? 1 : 2;
    if (method == 2 && static_cast<size_t>(k) * sizeof(float) > 200 * 1024) method = 1;
  }
  switch (method) {
    case 1: return assign_tiled(points, np, d, cent, k, out, exact, s);
    case 2: return assign_gemm(points, np, d, cent, k, out, exact, s);
    default: return assign_tc(points, np, d, cent, k, out, exact, s);
  }
}

}  // namespace hml

extern "C" hml_status hml_kmeans_assign(const float *points, int num_points, int dims,
                                        const float *centroids, int num_clusters,
                                        uint32_t *assignments, void *stream) {
  return hml::kmeans_assign(points, num_points, dims, centroids, num_clusters, assignments, 0,
                            nullptr, static_cast<cudaStream_t>(stream));
}

extern "C" hml_status hml_kmeans_assign_ex(const float *points, int num_points, int dims,
                                           const float *centroids, int num_clusters,
                                           uint32_t *assignments, int method,
                                           unsigned *exact_count, void *stream) {
  return hml::kmeans_assign(points, num_points, dims, centroids, num_clusters, assignments,
                            method, exact_count, static_cast<cudaStream_t>(stream));
}
