// sgemm_tc.cu -- split-BF16 SGEMM on the B200 tensor cores (tcgen05 + TMEM).
//
// FP32 operands are split into BF16 terms, a = a0 + a1 (+ a2), each term the
// BF16 rounding of what the previous terms left (every residual is exact in
// FP32), and the products that carry FP32-level information are accumulated
// in FP32:
//   BF16X3: a0*b0 + a0*b1 + a1*b0                          (2 planes, 3 MMAs)
//   BF16X6: a0*b0 + a0*b1 + a1*b0 + a0*b2 + a1*b1 + a2*b0  (3 planes, 6 MMAs)
// and two explicit forms with 11-bit planes: TF32X3 (kind::tf32) and FP16X3
// (FP16 hi/lo planes of operands scaled by powers of two: per row of each
// 32-deep block of A, per column of B; each block is accumulated in TMEM on
// its own and rescaled by the drain).
// The result is C = alpha * A * B + beta * C in FP32, the reference's
// hmlSgemm contract (src/hml_sgemm.cu:120-211) on a different machine.
//
// Data flow of one CTA (a 128-row tile of C, BN columns, a K range), in
// 32-deep K blocks:
//   * B is small (K x N): a pre-pass splits it once into BF16 planes stored
//     K-contiguous in a workspace ([plane][N_pad][K_pad]); a TMA warp loads
//     plane tiles straight into the UMMA canonical K-major layout (64-byte
//     swizzle, 32 BF16 per row).
//   * A streams from HBM exactly once: a TMA warp loads 128 x 32 FP32 tiles
//     into a ring of shared-memory slots.
//   * G converter warpgroups take the blocks round-robin (group g converts
//     blocks g, g+G, ...), so G blocks are in conversion at once.  Thread m of
//     a group owns row m of the tile, which is also TMEM lane m: it reads the
//     row's 32 FP32 values, splits them, and writes the BF16 planes into a
//     TMEM stage with tcgen05.st (two BF16 per 32-bit column).  The MMAs read
//     A from TMEM (the tcgen05.mma form with A in tensor memory), so the
//     converted planes never touch shared memory.
//   * NI threads (2 to 4, one per accumulator) issue tcgen05.mma (M=128,
//     N=BN, K=16; A from TMEM, B from shared memory; FP32 accumulator in
//     TMEM), each for every NI-th 64-deep chunk, and release each operand
//     stage (B slot + A stage) with one tcgen05.commit.
//   * the tensor core's FP32 accumulation truncates, so a long accumulation
//     chain in TMEM loses accuracy as K grows.  Each 64-deep chunk of K is
//     accumulated into one of NI TMEM accumulators; drain warpgroups read it
//     (tcgen05.ld) and add it into FP32 running sums held in registers
//     (round to nearest) while the tensor core fills the others.
//   * the drain warps apply alpha/beta; with split_k > 1 the CTAs of one
//     thread-block cluster sum their tiles in rank order through distributed
//     shared memory.
// Every wait is bounded (2 s of %globaltimer); on expiry the device error
// word is set, the CTA skips ahead, waits for its issued MMAs, frees its TMEM
// and returns.
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include <algorithm>
#include <cfloat>
#include <cstring>
#include <mutex>
#include <new>
#include <type_traits>
#include <utility>
#include <vector>

#include "hml_device.cuh"
#include "hml_internal.h"
#include "hml_lines.h"
#include "hml_tcgen05.cuh"
#include "hml_walk.h"

// The forms are compiled into a module each, so that a program loads the one it
// uses: this file alone is BF16X6 with the batches, and sgemm_tc_x3.cu, _tf32.cu
// and _fp16.cu include it for the others (HML_TC_PART is their NS).  The first
// call of a process took 28 ms with one module of all, 12 so.
#ifndef HML_TC_PART
#define HML_TC_PART 0
#endif

namespace hml {
namespace {

constexpr int kBM = 128;      // rows of C per CTA = UMMA M = TMEM lanes
constexpr int kBK = 32;       // K per block (one 64-byte BF16 swizzle row)
constexpr int kChunkK = 64;   // K accumulated in TMEM before an FP32 drain
constexpr int kTmemCols = 512;

// Tile shapes: 128-row tiles, one per CTA.  (256-row tiles on a CTA pair,
// tcgen05.mma.cta_group::2, were bitwise equal but slower on every measured
// shape -- the cross-CTA handshakes cost about 1 us per 32-deep block -- and
// are not built.)
struct TcShape {
  int bm, bn;
};
constexpr TcShape kTcShapes[] = {{128, 16}, {128, 32}, {128, 64}, {128, 128}};
constexpr int kNumTcShapes = sizeof(kTcShapes) / sizeof(kTcShapes[0]);

// How A reaches shared memory.  TMA needs 16-byte aligned bases and strides;
// an A without them (an odd leading dimension, a shifted base) is still read
// by TMA, through four maps: the strided lines of A (columns of an
// M-contiguous A, rows of a K-contiguous one) with index = r mod 4 lie 4 *
// ld * 4 bytes apart, a multiple of 16, and start e_r = 0..3 floats past a
// 16-byte boundary.  Map r covers class r from that boundary on, its boxes
// are 4 floats wider than the block, and the converters skip the e_r floats.
// (Against the 4-byte cp.async SIMT tiles that served these problems before:
// 20011 x 45 x 1501 row-major, 293 us -> 52 us a call on B200, A at 2.4 TB/s;
// what bounds it is the aligned form's converter and handshake pace.)
enum AMode : int {
  kAM = 0,   // M-contiguous: one 32 (k) x 128 (m) box a block
  kAK = 1,   // K-contiguous: one 128 (m) x 32 (k) box, 128-byte swizzle
  kAMU = 2,  // M-contiguous, unaligned: four 8 (k) x 132 (m) boxes
  kAKU = 3,  // K-contiguous, unaligned: four 32 (m) x 36 (k) boxes
};
__host__ __device__ constexpr bool am_kcontig(int am) { return am == kAK || am == kAKU; }
__host__ __device__ constexpr bool am_unaligned(int am) { return am >= kAMU; }
// The unaligned forms, which take the place of FP32 tiles, scale both operands
// by 2^16 before they are split: the third BF16 plane of an element below 2^-110
// would otherwise need bits below BF16's smallest subnormal, 2^-133 (with the
// scale every FP32 value, 2^-149 itself included, splits exactly).  Sums carry
// 2^32 until they are stored; one that leaves FP32's range for it is formed
// again in plain FP32 like every sum that is not finite.
constexpr float kAUScale = 0x1p16f, kAUUnscale = 0x1p-32f;
// The maps of A (one, or one per class) and the class offsets e_r.
template <int AM>
struct AMaps {
  CUtensorMap m[am_unaligned(AM) ? 4 : 1];
};

// Warp roles of one CTA:
//   warp 0       TMA loads of A (FP32 tiles)
//   warp 1       TMA loads of B (BF16 plane tiles)
//   warps 2..    NI MMA issuers (warp 2 also allocates TMEM); issuer i takes
//                the 64-deep chunks q = i, i+NI, ... into accumulator i
//   then, from the next warp index divisible by 4: G converter warpgroups,
//   then D drain warpgroups.
// A warp can reach only TMEM lanes 32 * (warp % 4) .. +31, so every
// warpgroup that touches TMEM starts at a warp index divisible by 4 and its
// warp q covers rows 32q .. 32q+31.
//
// Each thread's tcgen05.mma issue is serial (tens of ns an instruction), so
// at small N one thread cannot keep up with the HBM stream; NI threads issue
// into NI accumulators.  TMEM holds the NI accumulators (BN columns each)
// and so A stages (NS x 16 columns each, two BF16 per 32-bit column).
__host__ __device__ constexpr int tc_groups() { return 2; }
__host__ __device__ constexpr int tc_drain_groups(int bn) { return bn > 64 ? 2 : 1; }
// BF16-plane equivalents of a form's operand planes: NS = 2 and 3 (BF16X3,
// BF16X6), 4 (TF32X3: two 32-bit planes), 5 (FP16X3: two FP16 planes).
__host__ __device__ constexpr int tc_geom(int ns) { return ns == 5 ? 2 : ns; }
// TMEM columns of one converted A block: NS planes x 32 BF16 (2 per column).
__host__ __device__ constexpr int tc_stage_cols(int ns) { return tc_geom(ns) * kBK / 2; }
// Operand stages (B slot + A TMEM stage) with ni issuers: a multiple of
// 2 * ni (blocks per chunk x issuers), so that every stage is only ever used
// by one issuer and, as 2 * ni is even, by one converter group; at most 8.
__host__ __device__ constexpr int tc_stage_mult(int ni) { return 2 * ni; }
__host__ __device__ constexpr int tc_stages_for(int bn, int ns, int ni) {
  return (((kTmemCols - ni * bn) / tc_stage_cols(ns) < 8 ? (kTmemCols - ni * bn) /
                                                               tc_stage_cols(ns)
                                                         : 8) /
          tc_stage_mult(ni)) *
         tc_stage_mult(ni);
}
// The most issuers (4 at most, 2 at least) whose accumulators leave room
// for at least one stage multiple.
__host__ __device__ constexpr int tc_issuers(int bn, int ns) {
  return tc_stages_for(bn, ns, 4) >= tc_stage_mult(4)   ? 4
         : tc_stages_for(bn, ns, 3) >= tc_stage_mult(3) ? 3
                                                        : 2;
}
__host__ __device__ constexpr int tc_max_stages(int bn, int ns) {
  return tc_stages_for(bn, ns, tc_issuers(bn, ns));
}
__host__ __device__ constexpr int tc_conv_warp0(int bn, int ns) {
  return ((2 + tc_issuers(bn, ns) + 3) / 4) * 4;
}
__host__ __device__ constexpr int tc_warps(int bn, int ns) {
  return tc_conv_warp0(bn, ns) + 4 * tc_groups() + 4 * tc_drain_groups(bn);
}


// Split eight floats into NS BF16 planes, t0 = bf16(x), t1 = bf16(x - t0),
// ... (each residual is exact in FP32), packed two per 32-bit word with
// cvt.rn.bf16x2.f32 (the lower k in the low half, as in memory order).
__device__ __forceinline__ uint32_t bf16x2_rn(float lo, float hi) {
  uint32_t r;
  asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(hi), "f"(lo));
  return r;
}

// Releasing a shared-memory slot for the warp takes every lane's values to be
// in: a __syncwarp before one lane's arrival neither waits for the other
// lanes' loads to return nor keeps their use from being scheduled behind it,
// and TMA refills the slot at once (a build with registers to spare did so,
// and lost rows).  A slot is released after the block's first TMEM store,
// which takes words of values from all of the row -- except (EARLY) in a ring of
// 2 or 4 slots, which cannot wait for the operand stage that store needs (8192^3
// with 2 slots 5.95 ms, 6.58 with the later release; 18944 x 64 x 4096 with 4
// 74.8 us, 77.0), and in 128-wide BF16 tiles at any depth (18944 x 128 x 4096, 8 slots,
// 100.1 us, 104.2; 20000 x 300 x 6144 518, 540; narrower tiles do better later:
// 18944 x 16 x 4096 row-major 64.8, 62.2): there the arriving lane comes from a
// vote on words w computed from every value.
template <int N>
__device__ __forceinline__ void release_early(uint64_t *bar, const uint32_t (&w)[N], int lane) {
  uint32_t all = w[0];
#pragma unroll
  for (int i = 1; i < N; ++i) all |= w[i];
  const uint32_t vote = __ballot_sync(0xffffffffu, all != 0x5bd1e995u);
  if (lane == (vote ? __ffs(vote) - 1 : 0)) mbar_arrive(bar);
}

template <int NS>
__device__ __forceinline__ void pack8(const float (&x)[8], uint4 (&out)[NS]) {
  uint32_t w[NS][4];
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    float a = x[2 * j], b = x[2 * j + 1];
#pragma unroll
    for (int i = 0; i < NS; ++i) {
      const uint32_t t = bf16x2_rn(a, b);
      w[i][j] = t;
      if (i + 1 < NS) {
        a -= __uint_as_float(t << 16);
        b -= __uint_as_float(t & 0xFFFF0000u);
      }
    }
  }
#pragma unroll
  for (int i = 0; i < NS; ++i) out[i] = make_uint4(w[i][0], w[i][1], w[i][2], w[i][3]);
}

// One plane of the same split for 32 consecutive values of one row: word j
// holds elements 2j and 2j+1 rounded to BF16; unless this is the last plane,
// x is left holding the residuals for the next one.
template <bool LAST>
__device__ __forceinline__ void split_plane32(float (&x)[32], uint32_t (&w)[16]) {
#pragma unroll
  for (int j = 0; j < 16; ++j) {
    const uint32_t t = bf16x2_rn(x[2 * j], x[2 * j + 1]);
    w[j] = t;
    if (!LAST) {
      // both residuals with one packed FMA: fma(hi, -1, x) rounds the exact
      // x - hi, so the bits are those of the two subtractions
      const float2 h = make_float2(__uint_as_float(t << 16), __uint_as_float(t & 0xFFFF0000u));
      const float2 r =
          __ffma2_rn(h, make_float2(-1.0f, -1.0f), make_float2(x[2 * j], x[2 * j + 1]));
      x[2 * j] = r.x;
      x[2 * j + 1] = r.y;
    }
  }
}

// x = the 32 values of y from E on.
template <int E>
__device__ __forceinline__ void shifted32(const float (&y)[36], float (&x)[32]) {
#pragma unroll
  for (int k = 0; k < 32; ++k) x[k] = y[k + E];
}

// ------------------------------------------------------- FP16X3 split
// FP16 keeps 11 significant bits but only 5 exponent bits, so each FP32 row
// block of A (and each column of B) is first scaled by a power of two 2^S
// that brings its largest magnitude into [2^14, 2^15): then x*2^S = hi + lo
// with hi = fp16(x*2^S) and lo = fp16(x*2^S - hi) keeps 22 significant bits
// of every element within 2^-17 of the largest (the scaling is exact), and
// hi*hi + hi*lo + lo*hi (3 products) carries FP32-level information.  The
// biased exponent of the scale is clamped to [1, 253] so that both 2^S and
// 2^-S are normal floats; an all-zero or denormal block gets 2^126.
__device__ __forceinline__ int fh_scale_biased(float maxabs) {
  const int e = __float_as_int(maxabs) >> 23;  // biased exponent (maxabs >= 0)
  return min(max(268 - e, 1), 253);            // 127 + (14 - (e - 127))
}

// Two FP32 values rounded to FP16 (nearest even), packed: lo in the low half.
__device__ __forceinline__ uint32_t f16x2_rn(float lo, float hi) {
  uint32_t r;
  asm("cvt.rn.f16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(hi), "f"(lo));
  return r;
}

__device__ __forceinline__ float2 f16x2_to_f32(uint32_t h) {
  return __half22float2(*reinterpret_cast<const __half2 *>(&h));
}

// The hi and lo FP16 planes of 32 scaled values of one row: word j holds
// elements 2j and 2j+1; hi = fp16(v), lo = fp16(v - hi) with v = x * s, the
// residual exact in FP32 (hi is converted back to FP32 to form it).
__device__ __forceinline__ void split_fh32(const float (&x)[32], float s, uint32_t (&wh)[16],
                                           uint32_t (&wl)[16]) {
#pragma unroll
  for (int j = 0; j < 16; ++j) {
    const float a = __fmul_rn(x[2 * j], s), b = __fmul_rn(x[2 * j + 1], s);
    const uint32_t h = f16x2_rn(a, b);
    const float2 hf = f16x2_to_f32(h);
    wh[j] = h;
    wl[j] = f16x2_rn(__fsub_rn(a, hf.x), __fsub_rn(b, hf.y));
  }
}

// Largest magnitude of 32 values (a tree of maxima of absolute values).
__device__ __forceinline__ float maxabs32(const float (&x)[32]) {
  float m[16];
#pragma unroll
  for (int j = 0; j < 16; ++j) m[j] = fmaxf(fabsf(x[2 * j]), fabsf(x[2 * j + 1]));
#pragma unroll
  for (int w = 8; w >= 1; w >>= 1)
#pragma unroll
    for (int j = 0; j < w; ++j) m[j] = fmaxf(m[j], m[j + w]);
  return m[0];
}

// 2^e as a float for e in [-149, 127] (denormal below -126), 0 below.
[[maybe_unused]] __device__ __forceinline__ float exp2_int(int e) {
  if (e >= -126) return __int_as_float((min(e, 127) + 127) << 23);
  if (e >= -149) return __int_as_float(1 << (e + 149));
  return 0.0f;
}

// x * 2^e for an integer e, exact unless the result leaves the float range.
__device__ __forceinline__ float scale_pow2(float x, int e) {
  while (e > 126) { x *= 0x1p126f; e -= 126; }
  while (e < -126) { x *= 0x1p-126f; e += 126; }
  return x * __int_as_float((e + 127) << 23);
}

struct TcArgs {
  GemmProblem p;
  int split;       // CTAs per cluster along K
  int kc;          // K extent per split (multiple of kChunkK)
  int sa, so;      // A ring and operand-stage depths
  int n_pad;       // rows of one B plane in the workspace
  int e[4];        // unaligned A: floats before the data in class r's boxes
  // persistent form: `whole` tiles run whole, tile t by CTA t % gridDim.x, then
  // `tail` tiles split in K over `tsplit` CTAs each (K ranges of tkc)
  int64_t whole;
  int tail, tsplit, tkc;
  float *partial;      // [tail * tsplit][BN][kBM], a CTA's K range of its tail tile
  unsigned *arrivals;  // [tail], zero between launches
  int *err;
  const int *bexp;  // FP16X3: per column of B, the scale exponent S_n of its planes
};

// ------------------------------------------------------------ B planes
// planes[p][n][k] (k contiguous, zero padded to n_pad x k_pad): NS BF16
// planes, or for NS = 4 two 32-bit TF32 planes, hi = TF32(x) and
// lo = TF32(x - hi).
template <int NS>
__global__ void split_b_kernel(const float *B, int64_t sbk, int64_t sbn, int K, int N,
                               void *planes_out, int k_pad, int n_pad, float scale) {
  // the tensor-core kernel that reads the planes is launched as a
  // programmatic dependent: its set-up and A loads overlap this kernel
  allow_dependent_launch();
  using Index = std::conditional_t<NS <= 2, uint64_t, uint32_t>;
  const SplitWalk<Index> walk(sbk, sbn, n_pad, k_pad);
  for (Index c = blockIdx.x * blockDim.x + threadIdx.x; c < walk.chunks;
       c += gridDim.x * blockDim.x) {
    int n, k0;
    walk.at(c, &n, &k0);
    float x[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const int k = k0 + j;
      x[j] = (n < N && k < K)
                 ? scale * B[static_cast<int64_t>(k) * sbk + static_cast<int64_t>(n) * sbn]
                 : 0.0f;
    }
    if constexpr (NS == 4) {
      uint32_t *planes = static_cast<uint32_t *>(planes_out);
      uint32_t h[8], l[8];
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        h[j] = tf32_rna(x[j]);
        l[j] = tf32_rna(x[j] - __uint_as_float(h[j]));
      }
      uint32_t *ph = planes + static_cast<int64_t>(n) * k_pad + k0;
      uint32_t *pl = planes + (static_cast<int64_t>(n_pad) + n) * k_pad + k0;
      reinterpret_cast<uint4 *>(ph)[0] = make_uint4(h[0], h[1], h[2], h[3]);
      reinterpret_cast<uint4 *>(ph)[1] = make_uint4(h[4], h[5], h[6], h[7]);
      reinterpret_cast<uint4 *>(pl)[0] = make_uint4(l[0], l[1], l[2], l[3]);
      reinterpret_cast<uint4 *>(pl)[1] = make_uint4(l[4], l[5], l[6], l[7]);
    } else {
      __nv_bfloat16 *planes = static_cast<__nv_bfloat16 *>(planes_out);
      uint4 v[NS];
      pack8<NS>(x, v);
#pragma unroll
      for (int i = 0; i < NS; ++i)
        *reinterpret_cast<uint4 *>(planes + (static_cast<int64_t>(i) * n_pad + n) * k_pad + k0) =
            v[i];
    }
  }
}

// FP16X3 planes of B: column n is scaled by 2^S_n, which brings its largest
// magnitude over K into [2^14, 2^15), and split into planes[0][n][k] =
// fp16(b * 2^S_n) and planes[1][n][k] = fp16(b * 2^S_n - hi); S_n goes to
// bexp[n].  Padding columns (n >= N) get zero planes and kNoColumn.  One
// warp per column: the column's maximum, then its conversion, 8 values a
// lane at a time (16-byte stores).
constexpr int kNoColumn = -100000;

__global__ void split_b_fh_kernel(const float *B, int64_t sbk, int64_t sbn, int K, int N,
                                  uint32_t *planes, int *bexp, int k_pad, int n_pad) {
  allow_dependent_launch();
  const int wpb = blockDim.x >> 5, lane = threadIdx.x & 31;
  for (int n = blockIdx.x * wpb + (threadIdx.x >> 5); n < n_pad; n += gridDim.x * wpb) {
    const float *col = B + static_cast<int64_t>(n) * sbn;
    float mx = 0.0f;
    if (n < N)
      for (int k = lane; k < K; k += 32) mx = fmaxf(mx, fabsf(col[static_cast<int64_t>(k) * sbk]));
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    const int sb = fh_scale_biased(mx);
    const float sc = __int_as_float(sb << 23);
    if (lane == 0) bexp[n] = n < N ? sb - 127 : kNoColumn;
    // planes as 32-bit words: two FP16 per word, k_pad / 2 words per row
    uint32_t *ph = planes + static_cast<int64_t>(n) * (k_pad / 2);
    uint32_t *pl = planes + (static_cast<int64_t>(n_pad) + n) * (k_pad / 2);
    for (int k0 = lane * 8; k0 < k_pad; k0 += 256) {
      float x[8];
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const int k = k0 + j;
        x[j] = (n < N && k < K) ? col[static_cast<int64_t>(k) * sbk] : 0.0f;
      }
      uint32_t h[4], l[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float a = x[2 * j] * sc, b = x[2 * j + 1] * sc;
        h[j] = f16x2_rn(a, b);
        const float2 hf = f16x2_to_f32(h[j]);  // hi exactly as stored
        l[j] = f16x2_rn(a - hf.x, b - hf.y);
      }
      *reinterpret_cast<uint4 *>(ph + k0 / 2) = make_uint4(h[0], h[1], h[2], h[3]);
      *reinterpret_cast<uint4 *>(pl + k0 / 2) = make_uint4(l[0], l[1], l[2], l[3]);
    }
  }
}

// ------------------------------------------------------------- kernel
// Shared-memory plan of one CTA (tiles 1024-byte aligned):
//   A ring    sa slots of the FP32 A tile (16 KB), filled by TMA, released
//             by the converter group that read it;
//   B ring    so slots, each the NS B-plane tiles of one K block (TMA).
// TMEM: NI accumulators of BN columns, then so A stages of NS x 16 columns.
// Operand stage o = B slot o + A stage o, released together by one commit.
// sa is a multiple of G and so a multiple of 2 * NI, so each slot is only
// ever used by one converter group and each stage by one MMA issuer: a
// waiter has always seen the previous phase of its barrier complete.
struct TcPlan {
  int sa, so;
};

// Bytes of the A ring's slots, and of what lands in one: 16 KB, 18 KB for the
// wider boxes of an unaligned A (132 x 8 boxes leave 1.5 KB of it unused).
__host__ __device__ constexpr size_t tc_a_bytes(int am = kAM) {
  return am_unaligned(am) ? 4 * 36 * 32 * 4 : static_cast<size_t>(kBM) * kBK * 4;
}
__host__ __device__ constexpr int tc_a_tx(int am) {
  return am == kAMU ? 4 * 132 * 8 * 4 : static_cast<int>(tc_a_bytes(am));
}
__host__ __device__ constexpr size_t tc_b_bytes(int bn, int ns) {
  return static_cast<size_t>(tc_geom(ns)) * bn * kBK * 2;
}
// FP16X3: the ring of per-row scale exponents the converters hand to the
// drain warps, one entry per K block in flight (2 x the operand stages).
__host__ __device__ constexpr int tc_fh_ring(int so) { return 2 * so; }
// Scratch of the persistent form's drain warps (a row each of plain sums).
constexpr size_t kPersistScratch = 8 * 64 * 4 + 16;
size_t tc_plan_bytes(int bn, int ns, const TcPlan &pl, int am = kAM) {
  const size_t ring = ns == 5 ? static_cast<size_t>(tc_fh_ring(pl.so)) * (8 + kBM * 4) : 0;
  return 1024 + pl.sa * tc_a_bytes(am) + pl.so * tc_b_bytes(bn, ns) +
         8 * (2 * pl.sa + 2 * pl.so + 2 * 4 + 1) + 16 + ring + 16 +
         (am_unaligned(am) ? kPersistScratch : 0);
}

// The deepest operand-stage ring that fits TMEM and shared memory next to
// sa A slots; sa must be a multiple of G.
bool tc_plan(int bn, int ns, int sa, TcPlan *out, int am = kAM) {
  const int g = tc_groups();
  if (sa < g || sa % g != 0) return false;
  const int mult = tc_stage_mult(tc_issuers(bn, ns));
  for (int so = tc_max_stages(bn, ns); so >= mult; so -= mult) {
    const TcPlan pl = {sa, so};
    if (tc_plan_bytes(bn, ns, pl, am) <= 227 * 1024) {
      *out = pl;
      return true;
    }
  }
  return false;
}

__host__ __device__ constexpr uint32_t tc_pow2_cols(int cols) {
  return cols <= 32 ? 32 : cols <= 64 ? 64 : cols <= 128 ? 128 : cols <= 256 ? 256 : 512;
}
__host__ __device__ constexpr uint32_t tc_tmem_alloc_cols(int bn, int ns, int so) {
  return tc_pow2_cols(tc_issuers(bn, ns) * bn + so * tc_stage_cols(ns));
}

// n <= CN elements v of C from cp on, `step` apart: alpha * v + beta * C.
// beta's case is taken once and the address only stepped: with both formed
// for every element a tile's stores held up the accumulators (65536 x 64 x
// 128 34.9 us, 17.3 like this; x 128 x 4096 368 -> 353).
template <int CN>
__device__ __forceinline__ void store_run(float *cp, int64_t step, int n, const float (&v)[CN],
                                          float alpha, float beta) {
  if (beta == 0.0f) {
#pragma unroll
    for (int i = 0; i < CN; ++i, cp += step)
      if (i < n) *cp = axpby(alpha, v[i], 0.0f, cp);
  } else {
#pragma unroll
    for (int i = 0; i < CN; ++i, cp += step)
      if (i < n) *cp = axpby(alpha, v[i], beta, cp);
  }
}

// PERSIST: one CTA per SM walks several tiles ("segments" of its work), the
// loads, conversions and MMAs of the next running on while the drain warps
// finish a tile, so a tile's set-up, first loads and drain (9 to 12 us a tile
// otherwise, of about 60 at K = 4096) are paid once.  Consecutive CTAs take
// consecutive tiles, all at about the same K, so they share operands in L2.
// Which problems run so, and what it measured: tc_walk.
template <int BN, int NS, int AM, bool PERSIST, bool EARLY>
__global__ void __launch_bounds__(tc_warps(BN, NS) * 32, 1)
    tc_kernel(const __grid_constant__ AMaps<AM> tmA, const __grid_constant__ CUtensorMap tmB,
              TcArgs args) {
  constexpr bool AK = am_kcontig(AM), AU = am_unaligned(AM);
  // NS = 4 is the TF32 form: 2 planes of 32-bit TF32 (hi, lo), the TMEM and
  // shared-memory footprint of 4 BF16 planes
  constexpr bool TF = NS == 4;
  // NS = 5 is the FP16X3 form: 2 FP16 planes of scaled values (the footprint
  // of 2 BF16 planes), a power-of-two scale per row and 32-deep block of A
  // and per column of B, each block accumulated and drained on its own
  constexpr bool FH = NS == 5;
  constexpr int PL = TF ? 2 : tc_geom(NS);                   // planes
  constexpr int PLC = TF ? kBK : kBK / 2;                    // TMEM columns of a plane
  constexpr int KMMA = TF ? 8 : 16;                          // K of one MMA
  constexpr int G = tc_groups();
  constexpr int D = tc_drain_groups(BN);
  constexpr int DC = BN / D;                                 // columns per drain thread
  constexpr int NI = tc_issuers(BN, NS);                     // MMA issuers = accumulators
  constexpr int kThreads = tc_warps(BN, NS) * 32;
  constexpr int kConvWarp0 = tc_conv_warp0(BN, NS), kDrainWarp0 = kConvWarp0 + 4 * G;
  constexpr int A32_BYTES = static_cast<int>(tc_a_bytes(AM));  // FP32 A slot
  constexpr int BPL_BYTES = BN * kBK * (TF ? 4 : 2);         // one B plane tile
  constexpr int BSLOT = PL * BPL_BYTES;                      // one B slot
  constexpr int SC = tc_stage_cols(NS);                      // TMEM columns of an A stage
  static_assert(SC == PL * PLC, "stage columns");
  constexpr uint32_t IDESC =
      TF ? idesc_tf32(BN) : FH ? idesc_f16(BN) : idesc_bf16(BN);
  // blocks per TMEM chunk (FP16X3: one, the row scales change every block)
  constexpr int P = FH ? 1 : kChunkK / kBK;

  extern __shared__ uint8_t smem_raw[];
  uint8_t *smem = align_shared(smem_raw, 1024);
  const GemmProblem &p = args.p;
  const int SA = args.sa, SO = args.so;
  uint8_t *aring = smem;
  uint8_t *bring = aring + SA * A32_BYTES;
  uint64_t *afull = reinterpret_cast<uint64_t *>(bring + SO * BSLOT);  // [SA] tile landed
  uint64_t *aempty = afull + SA;     // [SA] the converter group has read the tile
  uint64_t *opfull = aempty + SA;    // [SO] B tiles landed and the A stage written
  uint64_t *opempty = opfull + SO;   // [SO] the MMAs reading the stage are done
  uint64_t *accfull = opempty + SO;   // [NI] accumulator holds a finished chunk
  uint64_t *accempty = accfull + NI;  // [NI] accumulator drained
  uint64_t *mmadone = accempty + NI;  // every issued MMA has completed
  // FP16X3: ring of R entries, one per K block in flight, each the 128 row
  // scale exponents of a block (sexp) and the barrier the converters arrive
  // on once they are written (sfull)
  const int R = FH ? tc_fh_ring(SO) : 0;
  uint64_t *sfull = mmadone + 1;      // [R]
  uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(sfull + R);
  int *bad_flag = reinterpret_cast<int *>(tmem_slot + 1);
  int *tmax_sh = bad_flag + 1;        // FP16X3: the largest column scale exponent of the tile
  int *sexp = align_shared(tmax_sh + 1, 16);  // [R][kBM]
  // PERSIST: whether the CTA arrived last at a tail tile; the drain warps' rows
  [[maybe_unused]] int *last_flag = tmax_sh;
  [[maybe_unused]] float *scratch = reinterpret_cast<float *>(sexp);

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int split = args.split;
  const int rank = split > 1 ? static_cast<int>(cluster_ctarank()) : 0;
  const int64_t m0 = static_cast<int64_t>(blockIdx.x / split) * kBM;
  const int n0 = blockIdx.y * BN;
  const int kbeg = rank * args.kc;
  const int kend = min(p.K, kbeg + args.kc);
  const int nkb = kend > kbeg ? (kend - kbeg + kBK - 1) / kBK : 0;
  const uint32_t tmem_cols = tc_tmem_alloc_cols(BN, NS, SO);

  // The CTA's segments: a tile (first row and column) and a K range in nkb
  // blocks.  Roles count blocks across segments: with PERSIST a segment has
  // whole chunks (the last may hold a block of zeros).
  struct Segment {
    int64_t m0;
    int n0, kbeg, kend, nkb;
    int tile, rank;  // the tail: the tile's index in it (else -1), the K range's
  };
  const bool has_tail =
      PERSIST && static_cast<int64_t>(blockIdx.x) < static_cast<int64_t>(args.tail) * args.tsplit;
  auto segment = [&](int i, Segment *sg) -> bool {
    if constexpr (!PERSIST) {
      *sg = {m0, n0, kbeg, kend, nkb, -1, 0};
      return i == 0;
    } else {
      int64_t t = blockIdx.x + static_cast<int64_t>(i) * gridDim.x;
      *sg = {0, 0, 0, p.K, 0, -1, 0};
      if (t >= args.whole) {
        if (!has_tail || t - blockIdx.x != args.whole) return false;  // (whole waves before it)
        sg->tile = static_cast<int>(blockIdx.x) / args.tsplit;
        sg->rank = static_cast<int>(blockIdx.x) % args.tsplit;
        t = args.whole + sg->tile;
        sg->kbeg = sg->rank * args.tkc;
        sg->kend = min(p.K, sg->kbeg + args.tkc);
      }
      // (a 32-bit division: C's tiles are far fewer than 2^31)
      const unsigned tiles_m = (static_cast<unsigned>(p.M) + kBM - 1) / kBM;
      const unsigned tu = static_cast<unsigned>(t);
      sg->m0 = static_cast<int64_t>(tu % tiles_m) * kBM;
      sg->n0 = static_cast<int>(tu / tiles_m) * BN;
      sg->nkb = sg->kend > sg->kbeg ? (sg->kend - sg->kbeg + P * kBK - 1) / (P * kBK) * P : 0;
      return true;
    }
  };
  Segment sg;

  if (tid == 0) {
    for (int s = 0; s < SA; ++s) {
      mbar_init(&afull[s], 1);
      mbar_init(&aempty[s], 4);
    }
    for (int o = 0; o < SO; ++o) {
      mbar_init(&opfull[o], 4 + 1);  // the converter group's warps + the B loader
      mbar_init(&opempty[o], 1);
    }
    for (int b = 0; b < NI; ++b) {
      mbar_init(&accfull[b], 1);
      mbar_init(&accempty[b], 4 * D);
    }
    mbar_init(mmadone, NI);  // one commit per MMA issuer
    for (int r = 0; r < R; ++r) mbar_init(&sfull[r], 4);  // the converter group's warps
    *bad_flag = 0;
    fence_mbar_init();
  }
  if (warp == 2) tmem_alloc(tmem_slot, tmem_cols);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;
  const uint32_t tacc = tmem;           // accumulator b: columns b*BN .. +BN-1
  const uint32_t tA = tmem + NI * BN;   // A stage o: columns NI*BN + o*SC .. +SC-1

  if (warp == 0) {
    // -------------------------------------------------------- TMA, A
    if (lane == 0) {
      for (const CUtensorMap &t : tmA.m) prefetch_tmap(&t);
      bool ok = true;
      for (int i = 0, base = 0; ok && segment(i, &sg); ++i, base += sg.nkb) {
        for (int kb = 0; kb < sg.nkb; ++kb) {
          const int s = (base + kb) % SA;
          ok = mbar_wait(&aempty[s], (((base + kb) / SA) & 1) ^ 1, args.err, kDevErrEmptyBarrier);
          if (!ok) {
            *bad_flag = 1;
            break;
          }
          uint8_t *dst = aring + s * A32_BYTES;
          const int k0 = sg.kbeg + kb * kBK;
          mbar_arrive_expect_tx(&afull[s], tc_a_tx(AM));
          if constexpr (AU) {
            // class r: rows (columns) r, r + 4, ... of the block, from a
            // 16-byte boundary; k0 and m0 are multiples of 32
#pragma unroll
            for (int r = 0; r < 4; ++r)
              if (AK)
                tma_load_2d(dst + r * (36 * 32 * 4), &tmA.m[r], &afull[s], k0,
                            static_cast<int>(sg.m0 / 4));
              else
                tma_load_2d(dst + r * (132 * 8 * 4), &tmA.m[r], &afull[s], static_cast<int>(sg.m0),
                            k0 / 4);
          } else if (AK) {  // 128 rows of 32 floats (128-byte swizzle)
            tma_load_2d(dst, &tmA.m[0], &afull[s], k0, static_cast<int>(sg.m0));
          } else {  // 32 rows (k) of 128 floats (m)
            tma_load_2d(dst, &tmA.m[0], &afull[s], static_cast<int>(sg.m0), k0);
          }
        }
      }
    }
  } else if (warp == 1) {
    // -------------------------------------------------------- TMA, B
    if (lane == 0) {
      prefetch_tmap(&tmB);
      // the B planes come from the kernel launched just before this one,
      // which may still be running (programmatic dependent launch); nothing
      // else this kernel reads depends on it
      wait_prior_grid();
      bool ok = true;
      for (int i = 0, base = 0; ok && segment(i, &sg); ++i, base += sg.nkb) {
        for (int kb = 0; kb < sg.nkb; ++kb) {
          const int o = (base + kb) % SO;
          ok = mbar_wait(&opempty[o], (((base + kb) / SO) & 1) ^ 1, args.err, kDevErrEmptyBarrier);
          if (!ok) {
            *bad_flag = 1;
            break;
          }
          uint8_t *dst = bring + o * BSLOT;
          const int k0 = sg.kbeg + kb * kBK;
          mbar_arrive_expect_tx(&opfull[o], BSLOT);
#pragma unroll
          for (int pl = 0; pl < PL; ++pl)
            tma_load_2d(dst + pl * BPL_BYTES, &tmB, &opfull[o], k0, pl * args.n_pad + sg.n0);
        }
      }
    }
  } else if (warp >= 2 && warp < 2 + NI) {
    // ---------------------------------------------------------- MMA
    // NI issuing threads, one per accumulator: issuer b takes the chunks
    // q = b, b+NI, ...  A commit tracks only the MMAs of the thread that
    // issues it.
    if (lane == 0) {
      const int b = warp - 2;
      const uint32_t dacc = tacc + static_cast<uint32_t>(b * BN);
      bool ok = true;
      // chunk q of a segment is chunk base / P + q of the CTA
      for (int i = 0, base = 0; ok && segment(i, &sg); ++i, base += sg.nkb) {
        for (int q = (b + NI - base / P % NI) % NI; q * P < sg.nkb && ok; q += NI) {
          const bool w = mbar_wait(&accempty[b], (((base / P + q) / NI) & 1) ^ 1, args.err,
                                   kDevErrEmptyBarrier);
          if (!w) {
            ok = false;
            break;
          }
          const int kb1 = min(sg.nkb, (q + 1) * P);
          // the products of block kb whose plane indices sum to t0 .. t1, the
          // smallest (largest sum) first; `fresh` zeroes the accumulator
          auto issue = [&](int kb, int t0, int t1, bool fresh) {
            const int o = (base + kb) % SO;
            const uint32_t astage = tA + static_cast<uint32_t>(o * SC);
            const uint64_t b_desc = sw64_desc(smem_u32(bring + o * BSLOT));
            uint32_t acc = fresh ? 0u : 1u;
#pragma unroll
            for (int t = PL - 1; t >= 0; --t) {
              if (t < t0 || t > t1) continue;
#pragma unroll
              for (int kk = 0; kk < kBK / KMMA; ++kk)
#pragma unroll
                for (int i = 0; i <= t; ++i) {
                  mma_bf16_ts(dacc, astage + static_cast<uint32_t>(i * PLC + kk * 8),
                              b_desc + static_cast<uint64_t>(((t - i) * BPL_BYTES + kk * 32) >> 4),
                              IDESC, acc);
                  acc = 1u;
                }
            }
          };
          for (int kb = q * P; kb < kb1; ++kb) {
            const int o = (base + kb) % SO;
            const bool first = kb == q * P;
            const bool w =
                mbar_wait(&opfull[o], ((base + kb) / SO) & 1, args.err, kDevErrFullBarrier);
            if (!w) {
              ok = false;
              break;
            }
            tc_fence_after();
            if constexpr (AU) {
              issue(kb, 1, PL - 1, first);
              continue;
            }
            const uint32_t astage = tA + static_cast<uint32_t>(o * SC);
            const uint64_t b_desc = TF ? sw128_desc(smem_u32(bring + o * BSLOT))
                                       : sw64_desc(smem_u32(bring + o * BSLOT));
#pragma unroll
            for (int kk = 0; kk < kBK / KMMA; ++kk) {
#pragma unroll
              for (int i = 0; i < PL; ++i)
#pragma unroll
                for (int j = 0; j < PL - i; ++j) {
                  // A plane i: PLC columns per plane, 8 per MMA step (16 BF16
                  // or 8 TF32 deep); B: 32 bytes per step; descriptor start
                  // addresses count 16-byte units
                  const uint32_t at = astage + static_cast<uint32_t>(i * PLC + kk * 8);
                  const uint64_t bd =
                      b_desc + static_cast<uint64_t>((j * BPL_BYTES + kk * 32) >> 4);
                  const uint32_t acc = (!first || kk > 0 || i > 0 || j > 0) ? 1u : 0u;
                  if constexpr (TF)
                    mma_tf32_ts(dacc, at, bd, IDESC, acc);
                  else
                    mma_bf16_ts(dacc, at, bd, IDESC, acc);
                }
            }
            mma_commit(&opempty[o]);
          }
          if constexpr (AU) {
            // the leading products of the whole chunk last: the tensor core
            // truncates on every accumulation, so only these 4 of a chunk's 24
            // lose bits of the full sum (error against FP64 at K = 1501:
            // 1.2e-7, 5.3e-7 in the order above, 1.8e-7 for the SIMT tiles;
            // the order above releases a stage earlier, 2 % at N = 128)
            for (int kb = q * P; ok && kb < kb1; ++kb) {
              issue(kb, 0, 0, false);
              mma_commit(&opempty[(base + kb) % SO]);
            }
          }
          if (ok) mma_commit(&accfull[b]);
        }
      }
      if (!ok) *bad_flag = 1;
      // tracks every MMA this thread issued
      mma_commit(mmadone);
    }
  } else if (warp >= kConvWarp0 && warp < kDrainWarp0) {
    // ------------------------------------------ converters (G groups)
    const int g = (warp - kConvWarp0) >> 2;
    const int m = tid & (kBM - 1);  // row of the tile == TMEM lane
    const uint32_t lanes = static_cast<uint32_t>((warp & 3) * 32) << 16;
    // kAKU: TMEM lane 32 w + l holds row 4 l + w (class w) of the tile
    [[maybe_unused]] const int e_w = AM == kAKU ? args.e[warp & 3] : 0;
    int blocks = 0;  // of all segments
    for (int i = 0; segment(i, &sg); ++i) blocks += sg.nkb;
    for (int kb = g; kb < blocks; kb += G) {
      const int s = kb % SA, o = kb % SO;
      bool w = mbar_wait(&afull[s], (kb / SA) & 1, args.err, kDevErrFullBarrier);
      if (!__all_sync(0xffffffffu, w)) {
        *bad_flag = 1;
        break;
      }
      const float *a32 = reinterpret_cast<const float *>(aring + s * A32_BYTES);
      float x[32];
      if constexpr (AM == kAKU) {
        // 36 floats of the lane's row (rows 144 bytes apart: 16-byte reads
        // without bank conflicts), the block's 32 from e_w on
        const float *row = a32 + (warp & 3) * (36 * 32) + lane * 36;
        float y[36];
#pragma unroll
        for (int c = 0; c < 9; ++c) {
          const float4 v = *reinterpret_cast<const float4 *>(row + 4 * c);
          y[4 * c + 0] = v.x; y[4 * c + 1] = v.y; y[4 * c + 2] = v.z; y[4 * c + 3] = v.w;
        }
        switch (e_w) {  // uniform over the warp
          case 0: shifted32<0>(y, x); break;
          case 1: shifted32<1>(y, x); break;
          case 2: shifted32<2>(y, x); break;
          default: shifted32<3>(y, x); break;
        }
      } else if constexpr (AM == kAMU) {
#pragma unroll
        for (int k = 0; k < 32; ++k)
          x[k] = a32[(k & 3) * (132 * 8) + (k >> 2) * 132 + m + args.e[k & 3]];
      } else if (AK) {
        // row m holds 32 floats in 128 bytes, 128-byte swizzle
#pragma unroll
        for (int c = 0; c < 8; ++c) {
          const float4 v = *reinterpret_cast<const float4 *>(a32 + m * 32 + ((c ^ (m & 7)) * 4));
          x[4 * c + 0] = v.x; x[4 * c + 1] = v.y; x[4 * c + 2] = v.z; x[4 * c + 3] = v.w;
        }
      } else {
#pragma unroll
        for (int k = 0; k < 32; ++k) x[k] = a32[k * kBM + m];
      }
      if constexpr (AU) {
#pragma unroll
        for (int k = 0; k < 32; k += 2) {
          const float2 t = __fmul2_rn(make_float2(x[k], x[k + 1]), make_float2(kAUScale, kAUScale));
          x[k] = t.x;
          x[k + 1] = t.y;
        }
      }
      uint32_t wv[16];
      [[maybe_unused]] uint32_t wl[16];
      [[maybe_unused]] int sexp_m = 0;
      if constexpr (TF) {
        // hi of the first 16 values
#pragma unroll
        for (int k = 0; k < 16; ++k) wv[k] = tf32_rna(x[k]);
      } else if constexpr (FH) {
        // the row's scale for this block from its largest magnitude, then
        // both planes
        const int sb = fh_scale_biased(maxabs32(x));
        sexp_m = sb - 127;
        split_fh32(x, __int_as_float(sb << 23), wv, wl);
      } else {
        split_plane32<NS == 1>(x, wv);
      }
      if constexpr (EARLY) {
        if constexpr (TF) {
          uint32_t all[16];
#pragma unroll
          for (int k = 0; k < 16; ++k) all[k] = wv[k] | __float_as_uint(x[16 + k]);
          release_early(&aempty[s], all, lane);
        } else {
          release_early(&aempty[s], wv, lane);
        }
      }
      // the A stage: wait until the MMAs that read it are done
      w = mbar_wait(&opempty[o], ((kb / SO) & 1) ^ 1, args.err, kDevErrEmptyBarrier);
      if (!__all_sync(0xffffffffu, w)) {
        *bad_flag = 1;
        break;
      }
      tc_fence_after();
      if constexpr (FH) {
        // the drain of this block reads the row's scale exponent (the entry
        // is free: the drain of block kb - R finished before the MMAs of
        // block kb - SO, which released this operand stage)
        sexp[(kb % R) * kBM + m] = sexp_m;
        __syncwarp();
        if (lane == 0) mbar_arrive(&sfull[kb % R]);
      }
      const uint32_t dst = tA + lanes + static_cast<uint32_t>(o * SC);
      auto release = [&]() {
        if (EARLY) return;
        __syncwarp();
        if (lane == 0) mbar_arrive(&aempty[s]);
      };
      if constexpr (TF) {
        // one TF32 per column: plane hi in columns 0..31 (k), lo in 32..63;
        // lo = TF32(x - hi), the residual being exact in FP32
        tmem_st16(dst, wv);
#pragma unroll
        for (int k = 0; k < 16; ++k) x[k] -= __uint_as_float(wv[k]);
#pragma unroll
        for (int k = 0; k < 16; ++k) wv[k] = tf32_rna(x[16 + k]);
        tmem_st16(dst + 16u, wv);
        release();
#pragma unroll
        for (int k = 0; k < 16; ++k) x[16 + k] -= __uint_as_float(wv[k]);
#pragma unroll
        for (int k = 0; k < 16; ++k) wv[k] = tf32_rna(x[k]);
        tmem_st16(dst + 32u, wv);
#pragma unroll
        for (int k = 0; k < 16; ++k) wv[k] = tf32_rna(x[16 + k]);
        tmem_st16(dst + 48u, wv);
      } else if constexpr (FH) {
        tmem_st16(dst, wv);
        release();
        tmem_st16(dst + 16u, wl);
      } else {
        tmem_st16(dst, wv);
        release();
        split_plane32<NS == 2>(x, wv);
        tmem_st16(dst + 16u, wv);
        if constexpr (NS == 3) {
          split_plane32<true>(x, wv);
          tmem_st16(dst + 32u, wv);
        }
      }
      tmem_wait_st();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&opfull[o]);
    }
  } else if (warp >= kDrainWarp0) {
    // ------------------------------------------ drain (D groups)
    const int d = (warp - kDrainWarp0) >> 2;
    const uint32_t lanes = static_cast<uint32_t>((warp & 3) * 32) << 16;
    const int mrow = tid & (kBM - 1);
    float sums[DC];  // FP32 running sums of row m, DC columns
#pragma unroll
    for (int i = 0; i < DC; ++i) sums[i] = 0.0f;
    [[maybe_unused]] int tmax = kNoColumn;
    if constexpr (FH) {
      // the tile's largest column scale exponent: the running sums hold
      // C(m, n) * 2^(S_n - tmax), never above |C(m, n)| (the column scales
      // come from the B-splitting kernel launched just before this one)
      wait_prior_grid();
      for (int c = lane; c < BN; c += 32)
        if (n0 + c < p.N) tmax = max(tmax, args.bexp[n0 + c]);
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) tmax = max(tmax, __shfl_xor_sync(0xffffffffu, tmax, o));
      if (tid == kDrainWarp0 * 32) *tmax_sh = tmax;
    }
    bool ok = true;
    for (int i = 0, base = 0; segment(i, &sg); ++i, base += sg.nkb) {
      for (int q = 0; ok && q * P < sg.nkb; ++q) {
        const int qc = base / P + q, b = qc % NI;  // chunk of the CTA, its accumulator
        bool w = mbar_wait(&accfull[b], (qc / NI) & 1, args.err, kDevErrMmaBarrier);
        [[maybe_unused]] float mult = 1.0f, mult2 = 1.0f;
        [[maybe_unused]] bool twostep = false;
        if constexpr (FH) {
          // block q's partial of row m is scaled by 2^(S_m,q + S_n): undo the
          // row's scale and the tile's largest column scale, 2^e.  Outside
          // the normal range the factor is applied in two exact steps
          // (2^(e -+ 126), then 2^(+-126)), so no contribution is lost or
          // clamped that FP32 itself would represent.
          if (w) w = mbar_wait(&sfull[q % R], (q / R) & 1, args.err, kDevErrFullBarrier);
          if (w) {
            const int e = -sexp[(q % R) * kBM + mrow] - tmax;
            twostep = e < -126 || e > 127;
            mult = exp2_int(e < -126 ? e + 126 : e > 127 ? e - 126 : e);
            mult2 = e < -126 ? 0x1p-126f : 0x1p126f;
          }
        }
        ok = __all_sync(0xffffffffu, w);  // tcgen05.ld is warp-collective
        if (!ok) {
          *bad_flag = 1;
          break;
        }
        tc_fence_after();
        const uint32_t src = tacc + lanes + static_cast<uint32_t>(b * BN + d * DC);
        if constexpr (FH && DC >= 16) {
          // up to 32 columns loaded before one wait (16 when the running sums
          // take 64 registers); packed FP32x2 FMAs
          constexpr int W = DC >= 64 ? 16 : DC >= 32 ? 32 : DC;
          const float2 m2 = make_float2(mult, mult), m22 = make_float2(mult2, mult2);
#pragma unroll
          for (int c = 0; c < DC; c += W) {
            uint32_t r0[W];
#pragma unroll
            for (int h = 0; h < W; h += 16)
              tmem_ld16(src + c + h, *reinterpret_cast<uint32_t(*)[16]>(r0 + h));
            tmem_wait_ld();
            if (!twostep) {
#pragma unroll
              for (int i = 0; i < W; i += 2) {
                const float2 r = make_float2(__uint_as_float(r0[i]), __uint_as_float(r0[i + 1]));
                const float2 t = __ffma2_rn(r, m2, make_float2(sums[c + i], sums[c + i + 1]));
                sums[c + i] = t.x;
                sums[c + i + 1] = t.y;
              }
            } else {
#pragma unroll
              for (int i = 0; i < W; i += 2) {
                const float2 r = make_float2(__uint_as_float(r0[i]), __uint_as_float(r0[i + 1]));
                const float2 t = __ffma2_rn(__fmul2_rn(r, m2), m22,
                                            make_float2(sums[c + i], sums[c + i + 1]));
                sums[c + i] = t.x;
                sums[c + i + 1] = t.y;
              }
            }
          }
        } else if constexpr (DC >= 16) {
#pragma unroll
          for (int c = 0; c < DC; c += 16) {
            uint32_t r0[16];
            tmem_ld16(src + c, r0);
            tmem_wait_ld();
#pragma unroll
            for (int i = 0; i < 16; ++i) sums[c + i] += __uint_as_float(r0[i]);
          }
        } else {
          static_assert(DC % 8 == 0, "drain width");
          uint32_t r0[8];
          tmem_ld8(src, r0);
          tmem_wait_ld();
          if constexpr (FH) {
            if (!twostep) {
#pragma unroll
              for (int i = 0; i < 8; ++i)
                sums[i] = __fmaf_rn(__uint_as_float(r0[i]), mult, sums[i]);
            } else {
#pragma unroll
              for (int i = 0; i < 8; ++i)
                sums[i] = __fmaf_rn(__fmul_rn(__uint_as_float(r0[i]), mult), mult2, sums[i]);
            }
          } else {
#pragma unroll
            for (int i = 0; i < 8; ++i) sums[i] += __uint_as_float(r0[i]);
          }
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&accempty[b]);
      }
      if constexpr (PERSIST) {
        // ------------------------------------------------ end of a segment
        // (after a wait that expired no tile is stored)
        const int m = AM == kAKU ? 4 * lane + (warp & 3) : mrow;  // row of the tile
        const int64_t gm = sg.m0 + m;
        const int nb = sg.n0 + d * DC;
        if constexpr (AU) {
          // rows with a non-finite sum again in plain FP32 (see below), through
          // the warp's scratch row
          bool odd = false;
#pragma unroll
          for (int c = 0; c < DC; ++c) {
            odd |= !(fabsf(sums[c]) <= FLT_MAX);
            sums[c] *= kAUUnscale;  // (infinities and NaN stay)
          }
          float *row = scratch + (warp - kDrainWarp0) * DC;
          for (unsigned todo = __ballot_sync(0xffffffffu, ok && odd && gm < p.M); todo;
               todo &= todo - 1) {
            const int l = __ffs(todo) - 1;
            const float *arow = p.A + __shfl_sync(0xffffffffu, gm, l) * p.sam;
            for (int n = nb; n < min(p.N, nb + DC); ++n) {
              float v = 0.0f;
              for (int64_t kk = sg.kbeg + lane; kk < sg.kend; kk += 32)
                v = fmaf(arow[kk * p.sak], p.B[kk * p.sbk + n * p.sbn], v);
              v = warp_sum(v);
              if (lane == 0) row[n - nb] = v;
            }
            __syncwarp();
            if (lane == l) {
#pragma unroll
              for (int c = 0; c < DC; ++c)
                if (!(fabsf(sums[c]) <= FLT_MAX) && nb + c < p.N) sums[c] = row[c];
            }
            __syncwarp();
          }
        }
        if (sg.tile >= 0) {
          // a K range of a tail tile, the CTA's last segment: published, and
          // summed at the end
          float *part = args.partial + mrow + (static_cast<int64_t>(blockIdx.x) * BN + d * DC) * kBM;
#pragma unroll
          for (int c = 0; c < DC; ++c) __stcg(part + c * kBM, sums[c]);
          __threadfence();
        } else if (ok && gm < p.M && nb < p.N) {
          store_run<DC>(p.C + gm * p.scm + static_cast<int64_t>(nb) * p.scn, p.scn, p.N - nb, sums,
                        p.alpha, p.beta);
        }
#pragma unroll
        for (int c = 0; c < DC; ++c) sums[c] = 0.0f;
      }
    }
    if constexpr (!PERSIST) {
      // ---------------------------------------------------- epilogue
      // (the running sums stay in this branch's registers; the barrier is the
      // one every other thread reaches below)
      __syncthreads();
      const bool failed = *bad_flag != 0;
      float *red = reinterpret_cast<float *>(smem);  // [BN][kBM], reuses the A ring
      const int m = AM == kAKU ? 4 * lane + (warp & 3) : tid & (kBM - 1);  // row of the tile
      const int64_t gm = m0 + m;
      if (failed) {
#pragma unroll
        for (int i = 0; i < DC; ++i) sums[i] = 0.0f;
      }
      if (split > 1 || AU) {
        if constexpr (AU) {
#pragma unroll
          for (int i = 0; i < DC; ++i) sums[i] *= kAUUnscale;
        }
#pragma unroll
        for (int i = 0; i < DC; ++i) red[(d * DC + i) * kBM + m] = sums[i];
        if constexpr (AU) {
          // an infinite operand (or one that rounds to BF16's infinity) has
          // NaN in its residual planes: non-finite sums are formed again in
          // plain FP32, as the SIMT kernels form them, the lanes of the warp
          // over k
          bool odd = false;
#pragma unroll
          for (int i = 0; i < DC; ++i) odd |= !(fabsf(sums[i]) <= FLT_MAX);
          __syncwarp();
          for (unsigned todo = __ballot_sync(0xffffffffu, odd && gm < p.M); todo;
               todo &= todo - 1) {
            const int mr = __shfl_sync(0xffffffffu, m, __ffs(todo) - 1);
            const float *arow = p.A + (m0 + mr) * p.sam;
            for (int n = n0 + d * DC; n < min(p.N, n0 + (d + 1) * DC); ++n) {
              if (fabsf(red[(n - n0) * kBM + mr]) <= FLT_MAX) continue;
              float v = 0.0f;
              for (int64_t k = kbeg + lane; k < kend; k += 32)
                v = fmaf(arow[k * p.sak], p.B[k * p.sbk + n * p.sbn], v);
              v = warp_sum(v);
              __syncwarp();
              if (lane == 0) red[(n - n0) * kBM + mr] = v;
            }
          }
        }
      } else if (gm < p.M && n0 + d * DC < p.N) {
        const int nb = n0 + d * DC;
        if constexpr (FH) {
#pragma unroll
          for (int i = 0; i < DC; ++i)
            if (nb + i < p.N) sums[i] = scale_pow2(sums[i], tmax - args.bexp[nb + i]);
        }
        store_run<DC>(p.C + gm * p.scm + static_cast<int64_t>(nb) * p.scn, p.scn, p.N - nb, sums,
                      p.alpha, p.beta);
      }
    }
  }
  if constexpr (PERSIST) {
    if (has_tail) {  // (uniform over the CTA)
      // The tail tile: the CTA that arrives last sums its K ranges in rank
      // order, as the cluster does in the other form (no CTA waits for
      // another); all threads, their roles done, 4 rows each.
      const int tile = static_cast<int>(blockIdx.x) / args.tsplit;
      __syncthreads();
      if (tid == 0) {
        __threadfence();
        const bool last =
            atomicAdd(&args.arrivals[tile], 1u) == static_cast<unsigned>(args.tsplit - 1);
        if (last) args.arrivals[tile] = 0u;  // ready for the next call
        *last_flag = last && *bad_flag == 0;
      }
      __syncthreads();
      if (*last_flag) {
        __threadfence();
        const int64_t t = args.whole + tile;  // n_pad == BN: the tile is its row tile
        const float4 *part = reinterpret_cast<const float4 *>(
            args.partial + static_cast<int64_t>(tile) * args.tsplit * BN * kBM);
        for (int e = tid; e < BN * kBM / 4; e += kThreads) {
          float4 sum = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 8
          for (int r = 0; r < args.tsplit; ++r) {
            const float4 v = __ldcg(part + static_cast<int64_t>(r) * (BN * kBM / 4) + e);
            sum.x += v.x; sum.y += v.y; sum.z += v.z; sum.w += v.w;
          }
          const float sv[4] = {sum.x, sum.y, sum.z, sum.w};
          const int n = e * 4 / kBM;
          const int pos = e * 4 % kBM;  // TMEM lane of the first
          const int step = AM == kAKU ? 4 : 1;
          const int64_t gm = t * kBM + (AM == kAKU ? 4 * (pos & 31) + (pos >> 5) : pos);
          if (n < p.N && gm < p.M)
            store_run<4>(p.C + gm * p.scm + static_cast<int64_t>(n) * p.scn, step * p.scm,
                         static_cast<int>((p.M - gm + step - 1) / step), sv, p.alpha, p.beta);
        }
      }
    }
  }
  if (!PERSIST && warp < kDrainWarp0) __syncthreads();
  if (!PERSIST && (split > 1 || AU)) {  // an unaligned A's tile always goes through shared memory
    [[maybe_unused]] int tmax_all = 0;
    if constexpr (FH) {
      wait_prior_grid();  // the column scale exponents below
      tmax_all = *tmax_sh;
    }
    if (split > 1)
      cluster_sync();
    else
      __syncthreads();
    const float *red = reinterpret_cast<const float *>(smem);
    constexpr int E = kBM * BN;
    const int per = E / split;
    const uint32_t base = smem_u32(red);
    for (int e4 = tid * 4; e4 < per; e4 += kThreads * 4) {
      const int e = rank * per + e4;
      float4 sum = make_float4(0.f, 0.f, 0.f, 0.f);
      for (int r = 0; r < split; ++r) {
        const float4 v = ld_dsmem4(mapa_shared(base + e * 4, r));
        sum.x += v.x; sum.y += v.y; sum.z += v.z; sum.w += v.w;
      }
      float sv[4] = {sum.x, sum.y, sum.z, sum.w};
      const int gn = n0 + e / kBM;  // (four rows of one column)
      const int64_t gm = m0 + e % kBM;
      if (gn < p.N && gm < p.M) {
        if constexpr (FH) {
#pragma unroll
          for (int qq = 0; qq < 4; ++qq) sv[qq] = scale_pow2(sv[qq], tmax_all - args.bexp[gn]);
        }
        store_run<4>(p.C + gm * p.scm + static_cast<int64_t>(gn) * p.scn, p.scm,
                     static_cast<int>(min(p.M - gm, static_cast<int64_t>(4))), sv, p.alpha, p.beta);
      }
    }
    if (split > 1) cluster_sync();
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 2) {
    // the TMEM is freed only once every issued MMA has completed
    bool w = true;
    if (lane == 0) w = mbar_wait(mmadone, 0, args.err, kDevErrMmaBarrier);
    __syncwarp();
    (void)w;
    tc_fence_after();
  }
  if (warp == 2) tmem_dealloc(tmem, tmem_cols);
}

}  // namespace

#if HML_TC_PART == 0
bool tc_config_fits(int bn, int ns, int stages) {
  TcPlan pl;
  return tc_plan(bn, ns, stages, &pl);
}
#endif

namespace {

// The persistent form's work: see TcArgs.
struct TcWalk {
  int64_t whole = 0;
  int tail = 0, tsplit = 1;
  float *partial = nullptr;
  unsigned *arrivals = nullptr;
};

// Launch of the kernel with the B planes already split into `planes`.
template <int BN, int NS, int AM, bool PERSIST = false>
hml_status launch_tc_planes(const GemmProblem &p, const hml_sgemm_config &c,
                            const __nv_bfloat16 *planes, int k_pad, int n_pad, int *err,
                            cudaStream_t s, bool automatic, const int *bexp = nullptr,
                            const TcWalk *walk = nullptr) {
  if (NS == 5 && !bexp) return HML_STATUS_INVALID_VALUE;
  AMaps<AM> ta;
  CUtensorMap tb;
  memset(&ta, 0, sizeof ta);
  memset(&tb, 0, sizeof tb);
  TcArgs args = {};
  bool ok = true;
  if constexpr (am_unaligned(AM)) {
    const bool ak = AM == kAKU;
    for (int r = 0; r < 4 && ok; ++r) {
      const LineClass c4 = line_class(p.A, ak ? p.sam : p.sak, ak ? p.M : p.K, ak ? p.K : p.M, r);
      args.e[r] = c4.skip;
      ok = tensor_map_2d(&ta.m[r], CU_TENSOR_MAP_DATA_TYPE_FLOAT32, c4.base, c4.len, c4.lines,
                         c4.stride, ak ? 36 : 132, ak ? 32 : 8, CU_TENSOR_MAP_SWIZZLE_NONE);
    }
  } else if (AM == kAK)
    ok = tensor_map_2d(&ta.m[0], CU_TENSOR_MAP_DATA_TYPE_FLOAT32, p.A, p.K, p.M, p.sam * 4, kBK,
                       kBM, CU_TENSOR_MAP_SWIZZLE_128B);
  else
    ok = tensor_map_2d(&ta.m[0], CU_TENSOR_MAP_DATA_TYPE_FLOAT32, p.A, p.M, p.K, p.sak * 4, kBM,
                       kBK, CU_TENSOR_MAP_SWIZZLE_NONE);
  if (ok) {
    if (NS == 4)  // two TF32 planes: rows of 32 x 4 bytes, 128-byte swizzle
      ok = tensor_map_2d(&tb, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, planes, k_pad,
                         static_cast<uint64_t>(2) * n_pad, static_cast<uint64_t>(k_pad) * 4, kBK,
                         BN, CU_TENSOR_MAP_SWIZZLE_128B);
    else  // 16-bit planes (BF16, or FP16 for NS = 5: TMA only moves the bytes)
      ok = tensor_map_2d(&tb, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, planes, k_pad,
                         static_cast<uint64_t>(tc_geom(NS)) * n_pad,
                         static_cast<uint64_t>(k_pad) * 2, kBK, BN,
                         CU_TENSOR_MAP_SWIZZLE_64B);
  }
  if (!ok) return HML_STATUS_CUDA_ERROR;
  args.p = p;
  args.split = c.split_k;
  const int kchunks = k_pad / kChunkK;
  args.kc = ((kchunks + c.split_k - 1) / c.split_k) * kChunkK;
  TcPlan plan;
  // A ring runs as deep as the configuration says; on the automatic path one of
  // 4 gets 6 where that fits and costs no operand stage (BF16X6, K = 4096, a
  // wave of row tiles, us with 4 and 6 slots: N = 16 74.7, 70.7; 64 76.9, 71.7;
  // 128 96, 97), and the persistent form, which only that path reaches and
  // whose slots are held until the operand stage is free (release_early), has
  // no use for one of 2.
  if (!tc_plan(BN, NS, c.stages, &plan, AM)) return HML_STATUS_INVALID_VALUE;
  if (automatic && (plan.sa == 4 || (PERSIST && plan.sa == 2))) {
    TcPlan deeper;
    for (int sa = 6; sa > plan.sa; sa -= 2)
      if (tc_plan(BN, NS, sa, &deeper, AM) && deeper.so >= plan.so) plan = deeper;
  }
  args.sa = plan.sa;
  args.so = plan.so;
  args.n_pad = n_pad;
  args.err = err;
  args.bexp = bexp;
  const size_t smem = tc_plan_bytes(BN, NS, plan, AM);
  constexpr bool kGrid = !PERSIST && !am_unaligned(AM);
  void (*kern)(AMaps<AM>, CUtensorMap, TcArgs) =
      plan.sa <= 4 ? tc_kernel<BN, NS, AM, PERSIST, kGrid>
                   : tc_kernel<BN, NS, AM, PERSIST, kGrid && BN == 128 && NS <= 3>;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       static_cast<int>(smem));
  if (e == cudaSuccess && c.split_k > 8)
    e = cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
  if (e != cudaSuccess) {
    note_cuda_error(e, "tc attributes");
    return HML_STATUS_CUDA_ERROR;
  }
  const int64_t tiles_m = (static_cast<int64_t>(p.M) + kBM - 1) / kBM;
  const int64_t tiles_n = n_pad / BN;
  if (tiles_m * c.split_k > 0x7fffffff || tiles_n > 65535) return HML_STATUS_NOT_SUPPORTED;
  dim3 grid(static_cast<unsigned>(tiles_m * c.split_k), static_cast<unsigned>(tiles_n));
  if constexpr (PERSIST) {
    args.whole = walk->whole;
    args.tail = walk->tail;
    args.tsplit = walk->tsplit;
    args.tkc = ((kchunks + walk->tsplit - 1) / walk->tsplit) * kChunkK;
    args.partial = walk->partial;
    args.arrivals = walk->arrivals;
    grid = dim3(static_cast<unsigned>(sm_count()));
  }
  // launched right after split_b_kernel wrote the planes: a programmatic
  // dependent whose B loader waits for it (wait_prior_grid)
  e = launch_k_ex(kern, grid, dim3(tc_warps(BN, NS) * 32), smem, s, c.split_k, true,
                  ta, tb, args);
  note_cuda_error(e, "tc launch");
  return cuda_status(e);
}

// How the last, partial wave of `tiles` row tiles on `slots` SMs is run on the
// automatic path: split in K so that its tiles take the idle SMs too, when it
// would leave at least half of them idle (1: as the others).  One CTA per SM:
// M = 65536, N = 32 is 3 full waves of 148 tiles and 68 more.
int tail_split(int64_t tiles, int64_t slots, int k_pad) {
  const int64_t rest = tiles % slots;
  if (tiles < slots || rest == 0 || 2 * rest > slots) return 1;
  int split = 1;
  while (split < 8 && 2 * split * rest <= slots && k_pad / (2 * split) >= 4 * kChunkK) split *= 2;
  return split;
}

// launch_tc_planes for a split_k = 1 configuration whose grid ends in a
// partial wave: the whole waves of row tiles run as configured and the rows
// of a last wave that tail_split splits as a second grid (disjoint rows of C,
// so the results are those of split_k = 2..8 on those rows).
template <int BN, int NS, int AM>
hml_status launch_tc_waves(const GemmProblem &p, const hml_sgemm_config &c,
                           const __nv_bfloat16 *planes, int k_pad, int n_pad, int *err,
                           cudaStream_t s) {
  const int64_t tiles = (static_cast<int64_t>(p.M) + kBM - 1) / kBM;
  const int64_t slots = sm_count();
  const int64_t full = (tiles / slots) * slots;
  const int split = c.split_k == 1 && n_pad == BN ? tail_split(tiles, slots, k_pad) : 1;
  if (split == 1)
    return launch_tc_planes<BN, NS, AM>(p, c, planes, k_pad, n_pad, err, s, true);
  const int64_t m1 = full * kBM;
  GemmProblem head = p, tail = p;
  head.M = static_cast<int>(m1);
  tail.M = p.M - static_cast<int>(m1);
  tail.A = p.A + m1 * p.sam;
  tail.C = p.C + m1 * p.scm;
  hml_sgemm_config ct = c;
  ct.split_k = split;
  hml_status st = launch_tc_planes<BN, NS, AM>(head, c, planes, k_pad, n_pad, err, s, true);
  if (st != HML_STATUS_SUCCESS) return st;
  return launch_tc_planes<BN, NS, AM>(tail, ct, planes, k_pad, n_pad, err, s, true);
}

// The persistent form's work for a split_k = 1 configuration on the automatic
// path; false where the grids above are as fast.  From two whole waves on it
// saves their set-up and drain (B200, grids -> persistent: 40000 x 64 x 200
// 26.3 -> 20.9 us, 37888 x 32 x 512 25.0 -> 21.7, 56832 x 16 x 1000 58.8 ->
// 50.1, 65536 x 128 x 1024 109 -> 96, 65536 x 32 x 4096 216 -> 209), and from
// one wave on when the split tail occupies half of the SMs (28416 x 32 x 1504
// 45.3 -> 43.3; a smaller tail's sum through memory costs what is saved:
// 21001 x 100 x 501 35.4 -> 37.4, 19200 x 128 x 4096 115 -> 112).  Several
// column tiles: over eight shapes from 65536 x 256 to 8192 x 8192, both orders of
// A, the persistent form was 1.1 to 1.3 times as fast at K = 512 (65536 x 256 128
// -> 97 us), 1.0 to 1.1 at 2048, within 4 % either way at 4096 and beyond, except
// 8192^3, where the grids are faster (5.38 ms, 5.85).
bool tc_walk(const GemmProblem &p, const hml_sgemm_config &c, int bn, int k_pad, int n_pad,
             TcWalk *w) {
  const int64_t tiles =
      (static_cast<int64_t>(p.M) + kBM - 1) / kBM * static_cast<int64_t>(n_pad / bn);
  const int64_t slots = sm_count();
  const int64_t full = tiles / slots * slots;
  if (c.split_k != 1 || full == 0 || tiles == slots) return false;
  if (n_pad != bn && p.K > 4096) return false;
  w->whole = tiles;
  const int split = n_pad == bn ? tail_split(tiles, slots, k_pad) : 1;
  if (split > 1) {
    w->whole = full;
    w->tail = static_cast<int>(tiles - full);
    w->tsplit = split;
  }
  return full > slots || 2 * static_cast<int64_t>(w->tail) * split > slots;
}

// The tail's partial sums and counters.  A problem's own need follows M modulo
// the rows of a wave, so that a smaller problem can need more than a larger one
// and would grow a buffer that a graph captured before it uses; the stream's
// first tensor-core call on the automatic path therefore reserves what any
// problem's tail can take (a CTA's tile each: tail * tsplit <= SMs, 9.7 MB on
// 148).  False when that is not to be had, under capture by a stream that did
// not make such a call: the tail then runs as a grid, with the same bits.
bool tail_buffers(cudaStream_t s, TcWalk *w) {
  const size_t sms = static_cast<size_t>(sm_count());
  const size_t bytes = sms * kTcShapes[kNumTcShapes - 1].bn * kBM * sizeof(float);
  const bool held = workspace_held(2, bytes, s);  // and with it the counters
  if (held && w->tail == 0) return true;
  if (!held && stream_capturing(s)) return false;
  void *ws = nullptr;  // (the counters first: slot 2 held means both are)
  if (tile_counters(sms, s, &w->arrivals) != HML_STATUS_SUCCESS ||
      workspace_slot(2, bytes, s, &ws) != HML_STATUS_SUCCESS) {
    cudaGetLastError();
    return false;
  }
  w->partial = static_cast<float *>(ws);
  return true;
}

// B -> BF16 planes in `planes` ([NS][n_pad][k_pad]).
template <int NS>
hml_status split_b(const GemmProblem &p, __nv_bfloat16 *planes, int k_pad, int n_pad,
                   cudaStream_t s, float scale = 1.0f) {
  const int64_t chunks = static_cast<int64_t>(n_pad) * (k_pad / 8);
  const int blocks = static_cast<int>(std::min<int64_t>((chunks + 255) / 256, 4 * sm_count()));
  count_launch();
  split_b_kernel<NS><<<blocks, 256, 0, s>>>(p.B, p.sbk, p.sbn, p.K, p.N, planes, k_pad, n_pad,
                                          scale);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) {
    note_cuda_error(e, "split_b");
    return HML_STATUS_CUDA_ERROR;
  }
  return HML_STATUS_SUCCESS;
}

// B -> the two FP16 planes of the FP16X3 form and the column scale
// exponents (bexp, n_pad ints).
hml_status split_b_fh(const GemmProblem &p, void *planes, int *bexp, int k_pad, int n_pad,
                      cudaStream_t s) {
  const int blocks = std::min(std::max(1, (n_pad + 7) / 8), 4 * sm_count());
  count_launch();
  split_b_fh_kernel<<<blocks, 256, 0, s>>>(p.B, p.sbk, p.sbn, p.K, p.N,
                                           static_cast<uint32_t *>(planes), bexp, k_pad, n_pad);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) {
    note_cuda_error(e, "split_b_fh");
    return HML_STATUS_CUDA_ERROR;
  }
  return HML_STATUS_SUCCESS;
}

template <int BN, int NS, int AM>
hml_status run_tc(const GemmProblem &p, const hml_sgemm_config &c, cudaStream_t s, bool waves) {
  const int k_pad = ((p.K + kChunkK - 1) / kChunkK) * kChunkK;
  const int n_pad = ((p.N + BN - 1) / BN) * BN;
  // B planes in the stream's workspace (FP16X3: then the column exponents)
  const size_t plane_bytes = static_cast<size_t>(n_pad) * k_pad * 2;
  const size_t planes_total = tc_geom(NS) * plane_bytes;
  const size_t extra = NS == 5 ? static_cast<size_t>(n_pad) * sizeof(int) : 0;
  // (an unaligned A has the SIMT tiles, which need none, to fall back on)
  if (am_unaligned(AM) && !workspace_held(0, planes_total + extra, s) && stream_capturing(s))
    return HML_STATUS_ALLOC_FAILED;
  void *ws = nullptr;
  hml_status st = workspace(planes_total + extra, s, &ws);
  if (st != HML_STATUS_SUCCESS) return st;
  TcWalk walk;
  bool persist = false;
  if constexpr (NS <= 3) {
    persist = waves && tc_walk(p, c, BN, k_pad, n_pad, &walk);
    if (waves && !tail_buffers(s, &walk) && walk.tail > 0) persist = false;
  }
  auto *planes = static_cast<__nv_bfloat16 *>(ws);
  if constexpr (NS == 5) {
    // planes_total is a multiple of 128 bytes (k_pad a multiple of 64)
    int *bexp = reinterpret_cast<int *>(static_cast<uint8_t *>(ws) + planes_total);
    st = split_b_fh(p, ws, bexp, k_pad, n_pad, s);
    if (st != HML_STATUS_SUCCESS) return st;
    return launch_tc_planes<BN, NS, AM>(p, c, planes, k_pad, n_pad, device_error_word(), s,
                                        waves, bexp);
  } else {
    st = split_b<NS>(p, planes, k_pad, n_pad, s, am_unaligned(AM) ? kAUScale : 1.0f);
    if (st != HML_STATUS_SUCCESS) return st;
    if constexpr (NS <= 3) {
      if (persist)
        return launch_tc_planes<BN, NS, AM, true>(p, c, planes, k_pad, n_pad,
                                                  device_error_word(), s, true, nullptr, &walk);
    }
    if (waves)
      return launch_tc_waves<BN, NS, AM>(p, c, planes, k_pad, n_pad, device_error_word(), s);
    return launch_tc_planes<BN, NS, AM>(p, c, planes, k_pad, n_pad, device_error_word(), s,
                                        false);
  }
}

template <int BN, int NS>
hml_status run_tc_layout(const GemmProblem &p, const hml_sgemm_config &c, cudaStream_t s,
                         bool waves) {
  return p.a_kcontig() ? run_tc<BN, NS, kAK>(p, c, s, waves)
                       : run_tc<BN, NS, kAM>(p, c, s, waves);
}

template <int NS>
hml_status run_tc_ns(const GemmProblem &p, const hml_sgemm_config &c, cudaStream_t s,
                     bool waves) {
  switch (c.tile_n) {
    case 16: return run_tc_layout<16, NS>(p, c, s, waves);
    case 32: return run_tc_layout<32, NS>(p, c, s, waves);
    case 64: return run_tc_layout<64, NS>(p, c, s, waves);
    case 128: return run_tc_layout<128, NS>(p, c, s, waves);
    default: return HML_STATUS_INVALID_VALUE;
  }
}

bool aligned16(const void *ptr) { return (reinterpret_cast<uintptr_t>(ptr) & 15u) == 0; }

template <int BN>
hml_status run_tc_unaligned(const GemmProblem &p, const hml_sgemm_config &c, cudaStream_t s) {
  return p.a_kcontig() ? run_tc<BN, 3, kAKU>(p, c, s, true) : run_tc<BN, 3, kAMU>(p, c, s, true);
}

// Where the allocation-free entry point keeps B's planes and its error word.
struct NoAllocAddrs {
  void *scratch = nullptr;
  int *err = nullptr;
};

// The launch of run_tc with the B planes in the static array and the static
// error word.
template <int BN, int NS, int AM>
hml_status run_tc_static(const GemmProblem &p, const hml_sgemm_config &c, const NoAllocAddrs &a,
                         cudaStream_t s) {
  const int k_pad = ((p.K + kChunkK - 1) / kChunkK) * kChunkK;
  const int n_pad = ((p.N + BN - 1) / BN) * BN;
  auto *planes = static_cast<__nv_bfloat16 *>(a.scratch);
  hml_status st = split_b<NS>(p, planes, k_pad, n_pad, s);
  if (st != HML_STATUS_SUCCESS) return st;
  return launch_tc_planes<BN, NS, AM>(p, c, planes, k_pad, n_pad, a.err, s, false);
}

template <int NS>
hml_status run_tc_static_ns(const GemmProblem &p, const hml_sgemm_config &c,
                            const NoAllocAddrs &a, cudaStream_t s) {
  const bool ak = p.a_kcontig();
  switch (c.tile_n) {
    case 16: return ak ? run_tc_static<16, NS, kAK>(p, c, a, s)
                       : run_tc_static<16, NS, kAM>(p, c, a, s);
    case 32: return ak ? run_tc_static<32, NS, kAK>(p, c, a, s)
                       : run_tc_static<32, NS, kAM>(p, c, a, s);
    case 64: return ak ? run_tc_static<64, NS, kAK>(p, c, a, s)
                       : run_tc_static<64, NS, kAM>(p, c, a, s);
    case 128: return ak ? run_tc_static<128, NS, kAK>(p, c, a, s)
                        : run_tc_static<128, NS, kAM>(p, c, a, s);
    default: return HML_STATUS_INVALID_VALUE;
  }
}

}  // namespace

#if HML_TC_PART
#define HML_TC_NAME2(name, part) name##part
#define HML_TC_NAME(name, part) HML_TC_NAME2(name, part)
hml_status HML_TC_NAME(run_tc_part, HML_TC_PART)(const GemmProblem &p, const hml_sgemm_config &c,
                                                 cudaStream_t s, bool waves) {
  return run_tc_ns<HML_TC_PART>(p, c, s, waves);
}
#if HML_TC_PART == 2
hml_status run_tc_static_part2(const GemmProblem &p, const hml_sgemm_config &c, void *scratch,
                               int *err, cudaStream_t s) {
  NoAllocAddrs a;
  a.scratch = scratch;
  a.err = err;
  return run_tc_static_ns<2>(p, c, a, s);
}
#endif
}  // namespace hml
#else
hml_status run_tc_part2(const GemmProblem &, const hml_sgemm_config &, cudaStream_t, bool);
hml_status run_tc_part4(const GemmProblem &, const hml_sgemm_config &, cudaStream_t, bool);
hml_status run_tc_part5(const GemmProblem &, const hml_sgemm_config &, cudaStream_t, bool);
hml_status run_tc_static_part2(const GemmProblem &, const hml_sgemm_config &, void *, int *,
                               cudaStream_t);

int tc_num_shapes() { return kNumTcShapes; }
void tc_shape(int v, int *bm, int *bn) {
  *bm = kTcShapes[v].bm;
  *bn = kTcShapes[v].bn;
}

// Planes of a split-precision family, in units of BF16 planes: TF32X3's two
// 32-bit planes take the room of four (its kernels are instantiated NS = 4).
// (FP16X3 is instantiated NS = 5: two 16-bit planes, the room of two BF16 ones)
int tc_ns(int algo) {
  return algo == HML_ALGO_BF16X3   ? 2
         : algo == HML_ALGO_BF16X6 ? 3
         : algo == HML_ALGO_FP16X3 ? 5
                                   : 4;
}

hml_status check_tc(const GemmProblem &p, const hml_sgemm_config &c) {
  if (c.algo != HML_ALGO_BF16X3 && c.algo != HML_ALGO_BF16X6 && c.algo != HML_ALGO_TF32X3 &&
      c.algo != HML_ALGO_FP16X3)
    return HML_STATUS_INVALID_VALUE;
  if (c.variant < 0 || c.variant >= kNumTcShapes) return HML_STATUS_INVALID_VALUE;
  if (c.tile_m != kTcShapes[c.variant].bm || c.tile_n != kTcShapes[c.variant].bn)
    return HML_STATUS_INVALID_VALUE;
  if (c.split_k < 1 || c.split_k > 16 || (c.split_k & (c.split_k - 1)) != 0)
    return HML_STATUS_INVALID_VALUE;
  if (c.stages < 2 || c.stages > 8) return HML_STATUS_INVALID_VALUE;
  if (!tc_config_fits(c.tile_n, tc_ns(c.algo), c.stages)) return HML_STATUS_INVALID_VALUE;
  // the A ring is reused for the split-K partial tile (an unaligned A's ring
  // always holds one: launch_tc_unaligned)
  if (c.split_k > 1 &&
      static_cast<size_t>(kBM) * c.tile_n * 4 > static_cast<size_t>(c.stages) * tc_a_bytes())
    return HML_STATUS_INVALID_VALUE;
  // TMA on A: 16-byte aligned base and row stride
  const int64_t sa = p.a_kcontig() ? p.sam : p.sak;
  if (!aligned16(p.A) || (sa * 4) % 16 != 0) return HML_STATUS_NOT_SUPPORTED;
  if (p.a_kcontig() ? p.sak != 1 : p.sam != 1) return HML_STATUS_NOT_SUPPORTED;
  if (p.M < 1 || p.N < 1 || p.K < 1) return HML_STATUS_NOT_SUPPORTED;
  return HML_STATUS_SUCCESS;
}

hml_status launch_tc(const GemmProblem &p, const hml_sgemm_config &c, cudaStream_t s,
                     bool waves) {
  hml_status st = check_tc(p, c);
  if (st != HML_STATUS_SUCCESS) return st;
  switch (c.algo) {
    case HML_ALGO_BF16X3: return run_tc_part2(p, c, s, waves);
    case HML_ALGO_BF16X6: return run_tc_ns<3>(p, c, s, waves);
    case HML_ALGO_FP16X3: return run_tc_part5(p, c, s, waves);
    default: return run_tc_part4(p, c, s, waves);
  }
}

// The unaligned form (BF16X6): any 4-byte aligned A with unit stride one way,
// M and K at least 4, and a stride TMA can encode (4 lines below 2^40 bytes).
bool tc_unaligned_ok(const GemmProblem &p) {
  const int64_t ld = p.a_kcontig() ? p.sam : p.sak;
  return (p.a_kcontig() ? p.sak == 1 : p.sam == 1) && p.M >= 4 && p.K >= 4 && p.N >= 1 &&
         (reinterpret_cast<uintptr_t>(p.A) & 3u) == 0 && ld >= 1 && ld * 16 < (int64_t(1) << 40);
}

hml_status launch_tc_unaligned(const GemmProblem &p, const hml_sgemm_config &cfg,
                               cudaStream_t s) {
  if (!tc_unaligned_ok(p) || cfg.algo != HML_ALGO_BF16X6) return HML_STATUS_NOT_SUPPORTED;
  hml_sgemm_config c = cfg;
  TcPlan pl;
  // the ring of the aligned form, at least the 64 KB of the widest tile, less
  // what its wider slots leave no room for
  c.stages = std::max(c.stages, 4);
  while (c.stages > 2 && !tc_plan(c.tile_n, 3, c.stages, &pl, kAKU)) c.stages -= 2;
  switch (c.tile_n) {
    case 16: return run_tc_unaligned<16>(p, c, s);
    case 32: return run_tc_unaligned<32>(p, c, s);
    case 64: return run_tc_unaligned<64>(p, c, s);
    case 128: return run_tc_unaligned<128>(p, c, s);
    default: return HML_STATUS_INVALID_VALUE;
  }
}

}  // namespace hml

// ------------------------------------------- batched split-BF16 (persistent)
//
// The batched plan (batched.cu) hands the problems it routes to the tensor
// cores to tc_batch_create.  Each tile width class (BN = 32, 64, 128) gets one
// persistent launch of tc_batch_kernel with one CTA per SM.  The class's
// (problem, 128-row tile, BN-column tile) items sit in device memory longest
// first, and a device-side work queue hands them out: the CTA's TMA-A thread
// takes the next item with an atomic on the class's queue head and publishes
// it to the CTA's other roles through a ring of item slots in shared memory
// (one mbarrier each way per slot), so every SM keeps pulling work until the
// queue is empty.  The pipeline inside a CTA is the single-problem kernel's
// (TMA warps, converter groups, MMA issuers with one TMEM accumulator each,
// drain warps) walking the 64-deep chunks of its items in the order taken;
// the TMA descriptors of every problem sit in device memory.  The last CTA
// to finish resets the queue, so a graph replays the launch as it is.  A
// tile's arithmetic is the single-problem kernel's with split_k = 1, so each
// result equals hml_sgemm_ex_config's for the same tile width, bit for bit,
// whichever CTA took it.
namespace hml {
namespace {

struct TcBatchProblem {
  float *C;
  int64_t scm, scn;
  int M, N;
  float alpha, beta;
  int n_pad;  // rows of one B plane
};

struct alignas(16) TcBatchItem {
  int prob, tm, tn;
  int cpt_akc;  // 2 * (64-deep chunks of K) + (A is K-contiguous): the
                // problem's, beside the tile so that a role that takes the
                // item waits for no further load
  __host__ __device__ int cpt() const { return cpt_akc >> 1; }
  __host__ __device__ bool akc() const { return cpt_akc & 1; }
};

struct TcBatchArgs {
  const CUtensorMap *tmA;       // [problems], 64-byte aligned
  const CUtensorMap *tmB;       // [problems]
  const TcBatchProblem *probs;  // [problems]
  const TcBatchItem *items;     // this class's items, longest first
  int nitems;
  unsigned *queue;              // [2]: queue head, CTAs finished (zero between launches)
  int sa, so;
  int first;                    // the plan's first tile kernel
  int zero;                     // 0 (see settled)
  int *err;
};

// Item slots between the CTA's TMA-A thread (which takes items from the
// queue) and its other roles.  More than the items a CTA can have in flight:
// an item is at least one chunk, and the pipeline holds at most
// sa + so blocks (<= 16) plus NI chunks (<= 4).
constexpr int kItemRing = 32;
constexpr int kNoItem = -1;  // the sentinel published once the queue is empty
// Queue indices a CTA's producer takes before it has loaded the item before
// them.  After an item of 16 chunks or more none: the round trips of the index
// and the record (about 1 us each) hide behind the ring the item leaves full.
// Shorter ones need some ahead, but never more than half a round of the items
// left, or the CTAs that start first take all of a short queue (four ahead
// always: 148 tiles of K = 4096 took 262 us, four after one another on 37 SMs;
// 78 now; 60 uneven problems 862 us, 329 with this order alone).
constexpr int kQueueAhead = 4;
__device__ __forceinline__ int queue_ahead(int cpt, unsigned taken, unsigned nitems) {
  const int want = cpt >= 16 ? 0 : cpt >= 8 ? 2 : kQueueAhead;
  const unsigned left = taken < nitems ? nitems - taken : 0u;
  return min(want, static_cast<int>(left / (2 * gridDim.x)));
}

// A role's walk through the items its CTA takes, in the order taken: item j
// of the sequence is read from ring slot j % kItemRing once published, and
// the slot is released right after the read (every role reads every item:
// the roles count chunks across item boundaries).
//
// The fields a role keeps are taken through an ALU step right where the record
// is read (`zero` is 0, which the compiler does not know).  Without it the
// issuers' code compared an item's chunk count before the load of it had
// returned where the way from one to the other was the loop's back edge alone
// -- at an issuer whose turn the item's only chunk was not -- and took the count
// of the item before: it then waited out its limit for a chunk too many (plans
// of problems of K <= 256, in one launch of 20; the results were right, 2 s
// late).
__device__ __forceinline__ int settled(int v, int zero) {
  asm volatile("xor.b32 %0, %0, %1;" : "+r"(v) : "r"(zero));
  return v;
}

struct QueueCursor {
  TcBatchItem it;
  const TcBatchProblem *pr;
  int j = 0, c = 0;
  bool end = false;
  // Reads item j; false when the wait for it expired.  `warp_role`: every
  // lane of the warp calls this, lane 0 releases the slot for the warp.
  __device__ __forceinline__ bool fetch(const TcBatchArgs &a, uint64_t *ifull, uint64_t *iempty,
                                        const TcBatchItem *ring, bool warp_role, int lane) {
    const int r = j % kItemRing;
    bool w = mbar_wait(&ifull[r], (j / kItemRing) & 1, a.err, kDevErrFullBarrier);
    if (warp_role) w = __all_sync(0xffffffffu, w);
    if (!w) return false;
    const TcBatchItem rec = ring[r];
    it.prob = settled(rec.prob, a.zero);
    it.tm = settled(rec.tm, a.zero);
    it.tn = settled(rec.tn, a.zero);
    it.cpt_akc = settled(rec.cpt_akc, a.zero);
    if (warp_role) {
      __syncwarp();
      if (lane == 0) mbar_arrive(&iempty[r]);
    } else {
      mbar_arrive(&iempty[r]);
    }
    end = it.prob == kNoItem;
    if (!end) pr = a.probs + it.prob;
    c = 0;
    return true;
  }
  // Advances past the current chunk, reading the next item at an item
  // boundary; false when a wait expired.
  __device__ __forceinline__ bool next(const TcBatchArgs &a, uint64_t *ifull, uint64_t *iempty,
                                       const TcBatchItem *ring, bool warp_role, int lane) {
    if (++c < it.cpt()) return true;
    ++j;
    return fetch(a, ifull, iempty, ring, warp_role, lane);
  }
};

// Drain warpgroups of the batched kernel: 32 columns each (its drain also
// finishes C tiles, so it keeps fewer running sums per thread).
__host__ __device__ constexpr int tcb_drain_groups(int bn) { return bn >= 32 ? bn / 32 : 1; }
__host__ __device__ constexpr int tcb_warps(int bn, int ns) {
  return tc_conv_warp0(bn, ns) + 4 * tc_groups() + 4 * tcb_drain_groups(bn);
}

template <int BN, int NS>
__global__ void __launch_bounds__(tcb_warps(BN, NS) * 32, 1) tc_batch_kernel(TcBatchArgs args) {
  // The tile kernels of a plan run at the same time: each is a programmatic
  // dependent of the one before it, and its CTAs take the SMs that one
  // leaves.  The first waits for the B planes (its B loader, the others start
  // on A) and only then lets the second start, so a later kernel finds the
  // planes complete and starts at once; its last CTA out waits for the kernel
  // before it, so the last kernel ends when all have.  (One after another:
  // 12 uneven problems 222 us, 134 like this; 60 problems 282, 265.)
  if (!args.first) allow_dependent_launch();
  constexpr int G = tc_groups();
  constexpr int D = tcb_drain_groups(BN);
  constexpr int DC = BN / D;
  constexpr int NI = tc_issuers(BN, NS);
  constexpr int kConvWarp0 = tc_conv_warp0(BN, NS), kDrainWarp0 = kConvWarp0 + 4 * G;
  constexpr int A32_BYTES = static_cast<int>(tc_a_bytes());
  constexpr int BPL_BYTES = BN * kBK * 2;
  constexpr int BSLOT = NS * BPL_BYTES;
  constexpr int SC = tc_stage_cols(NS);
  constexpr uint32_t IDESC = idesc_bf16(BN);
  constexpr int P = kChunkK / kBK;
  static_assert(G == P, "converter group g converts block g of every chunk");

  extern __shared__ uint8_t smem_raw[];
  uint8_t *smem = align_shared(smem_raw, 1024);
  const int SA = args.sa, SO = args.so;
  uint8_t *aring = smem;
  uint8_t *bring = aring + SA * A32_BYTES;
  uint64_t *afull = reinterpret_cast<uint64_t *>(bring + SO * BSLOT);
  uint64_t *aempty = afull + SA;
  uint64_t *opfull = aempty + SA;
  uint64_t *opempty = opfull + SO;
  uint64_t *accfull = opempty + SO;
  uint64_t *accempty = accfull + NI;
  uint64_t *mmadone = accempty + NI;
  uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(mmadone + 1);
  // item ring: slot published (producer) / slot read by every role
  uint64_t *ifull = reinterpret_cast<uint64_t *>(tmem_slot + 2);
  uint64_t *iempty = ifull + kItemRing;
  TcBatchItem *iring = reinterpret_cast<TcBatchItem *>(iempty + kItemRing);
  // readers of every item: the B loader, NI issuers, the converter and drain warps
  constexpr int kItemReaders = 1 + NI + 4 * G + 4 * D;

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const uint32_t tmem_cols = tc_tmem_alloc_cols(BN, NS, SO);

  if (tid == 0) {
    for (int s = 0; s < SA; ++s) {
      mbar_init(&afull[s], 1);
      mbar_init(&aempty[s], 4);
    }
    for (int o = 0; o < SO; ++o) {
      mbar_init(&opfull[o], 4 + 1);
      mbar_init(&opempty[o], 1);
    }
    for (int b = 0; b < NI; ++b) {
      mbar_init(&accfull[b], 1);
      mbar_init(&accempty[b], 4 * D);
    }
    mbar_init(mmadone, NI);
    for (int r = 0; r < kItemRing; ++r) {
      mbar_init(&ifull[r], 1);
      mbar_init(&iempty[r], kItemReaders);
    }
    fence_mbar_init();
  }
  if (warp == 2) tmem_alloc(tmem_slot, tmem_cols);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;
  const uint32_t tacc = tmem;
  const uint32_t tA = tmem + NI * BN;

  if (warp == 0) {
    // ------------------------------------------- queue + TMA, A
    // takes items from the class's queue, publishes each to the ring, then
    // loads its A blocks; a sentinel ends every role's walk
    if (lane == 0) {
      int blk = 0;
      // q[0 .. w-1]: the indices taken ahead, q[0] the next item's
      unsigned q[kQueueAhead];
#pragma unroll
      for (int i = 0; i < kQueueAhead; ++i) q[i] = 0u;
      q[0] = atomicAdd(&args.queue[0], 1u);
      int w = 1;
      const unsigned nitems = static_cast<unsigned>(args.nitems);
      const TcBatchItem none = {kNoItem, 0, 0, 0};
      TcBatchItem nxt = q[0] < nitems ? args.items[q[0]] : none;
      // the next item's map, acquired before it is used or prefetched
      auto acquire = [&]() {
        if (nxt.prob != kNoItem) acquire_tmap(args.tmA + nxt.prob);
      };
      acquire();
      for (int j = 0;; ++j) {
        const int r = j % kItemRing;
        if (!mbar_wait(&iempty[r], ((j / kItemRing) & 1) ^ 1, args.err, kDevErrEmptyBarrier))
          break;
        const TcBatchItem it = nxt;
        iring[r] = it;
        mbar_arrive(&ifull[r]);  // release: the slot's item is visible to the waiters
        if (it.prob == kNoItem) break;
        // slide the window and fill it up again (past the end: harmless)
        const int depth = queue_ahead(it.cpt(), q[0], nitems);
#pragma unroll
        for (int i = 0; i + 1 < kQueueAhead; ++i) q[i] = q[i + 1];
        --w;
#pragma unroll
        for (int i = 0; i < kQueueAhead; ++i)
          if (i >= w && i < depth) q[i] = atomicAdd(&args.queue[0], 1u);
        w = max(w, depth);
        const bool known = w > 0;
        const CUtensorMap *tm = args.tmA + it.prob;
        const int m0 = it.tm * kBM;
        const int blocks = it.cpt() * P;
        bool ok = true;
        for (int kq = 0; kq < blocks && ok; ++kq, ++blk) {
          const int k0 = kq * kBK;
          const int s = blk % SA;
          if (!mbar_wait(&aempty[s], ((blk / SA) & 1) ^ 1, args.err, kDevErrEmptyBarrier)) {
            ok = false;
            break;
          }
          mbar_arrive_expect_tx(&afull[s], A32_BYTES);
          // k beyond K (the last chunk of a problem) reads TMA's zero fill
          if (it.akc())
            tma_load_2d(aring + s * A32_BYTES, tm, &afull[s], k0, m0);
          else
            tma_load_2d(aring + s * A32_BYTES, tm, &afull[s], m0, k0);
          if (known && kq == 1) {  // (an item has at least two blocks)
            // the next item's record and map, behind the loads just issued
            nxt = q[0] < nitems ? args.items[q[0]] : none;
            acquire();
            if (nxt.prob != kNoItem) prefetch_tmap(args.tmA + nxt.prob);
          }
        }
        if (!ok) break;
        if (!known) {
          q[0] = atomicAdd(&args.queue[0], 1u);
          w = 1;
          nxt = q[0] < nitems ? args.items[q[0]] : none;
          acquire();
        }
      }
      // every atomic taken ahead has returned (its register is read) before
      // this thread's arrival on the finish counter, so the last CTA's reset
      // of the head comes after all of them
#pragma unroll
      for (int i = 0; i < kQueueAhead; ++i) asm volatile("" ::"r"(q[i]));
    }
  } else if (warp == 1) {
    // -------------------------------------------------------- TMA, B
    if (lane == 0) {
      if (args.first) {
        wait_prior_grid();  // the splitting kernel
        allow_dependent_launch();
      }
      QueueCursor cur;
      bool ok = cur.fetch(args, ifull, iempty, iring, false, lane);
      for (int blk = 0; ok && !cur.end;) {
        const CUtensorMap *tm = args.tmB + cur.it.prob;
        if (cur.c == 0) acquire_tmap(tm);
        const int n0 = cur.it.tn * BN;
        const int np = cur.pr->n_pad;
        for (int kb = 0; kb < P; ++kb, ++blk) {
          const int k0 = (cur.c * P + kb) * kBK;
          const int o = blk % SO;
          if (!mbar_wait(&opempty[o], ((blk / SO) & 1) ^ 1, args.err, kDevErrEmptyBarrier)) {
            ok = false;
            break;
          }
          uint8_t *dst = bring + o * BSLOT;
          mbar_arrive_expect_tx(&opfull[o], BSLOT);
#pragma unroll
          for (int i = 0; i < NS; ++i)
            tma_load_2d(dst + i * BPL_BYTES, tm, &opfull[o], k0, i * np + n0);
        }
        if (ok) ok = cur.next(args, ifull, iempty, iring, false, lane);
      }
    }
  } else if (warp >= 2 && warp < 2 + NI) {
    // ---------------------------------------------------------- MMA
    // issuer b takes the chunks q = b, b + NI, ... of the CTA's sequence
    if (lane == 0) {
      const int b = warp - 2;
      const uint32_t dacc = tacc + static_cast<uint32_t>(b * BN);
      QueueCursor cur;
      bool ok = cur.fetch(args, ifull, iempty, iring, false, lane);
      for (int q = 0; ok && !cur.end; ++q) {
        if (q % NI == b) {
          const int jq = q / NI;
          if (!mbar_wait(&accempty[b], (jq & 1) ^ 1, args.err, kDevErrEmptyBarrier)) break;
          for (int kb = 0; kb < P; ++kb) {
            const int blk = q * P + kb;
            const int o = blk % SO;
            if (!mbar_wait(&opfull[o], (blk / SO) & 1, args.err, kDevErrFullBarrier)) {
              ok = false;
              break;
            }
            tc_fence_after();
            const uint32_t astage = tA + static_cast<uint32_t>(o * SC);
            const uint64_t b_desc = sw64_desc(smem_u32(bring + o * BSLOT));
#pragma unroll
            for (int kk = 0; kk < kBK / 16; ++kk) {
#pragma unroll
              for (int i = 0; i < NS; ++i)
#pragma unroll
                for (int jj = 0; jj < NS - i; ++jj) {
                  const uint32_t at = astage + static_cast<uint32_t>(i * 16 + kk * 8);
                  const uint64_t bd =
                      b_desc + static_cast<uint64_t>((jj * BPL_BYTES + kk * 32) >> 4);
                  const uint32_t acc = (kb > 0 || kk > 0 || i > 0 || jj > 0) ? 1u : 0u;
                  mma_bf16_ts(dacc, at, bd, IDESC, acc);
                }
            }
            mma_commit(&opempty[o]);
          }
          if (!ok) break;
          mma_commit(&accfull[b]);
        }
        ok = cur.next(args, ifull, iempty, iring, false, lane);
      }
      mma_commit(mmadone);
    }
  } else if (warp >= kConvWarp0 && warp < kDrainWarp0) {
    // ------------------------------------------ converters (G groups)
    // group g converts block g of every chunk (G == P)
    const int g = (warp - kConvWarp0) >> 2;
    const int m = tid & (kBM - 1);
    const uint32_t lanes = static_cast<uint32_t>((warp & 3) * 32) << 16;
    QueueCursor cur;
    bool ok = cur.fetch(args, ifull, iempty, iring, true, lane);
    for (int q = 0; ok && !cur.end; ++q) {
      const int blk = q * P + g;
      const int s = blk % SA, o = blk % SO;
      bool w = mbar_wait(&afull[s], (blk / SA) & 1, args.err, kDevErrFullBarrier);
      if (!__all_sync(0xffffffffu, w)) break;
      const float *a32 = reinterpret_cast<const float *>(aring + s * A32_BYTES);
      float x[32];
      if (cur.it.akc()) {
        // row m holds 32 floats in 128 bytes, 128-byte swizzle
#pragma unroll
        for (int c = 0; c < 8; ++c) {
          const float4 v = *reinterpret_cast<const float4 *>(a32 + m * 32 + ((c ^ (m & 7)) * 4));
          x[4 * c + 0] = v.x; x[4 * c + 1] = v.y; x[4 * c + 2] = v.z; x[4 * c + 3] = v.w;
        }
      } else {
#pragma unroll
        for (int k = 0; k < 32; ++k) x[k] = a32[k * kBM + m];
      }
      uint32_t wv[16];
      split_plane32<NS == 1>(x, wv);
      w = mbar_wait(&opempty[o], ((blk / SO) & 1) ^ 1, args.err, kDevErrEmptyBarrier);
      if (!__all_sync(0xffffffffu, w)) break;
      tc_fence_after();
      const uint32_t dst = tA + lanes + static_cast<uint32_t>(o * SC);
      tmem_st16(dst, wv);
      __syncwarp();  // every lane's values are in: see release_early
      if (lane == 0) mbar_arrive(&aempty[s]);
      split_plane32<NS == 2>(x, wv);
      tmem_st16(dst + 16u, wv);
      if constexpr (NS == 3) {
        split_plane32<true>(x, wv);
        tmem_st16(dst + 32u, wv);
      }
      tmem_wait_st();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&opfull[o]);
      ok = cur.next(args, ifull, iempty, iring, true, lane);
    }
  } else if (warp >= kDrainWarp0) {
    // ------------------------------------------ drain (D groups)
    const int d = (warp - kDrainWarp0) >> 2;
    const int m = tid & (kBM - 1);
    const uint32_t lanes = static_cast<uint32_t>((warp & 3) * 32) << 16;
    float sums[DC];
#pragma unroll
    for (int i = 0; i < DC; ++i) sums[i] = 0.0f;
    QueueCursor cur;
    bool ok = cur.fetch(args, ifull, iempty, iring, true, lane);
    for (int q = 0; ok && !cur.end; ++q) {
      const int b = q % NI;
      const bool w = mbar_wait(&accfull[b], (q / NI) & 1, args.err, kDevErrMmaBarrier);
      if (!__all_sync(0xffffffffu, w)) break;
      tc_fence_after();
      const uint32_t src = tacc + lanes + static_cast<uint32_t>(b * BN + d * DC);
      if constexpr (DC >= 16) {
#pragma unroll
        for (int c = 0; c < DC; c += 16) {
          uint32_t r0[16];
          tmem_ld16(src + c, r0);
          tmem_wait_ld();
#pragma unroll
          for (int i = 0; i < 16; ++i) sums[c + i] += __uint_as_float(r0[i]);
        }
      } else {
        static_assert(DC % 8 == 0, "drain width");
        uint32_t r0[8];
        tmem_ld8(src, r0);
        tmem_wait_ld();
#pragma unroll
        for (int i = 0; i < 8; ++i) sums[i] += __uint_as_float(r0[i]);
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&accempty[b]);
      if (cur.c == cur.it.cpt() - 1) {
        // the item's last chunk: C tile (row m, columns d*DC ..) and reset
        // (the record by value: read through the pointer it would be loaded
        // again after every store, which cost 128-wide tiles 6 us each: 606208
        // x 128 x 128 319 us, 167 like this; 60 uneven problems 265 -> 257)
        const TcBatchProblem pr = *cur.pr;
        const int64_t gm = static_cast<int64_t>(cur.it.tm) * kBM + m;
        const int nb = cur.it.tn * BN + d * DC;
        if (gm < pr.M && nb < pr.N)
          store_run<DC>(pr.C + gm * pr.scm + static_cast<int64_t>(nb) * pr.scn, pr.scn, pr.N - nb,
                        sums, pr.alpha, pr.beta);
#pragma unroll
        for (int i = 0; i < DC; ++i) sums[i] = 0.0f;
      }
      ok = cur.next(args, ifull, iempty, iring, true, lane);
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 2) {
    bool w = true;
    if (lane == 0) w = mbar_wait(mmadone, 0, args.err, kDevErrMmaBarrier);
    __syncwarp();
    (void)w;
    tc_fence_after();
    tmem_dealloc(tmem, tmem_cols);
  }
  if (tid == 0) {
    // the last CTA out resets the queue for the next launch (every CTA's
    // last atomic on the head came before its own increment here)
    __threadfence();
    if (atomicAdd(&args.queue[1], 1u) == gridDim.x - 1) {
      args.queue[0] = 0u;
      args.queue[1] = 0u;
      __threadfence();
      if (!args.first) wait_prior_grid();
    }
  }
}

// B of every routed problem -> its BF16 planes, one launch: blockIdx.y is the
// problem, the x blocks stride over its (n, 8-deep k) chunks.
struct TcSplitDesc {
  const float *B;
  int64_t sbk, sbn;
  int K, N, k_pad, n_pad;
  __nv_bfloat16 *planes;
};

template <int NS>
__global__ void split_b_batch_kernel(const TcSplitDesc *descs) {
  allow_dependent_launch();  // the tensor-core kernels wait for the planes
  const TcSplitDesc d = descs[blockIdx.y];
  using Index = std::conditional_t<NS <= 2, uint64_t, uint32_t>;
  const SplitWalk<Index> walk(d.sbk, d.sbn, d.n_pad, d.k_pad);
  for (Index c = blockIdx.x * blockDim.x + threadIdx.x; c < walk.chunks;
       c += gridDim.x * blockDim.x) {
    int n, k0;
    walk.at(c, &n, &k0);
    float x[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const int k = k0 + j;
      x[j] = (n < d.N && k < d.K)
                 ? d.B[static_cast<int64_t>(k) * d.sbk + static_cast<int64_t>(n) * d.sbn]
                 : 0.0f;
    }
    uint4 v[NS];
    pack8<NS>(x, v);
#pragma unroll
    for (int i = 0; i < NS; ++i)
      *reinterpret_cast<uint4 *>(d.planes + (static_cast<int64_t>(i) * d.n_pad + n) * d.k_pad +
                                 k0) = v[i];
  }
}

constexpr int kBatchTcNS = 3;                     // BF16X6: FP32-level accuracy
constexpr int kBatchTcBN[] = {32, 64, 128};       // tile width classes

int batch_tc_class(int N) { return N <= 32 ? 0 : N <= 64 ? 1 : 2; }

}  // namespace

// Host side of the batched split-BF16 part of a plan.
struct TcBatch {
  int nprob = 0;
  int items = 0;
  int ctas = 0;                   // the widest class launch
  void *dev = nullptr;            // one device allocation holding everything below
  cudaStream_t owner = nullptr;   // stream of a stream-ordered allocation, if any
  const TcSplitDesc *splits = nullptr;
  int split_blocks = 1;
  struct Class {
    int grid = 0;
    size_t smem = 0;
    TcBatchArgs args = {};
  } cls[3];
};

// Problems the batched plan can run on the tensor cores: A addressable by TMA
// (16-byte aligned base, leading dimension a multiple of 16 bytes), a real
// product (K > 0, alpha != 0) and N > 8 (at N <= 8 the FP32 SIMT tile is
// faster).
bool tc_batch_eligible(const GemmProblem &p) {
  if (p.N <= 8 || p.M < 1 || p.K < 1 || p.alpha == 0.0f) return false;
  const int64_t sa = p.a_kcontig() ? p.sam : p.sak;
  if ((reinterpret_cast<uintptr_t>(p.A) & 15u) != 0 || (sa * 4) % 16 != 0) return false;
  if (p.a_kcontig() ? p.sak != 1 : p.sam != 1) return false;
  return true;
}

namespace {

size_t up256(size_t b) { return (b + 255) & ~static_cast<size_t>(255); }

// Shared memory of the item ring: slots plus their two barriers.
constexpr size_t kItemRingBytes = kItemRing * (sizeof(TcBatchItem) + 2 * sizeof(uint64_t)) + 16;

template <int BN>
hml_status tc_batch_class_setup(TcBatch::Class &c) {
  TcPlan plan;
  int sa = 8;
  while (sa >= 2 && !(tc_plan(BN, kBatchTcNS, sa, &plan) &&
                      tc_plan_bytes(BN, kBatchTcNS, plan) + kItemRingBytes <= 227 * 1024))
    sa -= 2;
  if (sa < 2) return HML_STATUS_NOT_SUPPORTED;
  c.args.sa = plan.sa;
  c.args.so = plan.so;
  c.smem = tc_plan_bytes(BN, kBatchTcNS, plan) + kItemRingBytes;
  const cudaError_t e = cudaFuncSetAttribute(tc_batch_kernel<BN, kBatchTcNS>,
                                             cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             static_cast<int>(c.smem));
  if (e != cudaSuccess) {
    note_cuda_error(e, "tc batch attributes");
    return HML_STATUS_CUDA_ERROR;
  }
  return HML_STATUS_SUCCESS;
}

}  // namespace

hml_status tc_batch_create(const GemmProblem *probs, int count, cudaStream_t stream_ordered,
                           TcBatch **out) {
  *out = nullptr;
  if (count <= 0) return HML_STATUS_SUCCESS;
  if (count > 65535) return HML_STATUS_NOT_SUPPORTED;  // grid.y of the split launch
  const int sms = sm_count();
  // per problem: class, padded sizes, planes
  std::vector<int> cls(count), k_pad(count), n_pad(count);
  std::vector<size_t> plane_off(count);
  size_t planes_bytes = 0;
  std::vector<std::vector<std::pair<int, TcBatchItem>>> items(3);  // (cost, item)
  int64_t max_chunks = 1;
  for (int i = 0; i < count; ++i) {
    const GemmProblem &p = probs[i];
    cls[i] = batch_tc_class(p.N);
    const int bn = kBatchTcBN[cls[i]];
    k_pad[i] = ((p.K + kChunkK - 1) / kChunkK) * kChunkK;
    n_pad[i] = ((p.N + bn - 1) / bn) * bn;
    plane_off[i] = planes_bytes;
    planes_bytes += up256(static_cast<size_t>(kBatchTcNS) * n_pad[i] * k_pad[i] * 2);
    max_chunks = std::max<int64_t>(max_chunks, static_cast<int64_t>(n_pad[i]) * (k_pad[i] / 8));
    const int64_t tm = (static_cast<int64_t>(p.M) + kBM - 1) / kBM, tn = n_pad[i] / bn;
    if (tm > 0x7fffffff) return HML_STATUS_NOT_SUPPORTED;
    for (int64_t x = 0; x < tm; ++x)
      for (int64_t y = 0; y < tn; ++y)
        items[cls[i]].push_back({k_pad[i] / kChunkK,
                                 TcBatchItem{i, static_cast<int>(x), static_cast<int>(y),
                                             k_pad[i] / kChunkK * 2 + (p.a_kcontig() ? 1 : 0)}});
  }
  // per class: the items longest first, the order the queue hands them out
  // (each CTA takes the next when it can: longest-processing-time first)
  std::vector<TcBatchItem> cls_items[3];
  size_t total_items = 0;
  for (int c = 0; c < 3; ++c) {
    auto &v = items[c];
    if (v.empty()) continue;
    if (v.size() > 0x7fffffffu) return HML_STATUS_NOT_SUPPORTED;
    std::stable_sort(v.begin(), v.end(),
                     [](const std::pair<int, TcBatchItem> &a, const std::pair<int, TcBatchItem> &b) {
                       return a.first > b.first;
                     });
    for (const auto &e : v) cls_items[c].push_back(e.second);
    total_items += v.size();
  }
  // device layout: tensor maps | problems | split descriptors | queues |
  // per class items | planes
  const size_t o_tmA = 0, o_tmB = up256(count * sizeof(CUtensorMap));
  const size_t o_prob = o_tmB + up256(count * sizeof(CUtensorMap));
  const size_t o_split = o_prob + up256(count * sizeof(TcBatchProblem));
  const size_t o_queue = o_split + up256(count * sizeof(TcSplitDesc));
  size_t o = o_queue + up256(3 * 2 * sizeof(unsigned));
  size_t o_items[3];
  for (int c = 0; c < 3; ++c) {
    o_items[c] = o;
    o += up256(cls_items[c].size() * sizeof(TcBatchItem));
  }
  const size_t o_planes = o;
  const size_t total = o_planes + planes_bytes;

  TcBatch *b = new (std::nothrow) TcBatch;
  if (!b) return HML_STATUS_ALLOC_FAILED;
  cudaError_t e = stream_ordered ? cudaMallocAsync(&b->dev, total, stream_ordered)
                                 : cudaMalloc(&b->dev, total);
  if (e != cudaSuccess) {
    note_cuda_error(e, "tc batch allocation");
    delete b;
    return HML_STATUS_ALLOC_FAILED;
  }
  b->owner = stream_ordered;
  uint8_t *base = static_cast<uint8_t *>(b->dev);
  // host images
  std::vector<CUtensorMap> tmA(count), tmB(count);
  std::vector<TcBatchProblem> hp(count);
  std::vector<TcSplitDesc> hs(count);
  bool ok = true;
  for (int i = 0; i < count && ok; ++i) {
    const GemmProblem &p = probs[i];
    const int bn = kBatchTcBN[cls[i]];
    auto *planes = reinterpret_cast<__nv_bfloat16 *>(base + o_planes + plane_off[i]);
    memset(&tmA[i], 0, sizeof(CUtensorMap));
    memset(&tmB[i], 0, sizeof(CUtensorMap));
    if (p.a_kcontig())
      ok = tensor_map_2d(&tmA[i], CU_TENSOR_MAP_DATA_TYPE_FLOAT32, p.A, p.K, p.M, p.sam * 4, kBK,
                         kBM, CU_TENSOR_MAP_SWIZZLE_128B);
    else
      ok = tensor_map_2d(&tmA[i], CU_TENSOR_MAP_DATA_TYPE_FLOAT32, p.A, p.M, p.K, p.sak * 4, kBM,
                         kBK, CU_TENSOR_MAP_SWIZZLE_NONE);
    if (ok)
      ok = tensor_map_2d(&tmB[i], CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, planes, k_pad[i],
                         static_cast<uint64_t>(kBatchTcNS) * n_pad[i],
                         static_cast<uint64_t>(k_pad[i]) * 2, kBK, bn, CU_TENSOR_MAP_SWIZZLE_64B);
    TcBatchProblem &q = hp[i];
    memset(&q, 0, sizeof q);
    q.C = p.C;
    q.scm = p.scm;
    q.scn = p.scn;
    q.M = p.M;
    q.N = p.N;
    q.alpha = p.alpha;
    q.beta = p.beta;
    q.n_pad = n_pad[i];
    hs[i] = TcSplitDesc{p.B, p.sbk, p.sbn, p.K, p.N, k_pad[i], n_pad[i], planes};
  }
  auto upload = [&](size_t off, const void *src, size_t bytes) {
    if (e != cudaSuccess || bytes == 0) return;
    e = stream_ordered ? cudaMemcpyAsync(base + off, src, bytes, cudaMemcpyHostToDevice,
                                         stream_ordered)
                       : cudaMemcpy(base + off, src, bytes, cudaMemcpyHostToDevice);
  };
  if (ok) {
    upload(o_tmA, tmA.data(), count * sizeof(CUtensorMap));
    upload(o_tmB, tmB.data(), count * sizeof(CUtensorMap));
    upload(o_prob, hp.data(), count * sizeof(TcBatchProblem));
    upload(o_split, hs.data(), count * sizeof(TcSplitDesc));
    for (int c = 0; c < 3; ++c)
      upload(o_items[c], cls_items[c].data(), cls_items[c].size() * sizeof(TcBatchItem));
    const unsigned zeros[6] = {0u, 0u, 0u, 0u, 0u, 0u};  // queue heads and finished counts
    upload(o_queue, zeros, sizeof zeros);
    // pageable sources: a synchronous copy has consumed them on return; the
    // stream-ordered ones have been staged by the driver before returning
  }
  hml_status st = ok ? cuda_status(e) : HML_STATUS_CUDA_ERROR;
  for (int c = 0; c < 3 && st == HML_STATUS_SUCCESS; ++c) {
    TcBatch::Class &k = b->cls[c];
    k.grid = static_cast<int>(std::min<size_t>(cls_items[c].size(), static_cast<size_t>(sms)));
    if (k.grid == 0) continue;
    st = c == 0   ? tc_batch_class_setup<32>(k)
         : c == 1 ? tc_batch_class_setup<64>(k)
                  : tc_batch_class_setup<128>(k);
    k.args.tmA = reinterpret_cast<const CUtensorMap *>(base + o_tmA);
    k.args.tmB = reinterpret_cast<const CUtensorMap *>(base + o_tmB);
    k.args.probs = reinterpret_cast<const TcBatchProblem *>(base + o_prob);
    k.args.items = reinterpret_cast<const TcBatchItem *>(base + o_items[c]);
    k.args.nitems = static_cast<int>(cls_items[c].size());
    k.args.queue = reinterpret_cast<unsigned *>(base + o_queue) + 2 * c;
    k.args.err = device_error_word();
    b->ctas = std::max(b->ctas, k.grid);
  }
  if (st != HML_STATUS_SUCCESS) {
    if (e != cudaSuccess) note_cuda_error(e, "tc batch upload");
    tc_batch_destroy(b);
    return st;
  }
  for (int c = 2; c >= 0; --c) {  // in launch order
    if (b->cls[c].grid == 0) continue;
    b->cls[c].args.first = 1;
    break;
  }
  b->nprob = count;
  b->items = static_cast<int>(total_items);
  b->splits = reinterpret_cast<const TcSplitDesc *>(base + o_split);
  b->split_blocks = static_cast<int>(std::min<int64_t>((max_chunks + 255) / 256, 64));
  *out = b;
  return HML_STATUS_SUCCESS;
}

hml_status tc_batch_launch(const TcBatch *b, cudaStream_t s) {
  if (!b || b->nprob == 0) return HML_STATUS_SUCCESS;
  count_launch();
  split_b_batch_kernel<kBatchTcNS>
      <<<dim3(static_cast<unsigned>(b->split_blocks), static_cast<unsigned>(b->nprob)), 256, 0,
         s>>>(b->splits);
  cudaError_t e = cudaGetLastError();
  // each tile kernel is a programmatic dependent of the kernel before it (see
  // the kernel's head); the widest class, whose tiles take longest, first
  for (int c = 2; c >= 0 && e == cudaSuccess; --c) {
    const TcBatch::Class &k = b->cls[c];
    if (k.grid == 0) continue;
    if (c == 0)
      e = launch_k_ex(tc_batch_kernel<32, kBatchTcNS>, dim3(k.grid),
                      dim3(tcb_warps(32, kBatchTcNS) * 32), k.smem, s, 1, true, k.args);
    else if (c == 1)
      e = launch_k_ex(tc_batch_kernel<64, kBatchTcNS>, dim3(k.grid),
                      dim3(tcb_warps(64, kBatchTcNS) * 32), k.smem, s, 1, true, k.args);
    else
      e = launch_k_ex(tc_batch_kernel<128, kBatchTcNS>, dim3(k.grid),
                      dim3(tcb_warps(128, kBatchTcNS) * 32), k.smem, s, 1, true, k.args);
  }
  note_cuda_error(e, "tc batch launch");
  return cuda_status(e);
}

void tc_batch_destroy(TcBatch *b) {
  if (!b) return;
  if (b->dev) {
    if (b->owner)
      cudaFreeAsync(b->dev, b->owner);
    else
      cudaFree(b->dev);
  }
  delete b;
}

// The configuration under which a batched plan runs an eligible problem:
// its tile width class and the A-ring depth the class launch uses; the
// single-problem kernel with this configuration computes the same bits.
hml_sgemm_config tc_batch_config(const GemmProblem &p) {
  const int bn = kBatchTcBN[batch_tc_class(p.N)];
  int sa = 8;
  TcPlan plan;
  while (sa > 2 && !tc_plan(bn, kBatchTcNS, sa, &plan)) sa -= 2;
  int var = 0;
  while (var + 1 < kNumTcShapes && kTcShapes[var].bn != bn) ++var;
  return hml_sgemm_config{HML_ALGO_BF16X6, kBM, bn, 1, sa, var};
}

int tc_batch_items(const TcBatch *b) { return b ? b->items : 0; }
int tc_batch_ctas(const TcBatch *b) { return b ? b->ctas : 0; }

}  // namespace hml

// ----------------------------------------------------- no-allocation variant
//
// hml_sgemm_ex_config_noalloc runs the split-BF16 kernel above without any
// device allocation.  Its only scratch, the BF16 planes of B, lives in a
// fixed-size array in this file's module instead of the per-stream workspace
// (which the library grows with cudaMalloc).  The array is part of the
// library's device image, so every GPU that loads the library holds it until
// the process exits.
namespace hml {
namespace {

constexpr size_t kNoAllocScratchBytes = size_t(4) << 20;  // 4 MiB per device
static __device__ __align__(256) unsigned char g_noalloc_scratch[kNoAllocScratchBytes];
// The error word of the bounded waits of calls made through this entry point:
// file scope too, so that no call allocates it.  hml_device_error reads and
// clears it together with the library's other error word.
static __device__ int g_noalloc_error;

constexpr int kNoAllocMaxDevices = 64;
std::mutex g_noalloc_mu;
NoAllocAddrs g_noalloc_addr[kNoAllocMaxDevices];

// Device addresses of the scratch array and the error word on the current
// device.  In host code the arrays' names are only host-side stand-ins, so
// the addresses are looked up once per device (with that device current) and
// cached.
hml_status noalloc_setup(NoAllocAddrs *out) {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) {
    note_cuda_error(e, "noalloc: cudaGetDevice");
    return HML_STATUS_CUDA_ERROR;
  }
  if (dev < 0 || dev >= kNoAllocMaxDevices) return HML_STATUS_NOT_SUPPORTED;
  std::lock_guard<std::mutex> lk(g_noalloc_mu);
  NoAllocAddrs &a = g_noalloc_addr[dev];
  if (!a.scratch) {
    void *scratch = nullptr, *err = nullptr;
    e = cudaGetSymbolAddress(&scratch, g_noalloc_scratch);
    if (e == cudaSuccess) e = cudaGetSymbolAddress(&err, g_noalloc_error);
    if (e != cudaSuccess || !scratch || !err) {
      note_cuda_error(e != cudaSuccess ? e : cudaErrorInvalidSymbol,
                      "noalloc: cudaGetSymbolAddress");
      return HML_STATUS_CUDA_ERROR;
    }
    a.err = static_cast<int *>(err);
    a.scratch = scratch;
  }
  *out = a;
  return HML_STATUS_SUCCESS;
}

size_t noalloc_bytes_needed(const GemmProblem &p, const hml_sgemm_config &c) {
  const int ns = c.algo == HML_ALGO_BF16X3 ? 2 : 3;
  const size_t k_pad = ((static_cast<size_t>(p.K) + kChunkK - 1) / kChunkK) * kChunkK;
  const size_t n_pad = ((static_cast<size_t>(p.N) + c.tile_n - 1) / c.tile_n) * c.tile_n;
  return static_cast<size_t>(ns) * n_pad * k_pad * 2;
}

}  // namespace

// Reads and clears the error word of the allocation-free entry point on the
// current device; 0 when that entry point was never set up there.  Copies to
// and from the symbol allocate nothing.
hml_status noalloc_take_error(int *code) {
  *code = 0;
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) {
    note_cuda_error(e, "noalloc: cudaGetDevice");
    return HML_STATUS_CUDA_ERROR;
  }
  if (dev < 0 || dev >= kNoAllocMaxDevices) return HML_STATUS_SUCCESS;
  {
    std::lock_guard<std::mutex> lk(g_noalloc_mu);
    if (!g_noalloc_addr[dev].err) return HML_STATUS_SUCCESS;
  }
  int h = 0;
  e = cudaMemcpyFromSymbol(&h, g_noalloc_error, sizeof(int));
  if (e == cudaSuccess && h != 0) {
    const int zero = 0;
    e = cudaMemcpyToSymbol(g_noalloc_error, &zero, sizeof(int));
  }
  note_cuda_error(e, "noalloc: error word");
  *code = h;
  return cuda_status(e);
}
}  // namespace hml

extern "C" hml_status hml_sgemm_ex_config_noalloc(hml_order order, hml_op transA, hml_op transB,
                                                  int M, int N, int K, float alpha, const float *A,
                                                  int lda, const float *B, int ldb, float beta,
                                                  float *C, int ldc, const hml_sgemm_config *config,
                                                  void *stream) {
  using namespace hml;
  if (!config || (config->algo != HML_ALGO_BF16X3 && config->algo != HML_ALGO_BF16X6))
    return HML_STATUS_INVALID_VALUE;
  GemmProblem p;
  hml_status st = gemm_from_blas(order, transA, transB, M, N, K, alpha, A, lda, B, ldb, beta, C,
                                 ldc, &p);
  if (st != HML_STATUS_SUCCESS) return st;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  if (p.M == 0 || p.N == 0) return HML_STATUS_SUCCESS;
  if (p.K == 0 || p.alpha == 0.0f) return launch_scale(p.C, p.M, p.N, p.scm, p.scn, p.beta, s);
  st = check_tc(p, *config);
  if (st != HML_STATUS_SUCCESS) return st;
  if (noalloc_bytes_needed(p, *config) > kNoAllocScratchBytes) {
    note_text_error("noalloc: the BF16 planes of B need more than the 4 MiB static scratch "
                    "(planes x ceil(min(M,N)/tile_n)*tile_n x ceil(K/64)*64 x 2 bytes)");
    return HML_STATUS_INVALID_VALUE;
  }
  NoAllocAddrs addrs;
  st = noalloc_setup(&addrs);
  if (st != HML_STATUS_SUCCESS) return st;
  return config->algo == HML_ALGO_BF16X3 ? run_tc_static_part2(p, *config, addrs.scratch, addrs.err, s)
                                         : run_tc_static_ns<3>(p, *config, addrs, s);
}
#endif  // HML_TC_PART
