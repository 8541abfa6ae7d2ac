// select.cu -- which configuration hml_sgemm_ex runs.
//
// Order of precedence (replacing the reference's static table lookup
// cfg[min(K,96)][ceil(min(N,96)/16)], src/hml_sgemm_kernel.cu:189-237):
//   1. the measured table of the autotuner (exact shape class, else the
//      nearest measured class in log space), when one is loaded;
//   2. the learned predictor, when one is loaded;
//   3. the heuristic below.
#include <algorithm>
#include <cmath>

#include "hml_select.h"
#include "hml_tune.h"

namespace hml {

int simt_num_shapes();
void simt_shape(int v, int *bm, int *bn, int *wk);
int simt_ctas_per_sm(int v);
int tc_num_shapes();
void tc_shape(int v, int *bm, int *bn);
bool tc_config_fits(int bn, int ns, int stages);
int tc_ns(int algo);
bool cfg_v1_sgemm_rule(int K, int N, int *type, int *row_stops);

namespace {

int pow2_at_least(int64_t x, int cap) {
  int s = 1;
  while (s < cap && s < x) s <<= 1;
  return s;
}

// pick split_k so the grid covers the machine about `waves` times while each
// CTA keeps at least `min_k` of K
int choose_split(int64_t tiles, int K, int ctas_per_sm, int min_k) {
  const int64_t want = static_cast<int64_t>(sm_count()) * ctas_per_sm;
  int split = tiles >= want ? 1 : pow2_at_least((want + tiles - 1) / tiles, 16);
  while (split > 1 && K / split < min_k) split >>= 1;
  return split;
}

}  // namespace

hml_sgemm_config heuristic_config(const GemmProblem &p, int algo) {
  hml_sgemm_config c = {};
  if (algo == HML_ALGO_BF16X3 || algo == HML_ALGO_BF16X6 || algo == HML_ALGO_TF32X3 ||
      algo == HML_ALGO_FP16X3) {
    int best = -1;
    // the narrowest single-CTA (128-row) tile that holds N
    for (int v = 0; v < tc_num_shapes(); ++v) {
      int bm, bn;
      tc_shape(v, &bm, &bn);
      if (bm != 128) continue;
      best = v;
      if (bn >= p.N) break;
    }
    if (best >= 0) {
      int bm, bn;
      tc_shape(best, &bm, &bn);
      const int64_t tiles = ((p.M + bm - 1) / bm) * static_cast<int64_t>((p.N + bn - 1) / bn);
      int stages = 2;
      for (int st : {4, 6, 8})
        if (tc_config_fits(bn, tc_ns(algo), st)) stages = st;
      c = {algo, bm, bn, choose_split(tiles, p.K, 1, 256), stages, best};
      return c;
    }
  }
  // SIMT, N <= 8 with contiguous columns of A: the stream-K kernel with the
  // narrowest NB that holds N and its deepest ring (measured on B200,
  // 65536 x 8 x 4096: 6.5 TB/s against 4.8 for the tiled kernel)
  for (int i = 0; i < stream_num_variants(); ++i) {
    const int nb = stream_tile_n(i);
    if (nb < p.N) continue;
    const hml_sgemm_config sc = {HML_ALGO_SIMT, 128, nb, 1, stream_max_stages(nb),
                                 simt_num_shapes() + i};
    if (check_stream(p, sc) == HML_STATUS_SUCCESS) return sc;
    break;
  }
  // SIMT, measured on B200 (M = 1024 to 65536, K = 4096, and squares to
  // 8192): 128-row tiles 8, 16, 32 and 64 wide up to those N, except 256 x 64
  // tiles of 4-row micro-tiles from N = 33 once M gives them 64 row tiles
  // (16384 x 64: 208 us against 228); above N = 64 those 256 x 64 tiles (52
  // TFLOP/s at N = 128) unless 32-wide tiles, at about 42 TFLOP/s, leave
  // enough fewer columns idle (N = 96: 1.27 ms against 1.31)
  int var;
  if (p.N <= 8) var = 1;
  else if (p.N <= 16) var = 0;
  else if (p.N <= 32) var = 2;
  else if (p.N <= 64) var = p.M >= 64 * 256 ? 6 : 7;
  else {
    const int64_t cols32 = (p.N + 31) / 32 * 32, cols64 = (p.N + 63) / 64 * 64;
    var = cols32 * 52 < cols64 * 42 ? 2 : 6;
  }
  return simt_config(p, var);
}

// The tiled SIMT configuration of micro-tile shape `var` for this problem.
// split_k so the grid covers every CTA slot of the machine, at most 8 (4096
// x 32 x 4096: 41 us against 68 at 16), and 2 for tiles
// of two CTAs an SM where the grid is under two waves and K is long (65536
// x 128 x 4096 on 256 x 64 tiles: 1.31 ms; one CTA an SM measured slower
// split); a 3-deep ring where both CTAs of an SM fit with it, else 2
// (deeper rings measured no faster and cost the second CTA).
hml_sgemm_config simt_config(const GemmProblem &p, int var) {
  int bm, bn, wk;
  simt_shape(var, &bm, &bn, &wk);
  const int per_sm = simt_ctas_per_sm(var);
  const int64_t tiles = ((p.M + bm - 1) / bm) * static_cast<int64_t>((p.N + bn - 1) / bn);
  int split = std::min(choose_split(tiles, p.K, per_sm, 128), 8);
  if (split == 1 && per_sm == 2 && tiles < 2LL * sm_count() * per_sm && p.K >= 2048) split = 2;
  // the per-CTA share of shared memory, less barriers and alignment slack
  const size_t budget = (227 * 1024) / per_sm - 2048;
  const int stages = static_cast<size_t>(bm + bn) * 128 * 3 <= budget ? 3 : 2;
  return hml_sgemm_config{HML_ALGO_SIMT, bm, bn, split, stages, var};
}

// A reference v1 SGEMM rule (src/hml_sgemm_kernel.cu:189-237: kernel type
// and rowStops for the class K' = min(K, 96), colStops = ceil(min(N, 96) /
// 16) of a row-major M x N x K problem) mapped onto the tiled SIMT family,
// the counterpart of the reference's tiled SIMT kernels: a tile of
// 16 * rowStops rows (basic kernel: 6 x 6 stops) becomes the 128- or
// 256-row SIMT tile nearest to it, its 16 * colStops columns the narrowest
// SIMT tile width that holds min(N, 16 * colStops) of the problem's columns.
// False when no rule applies or the mapped configuration cannot run.
bool v1_rule_config(const GemmProblem &p, int K_row, int N_row, hml_sgemm_config *c) {
  int type = 0, row_stops = 0;
  if (!cfg_v1_sgemm_rule(K_row, N_row, &type, &row_stops)) return false;
  const int col_stops = type == 0 ? 6 : (std::min(N_row, 96) + 15) / 16;
  const int rows = 16 * (type == 0 ? 6 : row_stops);
  const int want_m = rows >= 192 ? 256 : 128;
  const int want_n = std::min(p.N, 16 * col_stops);
  int best = -1, best_bn = 0, widest = -1, widest_bn = 0;
  for (int v = 0; v < simt_num_shapes(); ++v) {
    int bm, bn, wk;
    simt_shape(v, &bm, &bn, &wk);
    if (bm != want_m) continue;
    if (bn >= want_n && (best < 0 || bn < best_bn)) {
      best = v;
      best_bn = bn;
    }
    if (bn > widest_bn) {
      widest = v;
      widest_bn = bn;
    }
  }
  if (best < 0) best = widest;
  if (best < 0) return false;
  const hml_sgemm_config cand = simt_config(p, best);
  if (!check_config_ok(p, cand)) return false;
  *c = cand;
  return true;
}

// A predicted split-BF16 configuration brought to the tile that holds N where
// that is always the better one; the network, smooth in N and M, misses it
// near the edges (65536 x 64 x 4096, A K-contiguous: 311 us with the 128-wide
// tile it takes, 238 with the 64-wide; 14031 x 80 x 1488: 36 us with the
// 128-wide, 50 with two 64-wide).  Timed both ways:
//   * a tile twice as wide as N needs is no faster (32 < N <= 64 15 % slower at
//     the median, narrower N likewise);
//   * several narrower tiles are no faster where the row tiles fill more than
//     half of the SMs but one wave, or two waves and more (20 to 40 % slower at
//     the median; elsewhere they often win);
//   * from two waves on, K is better whole.
// The family stays the network's: the SIMT sums of a short K are closer to the
// exact ones (about 1e-7 of the largest, BF16X6 5e-7).
static void fit_tile_to_n(const GemmProblem &p, hml_sgemm_config *c) {
  if (c->algo != HML_ALGO_BF16X6 && c->algo != HML_ALGO_BF16X3) return;
  hml_sgemm_config n = heuristic_config(p, c->algo);
  if (n.algo != c->algo) return;
  const int64_t tiles = (static_cast<int64_t>(p.M) + 127) / 128, sms = sm_count();
  const bool holds = n.tile_n >= p.N;
  const bool waves = tiles >= 2 * sms, one = 2 * tiles > sms && tiles <= sms;
  const bool wider = 2 * n.tile_n <= c->tile_n;
  const bool narrower = holds && c->tile_n < n.tile_n && (waves || one);
  if (!wider && !narrower && !(holds && waves && c->split_k > 1)) return;
  n.split_k = waves || narrower ? 1 : c->split_k;
  if (check_config_ok(p, n)) *c = n;
}

hml_status select_config(const GemmProblem &p, hml_sgemm_config *c, cudaStream_t s) {
  if (tuned_lookup(p, c) && check_config_ok(p, *c)) return HML_STATUS_SUCCESS;
  if (predictor_lookup(p, c, s) && check_config_ok(p, *c)) {
    fit_tile_to_n(p, c);
    return HML_STATUS_SUCCESS;
  }
  // Measured on B200 (M = 65536, K = 4096): FP32 SIMT wins at N <= 16 (the
  // HBM-bound GEMV-like shapes); the split-BF16 tensor-core forms win from
  // N = 32 on.  BF16X6 keeps FP32-level accuracy; BF16X3 (faster, ~2**-17)
  // only in the fast math mode.
  if (p.N > 16 && p.M >= 1024 && p.K >= 64) {
    const int algo = math_mode() == HML_MATH_FAST ? HML_ALGO_BF16X3 : HML_ALGO_BF16X6;
    const hml_sgemm_config tc = heuristic_config(p, algo);
    if (check_config_ok(p, tc)) {
      *c = tc;
      return HML_STATUS_SUCCESS;
    }
  }
  *c = heuristic_config(p, HML_ALGO_SIMT);
  return HML_STATUS_SUCCESS;
}

// The BF16X6 tile of a problem with an unaligned A that an addressable one would
// be SIMT for, or one of K < 256 taken whole: the narrowest whose grid is one wave at most, K split as ever.
// These are short, and their time is a CTA's rather than the machine's (B200, K
// odd, row-major, the tile that holds N / this one / SIMT: 1501 x 300 x 101 25.1,
// 15.5, 15.5 us; 3257 x 104 x 127 24.0, 13.1, 18.9; 1021 x 130 x 301 25.1, 13.1,
// 17.2; 1501 x 40 x 601 18.9, 14.8, 16.9).  From K = 256 on the measured
// BF16X6 choice is the better one (1021 x 256 x 601 16.8 us, 25.0).
static hml_sgemm_config unaligned_tile(const GemmProblem &p) {
  hml_sgemm_config c = heuristic_config(p, HML_ALGO_BF16X6);
  const int64_t rows = (static_cast<int64_t>(p.M) + 127) / 128;
  for (int v = c.variant - 1; v >= 0; --v) {
    int bm, bn;
    tc_shape(v, &bm, &bn);
    const int64_t tiles = rows * ((p.N + bn - 1) / bn);
    if (tiles > sm_count()) break;
    c.tile_n = bn;
    c.variant = v;
    c.split_k = choose_split(tiles, p.K, 1, 256);
  }
  return c;
}

// Where the tensor cores take a problem whose A TMA cannot address as it
// stands: wherever they would take it with an addressable A, and where SIMT
// would from M K max(N, 8) = 2^25 on, with 40 row tiles from M K N = 2^24 on.
// The SIMT tiles then stage A with 4-byte cp.async and fall behind early
// (B200, odd K row-major: 2048 x 16 x 1025, at the line, 15.0 us against 12.1;
// 32768 x 8 x 1025 82 against 48; 32768 x 64 x 3001 737 against 119; 5968 x 10
// x 438 18.9 against 12.6; 12001 x 6 x 301 15.5 against 11.1); below the lines
// one launch beats two (2048 x 8 x 257 7.8 us against 10.3; 4001 x 12 x 501
// 12.7 against 14.1; 30001 x 2 x 101 10.8 against 13.3).  Not below K = 100:
// from there on the error is no larger than SIMT's (RMS 0.7 to 0.9 of it over
// N = 2 to 100, K = 101 to 3001), at K = 65 its maximum is (1.7e-7 against
// 1.2e-7).
//
// A record that the program measured or loaded for exactly this shape stands if
// it can run A as it is.  Else one selection serves both ways: the choice for
// the same problem with an addressable A, which where it is SIMT and can read A
// is also the choice among the configurations that can.
hml_status select_auto(const GemmProblem &p, hml_sgemm_config *c, bool *unaligned,
                       cudaStream_t s) {
  *unaligned = false;
  const int64_t ld = p.a_kcontig() ? p.sam : p.sak;
  const bool base_ok = (reinterpret_cast<uintptr_t>(p.A) & 15u) == 0;
  if ((base_ok && ld % 4 == 0) || !tc_unaligned_ok(p)) return select_config(p, c, s);
  if (tuned_by_user(p, c) && check_config_ok(p, *c)) return HML_STATUS_SUCCESS;
  GemmProblem q = p;
  q.A = reinterpret_cast<const float *>(reinterpret_cast<uintptr_t>(p.A) & ~uintptr_t(15));
  (p.a_kcontig() ? q.sam : q.sak) = (ld + 3) / 4 * 4;
  if (select_config(q, c, s) != HML_STATUS_SUCCESS) return select_config(p, c, s);
  const double mk = static_cast<double>(p.M) * p.K;
  if (c->algo == HML_ALGO_SIMT &&
      (p.K < 100 || (mk * std::max(p.N, 8) < 0x1p25 && (p.M < 40 * 128 || mk * p.N < 0x1p24))))
    return check_config_ok(p, *c) ? HML_STATUS_SUCCESS : select_config(p, c, s);
  if (c->algo != HML_ALGO_BF16X6 || (p.K < 256 && c->split_k == 1)) *c = unaligned_tile(q);
  *unaligned = true;
  return HML_STATUS_SUCCESS;
}

}  // namespace hml
