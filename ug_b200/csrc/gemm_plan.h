// Which shape a product runs on: host arithmetic only, by predicted time.
#pragma once
#include <algorithm>
#include <cstddef>

// ---- tcgen05 kernel (gemm_tcgen05.cu) -------------------------------------------------------------------------------
constexpr int UGB_TC_BK = 64;              // k elements of a block: one 128-byte swizzle row of 16-bit values

// Number of partials ugb_tc_gemm writes for a requested split factor.
inline int ugb_tc_gemm_effective_splits(size_t k, int splits) {
  const int k_blocks = (int)((k + UGB_TC_BK - 1) / UGB_TC_BK);
  if (splits < 1) splits = 1;
  if (splits > k_blocks) splits = k_blocks;
  const int per = (k_blocks + splits - 1) / splits;
  return (k_blocks + per - 1) / per;
}

// Tile shape for more than 64 rows: width, 256-row tiles on pairs of CTAs, and a k split where the caller takes f32 partials
// (max_splits > 1; the pair shapes do not split).  `pairs`: pairs may be chosen at all.
struct ugb_tc_plan { int bn = 0, splits = 1; bool pair = false; };

// Time of a product, in us: a launch and its epilogue, and for every round of tiles its k blocks at the pace that a tile of this
// shape keeps, which falls as more SMs are at work (L2, and the clock under the power limit).  Fitted to timed products of 100-4096
// rows, bf16, [n, k] weights.  Against every shape on 32 of them (100 to 4096 rows, n of 2048 to 11264, k of 2048 and 5632) the choice is within
// 2 % of the best on 29 and 7 % off at most.  256 x 256 pairs above 128 rows and 128 x 64 below, the rule before, take 17.7 us for
// [777, 2048] x [2560, 2048]^T where the choice takes 12.0, 16.3 and 11.6 for x [2048, 2048]^T, 37.6 and 35.4 for x [11264, 2048]^T, 32.6 and 23.5
// for [777, 5632] x [2048, 5632]^T; from 2048 rows on mostly the same shape.
inline ugb_tc_plan ugb_tc_gemm_plan(int sm_count, size_t batch, size_t m, size_t n, size_t k, bool b_is_nk, bool pairs, int max_splits) {
  static const struct { int bn; bool pair; float pace, crowd, fixed; } shapes[] = {
      {256, true, .269f, .097f, 10.4f}, {192, true, .211f, .066f, 9.7f}, {128, true, .210f, .023f, 8.4f}, {256, false, .360f, .071f, 9.0f},
      {192, false, .255f, .058f, 8.4f}, {128, false, .212f, .032f, 7.7f}, {64, false, .186f, .008f, 7.8f}};
  const size_t k_blocks = (k + UGB_TC_BK - 1) / UGB_TC_BK;
  ugb_tc_plan best;
  float least = 0.f;
  for (const auto &s : shapes) {
    if (s.pair && (!pairs || m <= 128 || sm_count < 2)) continue;
    if (s.pair && s.bn == 192 && !b_is_nk) continue;                   // n-major B is boxed in 64-column pieces
    const size_t rows = s.pair ? 256 : 128, slots = s.pair ? sm_count / 2 : sm_count;
    const size_t tiles = (m + rows - 1) / rows * ((n + s.bn - 1) / s.bn) * batch;
    for (int want = 1; want <= (s.pair ? 1 : max_splits); ++want) {
      const int splits = ugb_tc_gemm_effective_splits(k, want);
      if (splits != want) continue;
      const size_t work = tiles * splits, rounds = (work + slots - 1) / slots;
      const float busy = work < slots ? (float)work / slots : 1.f;
      float t = s.fixed + (rounds - 1) + rounds * ((k_blocks + splits - 1) / splits) * (s.pace + s.crowd * busy);
      t += (splits - 1) * (float)(m * n) * 8e-6f / 3.f;                // each further partial is written and read, about 3 TB/s
      if (s.bn == 256 && s.pair) t *= 0.95f;                           // the shape that everything large runs on: only for a clear gain
      if (least == 0.f || t < least) { least = t; best.bn = s.bn; best.splits = splits; best.pair = s.pair; }
    }
  }
  return best;
}

// ---- FFMA kernel (matmul.cu) ------------------------------------------------------------------------------------------
// Warps over rows and over a slice's k, and CTAs along k, for a product on f32_tile_kernel: the least time of the fullest SM.
// In SM cycles, fitted to 49 timed combinations of eight products of 40-2048 rows (off by 4 % on average): the share of the FMA
// pipe that one CTA on an SM or several reach, what the k split inside a CTA costs of it, and what a CTA spends besides.
// Turned: columns that leave most of a 128-wide tile empty are the rows of a 32- or 64-row tile instead; the results are then
// stored one by one, about SCATTER cycles per 32 rows of a tile (64 times [1339, 597] x [597, 19] in bf16 506 us as it lies, 303 turned).
struct ugb_f32_shape { int wm, wk, split; double cost; bool turned; };
inline ugb_f32_shape ugb_f32_gemm_shape(int sm_count, size_t b, size_t m, size_t n, size_t k) {
  constexpr double ONE = 0.62, SEVERAL = 0.75, SHARE[] = {1.0, 0.85, 0.72}, CTA = 1300, REDUCE = 2600, RANK = 400, SCATTER = 4000;
  ugb_f32_shape best{4, 1, 1, 0, false};
  auto consider = [&](int i, bool turned) {
    const int wm = 4 >> i, wk = 1 << i;
    const size_t rows = ((turned ? n : m) + 32 * wm - 1) / (32 * wm), tiles = rows * (((turned ? m : n) + 127) / 128) * b;
    if (rows > 65535) return;
    for (int split = 1; split == 1 || (split <= 8 && k / split >= 64); split *= 2) {
      const double ctas = (double)((tiles * split + sm_count - 1) / sm_count);
      const double mma = 32.0 * wm * ((k + split - 1) / split) / (SHARE[i] * (ctas < 2 ? ONE : SEVERAL));
      const double cost = ctas * (mma + CTA + (wk * split > 1 ? REDUCE : 0) + (split > 1 ? RANK * split : 0) + (turned ? SCATTER * wm / split : 0));
      if (best.cost == 0 || cost < best.cost) best = {wm, wk, split, cost, turned};
    }
  };
  for (int i = 0; i < 3; ++i) consider(i, false);
  if (n <= 64 && n < m)
    for (int i = 1; i < 3; ++i) consider(i, true);
  return best;
}

// ---- f32 products on the tensor cores (gemm_f32_split.cu) -------------------------------------------------------------------
// Tile width and split of k by predicted time, and whether that is less than the FFMA kernel's.  In us, fitted to 142 timed combinations of 33
// products of 17-2048 rows (off by 5 % on average, too little by up to 15 % where many short tiles store their results; the choice is the best on all): a launch, per round of tiles a fixed part and 32-k
// stages that widen with the tile and slow down a little as more SMs are at work, and the exchange of sums.  Clusters of 4 and 8 find fewer
// SMs: those of a cluster have to be neighbours.
//
// Short sums stay with the FFMA kernel, whose error may be the smaller one there.  It forms a result in wk * split chains of additions; the tensor
// core's cut-off sums of 16 products are ahead of chains of 100 and more whatever is summed.  Worst are softmax probabilities (of
// deviation 3 and 8) times values of one sign: at chains of 30 to 40 additions up to 1.26 times the FFMA kernel's error, 40 to 56 1.18, 56 to 80 1.09, 80 to
// 96 1.04, above 0.93; values of normal distribution 0.4 to 0.5, uniform ones 0.7 to 0.8 (2-norms against 64 bits, 2400 products of 130 sizes).
constexpr size_t UGB_F32_SPLIT_CHAIN = 100;
struct ugb_f32_split_plan { int bn = 0, split = 1; };          // bn 0: not on the tensor cores
inline ugb_f32_split_plan ugb_f32_gemm_split_plan(int sm_count, size_t b, size_t m, size_t n, size_t k, bool rows_contiguous) {
  ugb_f32_split_plan best;
  if (m == 0 || n == 0 || b == 0) return best;
  if (n <= 32 && n < m) return best;       // a quarter of the 128 lanes: the FFMA kernel's turned tiles (5 of [3922, 88] x [88, 8] 14.9 us here, 11.2 there)
  const ugb_f32_shape ffma = ugb_f32_gemm_shape(sm_count, b, m, n, k);
  if (k < UGB_F32_SPLIT_CHAIN * ffma.wk * ffma.split) return best;
  double least = 0.93 * (ffma.cost / 1900 + 2.5);
  for (int split = 1; split <= 8 && (split == 1 || k / split >= 64); split *= 2)
    for (int bn : {32, 64, 96}) {
      if (rows_contiguous && bn != 64) continue;
      const size_t tiles = (n + 127) / 128 * ((m + bn - 1) / bn) * b * split, slots = std::max<size_t>(split, split <= 2 ? sm_count : sm_count * (split == 4 ? 92 : 75) / 100);
      if (split > 1 && tiles > slots) continue;                        // several rounds are better spent on whole sums (2048 x 4096 x 2048, 96 rows: 420 against 369)
      const double stages = (double)(((k + split - 1) / split + 31) / 32), busy = std::min(1.0, (double)tiles / sm_count);
      const double us = 2.0 + (double)((tiles + slots - 1) / slots) * (3.6 + stages * (0.521 + 0.0056 * bn) * (0.9 + 0.1 * busy)) + (split > 1 ? 1.3 + 0.0145 * bn : 0);
      if (us < least) { least = us; best = {bn, split}; }
    }
  return best;
}
