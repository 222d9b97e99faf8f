// The tile kernel's choice between whole tiles and stream-K (gemm_tcgen05.cu), from sizes alone.
#pragma once
#include <algorithm>

namespace ogb {

// Stream-K pays when round-robin tiles would leave a large part of the last wave idle and the fix-up is cheap next
// to a tile: every CTA boundary that falls inside a tile costs one fp32 partial written and read back and a flag wait
// in the finisher.  `fix` is that cost in k-blocks of tensor-core time.  Measured on the 7B shapes (tile widths 32 - 256
// with and without stream-K, M = 32 - 1472): about 40 for a plain epilogue -- with 13 the estimate chose wide stream-K
// tiles for K = 3584 projections that ran 1.3 - 1.5x slower than plain 128-wide tiles -- while the scatter epilogue of
// the tensor-parallel path, whose tiles end in stores to other GPUs, keeps the 13 it was tuned with, and all tiles cut.
constexpr float kSkFixPlain = 40.0f;
constexpr float kSkFixScatter = 13.0f;
// A finisher adds the partials of a tile one after the other, so the fix-up grows with the CTAs that share a tile once they are many
// (8 tiles on 148 SMs, 19 each, took 123 us where whole tiles take 20).
constexpr float kSkShared = 6.0f;
// With whole waves after the cut tiles (sk_cut_tiles) the fix-ups pass under the main loops of the tiles after them, as long as those
// are long enough.  A CTA's partial costs about 25 k-blocks to write and add (0.3 us each at 256 columns): 7100 and 2304 rows against
// 3584 x 18944 gain 1244 -> 690 and 298 -> 234 us; with K = 3584 (2304 rows: 54 -> 71 us) the fix-ups are what is left.  Where the main
// loops are too short for that, all tiles of 256 columns may be cut, as long as W stays in L2 for the CTAs that read it out of step: 4096 rows
// against 3584 x 5120 (37 MB) 146 us in whole tiles, 125 so; 7100 against 2048 x 4096 125, 104; but 512 against 28672 x 5120 (294 MB) 161, 178,
// and 300 against 28672 x 4096 in tiles of 192 98, 144.
constexpr float kSkPartial = 25.0f;
constexpr long long kSkAllBytes = 150ll << 20;

// How many of a launch's first tiles stream-K cuts into ranges: all when there are fewer than CTAs, else those of the incomplete last wave,
// and a wave more where they are so few that many CTAs would share each of them.
inline int sk_cut_tiles(int tiles, int ctas) {
  if (tiles <= ctas) return tiles;
  const int rest = tiles % ctas;
  return 2 * ctas > 7 * rest ? rest + ctas : rest;
}

// What the partials of the CTAs that share a tile cost, in k-blocks, when `cut` tiles are.
inline float sk_partials(int cut, int sms) { return kSkPartial * (1.f + static_cast<float>(sms) / static_cast<float>(std::max(cut, 1))); }

// A launch's rule: the fix-up's cost, whether all tiles are cut always, or where cutting the last does not pay, and whether stream-K may be
// chosen at all.
struct SkRule {
  float fix;
  bool all, all_else, enabled;
  int cut(int tiles, int k_blocks, int sms) const {
    const int last = all ? tiles : sk_cut_tiles(tiles, sms);
    return all_else && !pays(tiles, last, k_blocks, sms) ? tiles : last;
  }
  // partials of the last tiles pass under the whole ones
  static bool pays(int tiles, int cut, int k_blocks, int sms) { return cut == tiles || sk_partials(cut, sms) < 0.5f * static_cast<float>(k_blocks); }
};
inline SkRule sk_rule(bool scatter, bool tile_sums, bool enabled, int width, long long n, long long k) {
  return SkRule{scatter ? kSkFixScatter : kSkFixPlain, scatter || tile_sums, width == 256 && n * k * 2 <= kSkAllBytes, enabled};
}

// The cost of the fix-ups of a launch, in k-blocks.
inline float sk_fix(int tiles, int k_blocks, int sms, const SkRule& rule) {
  const int cut = rule.cut(tiles, k_blocks, sms);
  if (cut < tiles) return SkRule::pays(tiles, cut, k_blocks, sms) ? 0.25f * sk_partials(cut, sms) : 1e6f;
  const float shared = static_cast<float>(sms) / static_cast<float>(tiles);
  return shared > kSkShared ? rule.fix * shared / kSkShared : rule.fix;
}
inline bool stream_k_applies(int tiles, int k_blocks, int sms, const SkRule& rule) {
  if (!rule.enabled || tiles % sms == 0 || static_cast<long long>(tiles) * k_blocks < 2LL * sms) return false;
  const float w = static_cast<float>(tiles) / static_cast<float>(sms);
  const float dp = static_cast<float>((tiles + sms - 1) / sms);
  const float sk = w + sk_fix(tiles, k_blocks, sms, rule) / static_cast<float>(k_blocks);
  return sk < 0.93f * dp;
}
// Relative duration of a launch with `tiles` tiles of relative cost `cost`: whole waves when tiles are dealt
// round-robin, the exact share plus the fix-up when stream-K spreads the k-blocks evenly.
inline float launch_cost(int tiles, int k_blocks, int sms, float cost, const SkRule& rule) {
  if (stream_k_applies(tiles, k_blocks, sms, rule))
    return (static_cast<float>(tiles) / static_cast<float>(sms) + sk_fix(tiles, k_blocks, sms, rule) / static_cast<float>(k_blocks)) * cost;
  return static_cast<float>((tiles + sms - 1) / sms) * cost;
}

// ----------------------------------------------------------------------------------------
// Products with few rows (gemm_rows.cuh), or the tile kernel.  All times in us on B200, weights from HBM, tile kernel -> few rows.
// ----------------------------------------------------------------------------------------
constexpr int kRowsMaxM = 256;              // rows of the activation tile (the MMA's N)
constexpr int kRowsGatedM = 32;             // of a gated product's
constexpr int kRowsRangesM = 48;            // of one over more tiles than SMs

// Rows up to which a product over `tiles` tiles of 128 columns (of 128 gate and 128 up columns, when gated) comes to the kernels for few rows.
inline int rows_limit(int tiles, int k_blocks, bool gated, bool residual, int sms) {
  if (tiles > sms) {
    // ranges: a tile's epilogue has to pass under the k-blocks of the others, so a range needs enough of them.  N x K at 1 row: 152064 x 3584
    // 225 -> 170, 151936 x 896 79 -> 70, 32000 x 2048 40 -> 39, but 32000 x 896 24 -> 29, 20000 x 576 16 -> 23, and with tiles of 9 k-blocks
    // 151936 x 576 51 -> 57 at 16 rows; at 48: 151936 x 2048 126 -> 125, 65536 x 2048 65 -> 70, 151936 x 896 68 -> 76.
    const long long blocks = static_cast<long long>(tiles) * k_blocks * (gated ? 2 : 1);
    if (k_blocks < 12 || blocks < 52LL * sms) return 0;
    return blocks < 150LL * sms || gated ? kRowsGatedM : kRowsRangesM;
  }
  // One CTA or a cluster per tile.  The tile kernel reads 128 rows of activations for each of its tiles, this one as many as there are, so the line
  // falls with the rows; and it falls with the tiles, as fewer CTAs share a tile and more of the chip is busy in the tile kernel too.
  if (tiles > sms / 2) {
    // a CTA per tile: 16640 x 3584 42 -> 35 at 1 row, 37 -> 37 at 48, 38 -> 42 at 128; 9600 x 2048 26 -> 21, 22 -> 23, 22 -> 27; gated 37888 x 3584
    // 57 -> 49 at 16, 37888 x 2048 44 -> 43 at 16, 42 -> 45 at 32
    if (gated) return k_blocks >= 48 ? kRowsGatedM : 16;
    return k_blocks >= 48 ? 48 : 32;
  }
  if (gated) return kRowsGatedM;
  if (3 * tiles > sms) {
    // two: 7168 x 2048 22 -> 19 at 1 row, 20 -> 19 at 48, 19 -> 21 at 64; x 3584 27 -> 27 at 128, 29 -> 31 at 200; x 8192 52 -> 53 at 256
    return k_blocks >= 96 ? kRowsMaxM : k_blocks >= 48 ? 128 : 48;
  }
  // three to eight: 4608 x 3584 27 -> 13 at 1 row, 22 -> 19 at 256; 3584 x 18944 86 -> 31, 110 -> 48; 3584 x 2048 18 -> 19 at 128, 18 -> 21 at 256;
  // 3584 x 896 13 -> 13 at 64, 12 -> 14 at 128.  With a residual all of them: the sum with it is rounded once here, twice in the tile kernel.
  return residual || k_blocks >= 48 ? kRowsMaxM : k_blocks >= 24 ? 128 : 64;
}
inline bool rows_applies(int m, int n, int k_blocks, bool gated, bool residual, int sms) {
  const int width = gated ? 256 : 128;
  return m <= rows_limit((n + width - 1) / width, k_blocks, gated, residual, sms);
}

// int4 weights (gemm_w4a16.cu): `tiles` of 128 rows of W (of 128 gate and 128 up rows, when gated).  Against gemm_w4a16_tcgen05_kernel, which has
// 64- or 128-column tiles, a CTA each, and its dequantisers' pace:
//   gated: better at all sizes up to 160 rows but ranges of few k-blocks (896 x 40960 at 48 rows 38 -> 46)
//   clusters of three CTAs and more per tile: 896 x 4864 37 -> 16 at 8 rows, 44 -> 21 at 256; 4096 x 896 14 -> 14 at 48, 15 -> 16 at 128
//   two: 6144 x 4096 42 -> 31 at 8 rows, 33 -> 34 at 128, 41 -> 37 at 256; 6144 x 896 15 -> 14 at 8, 14 -> 16 at 64
//   one: every CTA dequantises 128 rows where the other kernel's takes 64: 9728 x 4096 43 -> 49 at 8 rows, 43 -> 53 at 128; but that one has no 64-column
//     tiles left to fill the SMs with beyond 14000, and up to 8 rows its 128-row tile costs: 14336 x 4096 51 -> 49, 18944 x 4096 66 -> 51
//   ranges: up to 32 rows where the other kernel's last wave is short: 22016 x 4096 (172 tiles on 148 SMs) 76 -> 61 at 32 rows, at 48 76 -> 66;
//     32000 x 2048 (250 tiles) 56 -> 49 at 16, 44 -> 49 at 32; up to 8 rows 32000 x 4096 111 -> 83; 896 in K 27 -> 29
inline bool w4_rows_applies(int m, int tiles, int k_blocks, bool gated, int sms) {
  if (m > kRowsMaxM) return false;
  if (tiles > sms) {
    if (m > kRowsRangesM) return false;
    if (gated) return m <= kRowsGatedM || k_blocks >= 24;
    if (k_blocks < 24) return false;
    return m <= 8 || (4 * (tiles % sms) < sms && tiles < 2 * sms && (m <= 32 || k_blocks >= 48));
  }
  if (gated) return true;
  if (tiles > sms / 2) return m <= 8 && 4 * tiles >= 3 * sms && k_blocks <= 96;
  if (7 * tiles > 2 * sms) return k_blocks >= 48 || m <= 16;
  return k_blocks >= 24 || m <= 64;
}

}  // namespace ogb
