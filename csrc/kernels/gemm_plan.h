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
// 3584 x 18944 gain 1244 -> 690 and 298 -> 234 us; with K = 3584 (2304 rows: 54 -> 71 us) the fix-ups are what is left.
constexpr float kSkPartial = 25.0f;

// How many of a launch's first tiles stream-K cuts into ranges: all when there are fewer than CTAs, else those of the incomplete last wave,
// and a wave more where they are so few that many CTAs would share each of them.
inline int sk_cut_tiles(int tiles, int ctas) {
  if (tiles <= ctas) return tiles;
  const int rest = tiles % ctas;
  return 2 * ctas > 7 * rest ? rest + ctas : rest;
}

// A launch's rule: the fix-up's cost, whether all tiles are cut, and whether stream-K may be chosen at all.
struct SkRule {
  float fix;
  bool all, enabled;
  int cut(int tiles, int sms) const { return all ? tiles : sk_cut_tiles(tiles, sms); }
};
inline SkRule sk_rule(bool scatter, bool tile_sums, bool enabled) { return SkRule{scatter ? kSkFixScatter : kSkFixPlain, scatter || tile_sums, enabled}; }

// The cost of the fix-ups of a launch, in k-blocks.
inline float sk_fix(int tiles, int k_blocks, int sms, const SkRule& rule) {
  const int cut = rule.cut(tiles, sms);
  const float shared = static_cast<float>(sms) / static_cast<float>(std::max(cut, 1));
  if (cut < tiles) {
    const float own = kSkPartial * (1.f + shared);
    return own < 0.5f * static_cast<float>(k_blocks) ? 0.25f * own : 1e6f;
  }
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

}  // namespace ogb
