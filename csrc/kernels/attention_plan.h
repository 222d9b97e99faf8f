// How prompts over one-byte pages share a tile's keys among the CTAs of a cluster (attention_fp8.cu), from sizes alone.
#pragma once

#ifdef __CUDACC__
#define OGB_BOTH __host__ __device__
#else
#define OGB_BOTH
#endif

namespace ogb {

// log2 of the rows that a head takes among the 64 accumulator rows of a tile with `rows` query rows: 64, 32, 16 or 8 rows, 1, 2, 4 or 8 heads.
OGB_BOTH inline int prefill_row_bits(int rows) { return rows > 32 ? 6 : rows > 16 ? 5 : rows > 8 ? 4 : 3; }

// The merge takes about as long as three blocks of 64 keys (10 us, 3.5 us): a tile of fewer than this is walked by one CTA (5 blocks: 25 us
// whole, 29 shared).
constexpr int kShareBlocks = 8;

// CTAs that may share a tile: as many as have an SM of their own when the tiles have `q_rows / tiles` rows each.  Two of these CTAs on an SM take
// 6 us a block instead of 3.5 (4 sequences of 16 rows and 6000 keys, 28 heads over 4: 331 us whole, 152 in clusters of 8, 97 in clusters of 4;
// 64 rows and 1000 keys: 68 whole, 140 in clusters of 8).  max_keys: what no context is longer than; a cluster whose CTAs leave at once
// costs 4 us.
inline int prefill_splits(int tiles, int q_rows, int hkv, int group, long long max_keys, int sms) {
  const int heads = 64 >> prefill_row_bits((q_rows + tiles - 1) / tiles);
  const long long ctas = static_cast<long long>(tiles) * hkv * ((group + heads - 1) / heads), blocks = (max_keys + 63) / 64;
  int splits = 1;
  while (splits < 8 && 2 * splits * ctas <= sms && blocks >= kShareBlocks && 4 * splits <= blocks) splits *= 2;
  return splits;
}

// Of those, the ones that do share a tile with `blocks` blocks: two blocks each and more.  The others leave at once.
OGB_BOTH inline int prefill_shares(int splits, int blocks) {
  int n = 1;
  while (blocks >= kShareBlocks && 2 * n <= splits && 4 * n <= blocks) n *= 2;
  return n;
}

}  // namespace ogb
