// Shared by the products on the tensor cores (gemm_tcgen05.cu, gemm_w4a16.cu): epilogue kinds, activations, division of the work.
#pragma once
#include "common.cuh"

namespace ogb {

constexpr int kBK = 64;  // 64 bf16 = one 128-byte swizzle row

enum GemmEpilogue : int { kEpiNone = 0, kEpiResidual = 1, kEpiSwiGLU = 2, kEpiScatter = 3 };

// Activations ahead of a bf16 rounding: relative errors of a few 1e-7, absolute ones of 1e-7 next to zero.
// 0.5 z (1 + tanh(a)) = z / (1 + exp(-2 a))
OGB_DEVICE float gelu_tanh_fast(float z) {
  const float a = 0.7978845608028654f * fmaf(0.044715f * z * z, z, z);
  return z / (1.f + __expf(fminf(-2.f * a, 80.f)));
}
// the gated epilogue's value for a gate and an up column
OGB_DEVICE float gated_act(const ActArgs& act, float g, float u) {
  if (act.kind == kActGeluTanh) return gelu_tanh_fast(g) * u;
  if (act.kind == kActClampGlu) {
    g = fminf(g, act.a);
    u = fminf(fmaxf(u, -act.a), act.a);
    return g / (1.f + __expf(fminf(-kClampGluSlope * g, 80.f))) * (u + 1.f);
  }
  return g / (1.f + __expf(-g)) * u;
}
// the plain epilogue's value for a result
OGB_DEVICE float plain_act(const ActArgs& act, float v) {
  if (act.kind == kActRelu2) {
    v = fmaxf(v, 0.f);
    return v * v;
  }
  if (act.kind == kActXielu) return fmaf(0.5f, v, v > 0.f ? act.a * v * v : act.b * (__expf(v) - 1.f - v));
  return v;
}

// ----------------------------------------------------------------------------------------
// Work decomposition.  Data-parallel: output tiles are dealt round-robin to the persistent CTAs and a CTA runs the
// whole K loop of each of its tiles.  Stream-K: the (tile, k-block) iterations of all tiles are laid end to end and cut
// into one contiguous, equally long range per CTA, so every SM does the same amount of tensor-core work even when
// the tile count is not a multiple of the SM count.  A range may begin or end in the middle of a tile: the CTA whose
// range holds a tile's last k-block finishes the tile; CTAs that hold an earlier part of it leave their fp32
// accumulator in a workspace slot (one slot per CTA: a range ends inside at most one tile) and raise a flag; the
// finisher, which always has the higher block index, waits for those flags (bounded) and adds the partials before
// its epilogue.  Waiting only on lower-numbered CTAs keeps the scheme free of deadlock whatever the residency, and
// walking every range backwards (GemmWork::next) makes partials the first thing a CTA produces and fix-ups the last.
// With more tiles than CTAs only those of about the last wave are cut (sk_cut_tiles in gemm_plan.h), and they come first: the whole waves that follow
// are dealt round-robin, so that CTAs walk K in step and share what they read through L2 (cut from end to end, 7100 rows
// against a 3584 x 18944 projection drew every operand from HBM again and again: 1101 us), and a fix-up's wait passes
// under the main loop of the tile after it.  Where the order of the sums must stay (tile_sums) and in the scatter epilogue of the
// tensor-parallel path, whose tiles arrive at other GPUs in the order of the ranges, all tiles are cut.
// ----------------------------------------------------------------------------------------
// Tiles of many rows: 16 tiles of A at a time against every tile of W, so that the tiles under way at one moment (about 148) span
// 2048 rows of A and 2400 of W instead of all of A and two tiles of W.
// For an A that does not stay in L2 beside W (kRasterBytes); one that does has the other order a little faster (7100 rows against 37888 x
// 3584, A of 51 MB: 1342 -> 1400 us in groups).
constexpr int kRasterM = 16;
constexpr long long kRasterBytes = 96ll << 20;
OGB_DEVICE void raster_tile(int tile, int m_tiles, int n_tiles, bool grouped, int& mt, int& nt) {
  if (!grouped || m_tiles <= kRasterM) {
    mt = tile % m_tiles;
    nt = tile / m_tiles;
    return;
  }
  const int g = tile / (kRasterM * n_tiles), first = g * kRasterM;
  const int rows = min(kRasterM, m_tiles - first), t = tile - first * n_tiles;
  mt = first + t % rows;
  nt = t / rows;
}

struct GemmSeg {
  int tile, kb0, kb1;
};

struct GemmWork {
  int k_blocks, num_tiles, stride, tile;   // data-parallel cursor
  long long it, it_end;                    // stream-K cursor over iterations
  long long sk_total;                      // iterations that are cut into ranges
  OGB_DEVICE static long long range_begin(long long total, int ctas, int b) {
    const long long base = total / ctas, rem = total % ctas;
    return b * base + (b < rem ? b : rem);
  }
  // the CTA whose range holds iteration i
  OGB_DEVICE static int owner(long long total, int ctas, long long i) {
    const long long base = total / ctas, rem = total % ctas;
    const long long cut = (base + 1) * rem;
    return i < cut ? static_cast<int>(i / (base + 1)) : static_cast<int>(rem + (i - cut) / base);
  }
  // cut: how many of the first tiles are cut into ranges (0: no stream-K)
  OGB_DEVICE GemmWork(int cut, int tiles, int kblocks) : k_blocks(kblocks), num_tiles(tiles) {
    stride = gridDim.x;
    tile = cut + blockIdx.x;
    sk_total = static_cast<long long>(cut) * kblocks;
    it = range_begin(sk_total, stride, blockIdx.x);
    it_end = range_begin(sk_total, stride, blockIdx.x + 1);
  }
  OGB_DEVICE bool next(GemmSeg& s) {
    if (it_end <= it) {
      if (tile >= num_tiles) return false;
      s.tile = tile; s.kb0 = 0; s.kb1 = k_blocks;
      tile += stride;
      return true;
    }
    // The range is walked from its end to its beginning.  The segment at the end of the range is the head of a tile
    // that a higher-numbered CTA finishes: it is produced first, so the finisher -- for which that tile's tail is the
    // *last* segment -- finds the partial waiting instead of stalling on a neighbour that has its whole range to go.
    s.tile = static_cast<int>((it_end - 1) / k_blocks);
    const long long tile_start = static_cast<long long>(s.tile) * k_blocks;
    const long long seg_begin = tile_start > it ? tile_start : it;
    s.kb0 = static_cast<int>(seg_begin - tile_start);
    s.kb1 = static_cast<int>(it_end - tile_start);
    it_end = seg_begin;
    return true;
  }
};

}  // namespace ogb
