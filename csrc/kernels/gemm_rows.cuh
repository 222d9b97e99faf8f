// Products with few rows: C[M,N] = A[M,K] * W[N,K]^T for M up to a few hundred (decode steps, short prompts, LM heads).
//
// What bounds them is the stream of W from HBM; the tile kernel (gemm_tcgen05.cu) cannot keep it going at these sizes: its A tile
// has 128 rows, most of them padding, and 32- to 256-wide tiles of N leave SMs idle (28 tiles of a 3584-wide projection on 148
// SMs) or spend their time in a serial fix-up.  Here the operands change places: 128 rows of W are the M side of tcgen05.mma, the
// activations its N side, padded to a multiple of 16 rows only, so a stage of the ring is W almost alone (18 KB at 16 rows).
// How the work is divided:
//   * fewer tiles than SMs: a cluster of up to 8 CTAs shares a tile, each takes a part of K.  When its products have retired a CTA
//     lays its fp32 accumulator into the ring it no longer needs; after one cluster barrier every CTA sums its share of the rows out of
//     all shared memories.  No partial crosses L2 and nobody waits for a flag;
//   * more tiles than SMs (LM heads): the (tile, k-block) iterations are laid end to end and cut into equally long ranges, one per
//     SM.  A tile that two ranges share is summed by whichever arrives last: the other leaves its fp32 partial in a workspace
//     slot and goes on.  The partials are added in the order of the ranges (the result does not depend on who is last), a tile's counter
//     wraps to zero, so a replayed graph finds it as the first run did, and a range does its shared tiles first, so that the sums
//     pass under the whole tiles that follow.
// A row of the result leaves as 256 contiguous bytes per warp (four columns a lane); the 64-byte pieces that a thread-per-column
// epilogue stores took longer than the products from 64 rows on.
// TW = 2 takes 128 gate rows of W and their 128 up rows per tile (two accumulators): a packed gated projection, 128 columns of C.
//
// Measured on B200 (weights not in L2): see the rule in gemm_plan.h.
#pragma once
#include <cooperative_groups.h>

#include <map>
#include <mutex>
#include <tuple>

#include "gemm_common.cuh"
#include "gemm_plan.h"

namespace ogb {

constexpr int kRowsThreads = 192;
constexpr int kRowsMaxStages = 12;
constexpr int kRowsSmemMax = 227 * 1024;
constexpr int kRowsBarBytes = 512;
constexpr int kRowsMaxSplit = 8;            // the portable cluster size
constexpr int kRowsStage = 32 * 128 * 4;    // staging of 32 result rows of an accumulator (ranges)

struct RowsGemmParams {
  __nv_bfloat16* C;
  float* C_f32;
  const __nv_bfloat16* bias;                // N readable values, also without has_bias: the load may be made ahead of the test
  const __nv_bfloat16* residual;
  int has_bias;
  int M, N, ldc, ldr;
  int mn;                                   // rows of the activation tile: a multiple of 16, at most kRowsMaxM
  int n_tiles, k_blocks, stages;
  int splits;                               // CTAs (a cluster) per tile; 0: ranges
  int* status;
  float* ws;                                // ranges: [CTA][2][TW][4 quarters][rows / 4][32 columns][4 rows], rows a multiple of 32
  unsigned int* counters;                   // ranges: [CTA], zero between launches
};

// The calling thread's workspace (ogb_launch_scope) where it is large enough for a launch of at most `ctas` CTAs; null: the product is not
// one for these kernels (kRowsDeclined).
constexpr int kRowsDeclined = INT32_MIN;
void* rows_workspace(int ctas, int tw, int mn);
size_t rows_counter_bytes(int ctas);

// CTAs per tile: as many as can run at once in clusters (whole clusters have to fit the hardware's groups of SMs, which the driver knows) and
// leave each two k-blocks.
template <typename Kernel>
static int rows_pick_splits(Kernel kernel, int threads, int smem, int tiles, int k_blocks) {
  static std::mutex mu;
  static std::map<std::tuple<int, const void*, int>, int> most;  // (device, kernel, shared memory and split) -> clusters at once
  int device = 0;
  if (cudaGetDevice(&device) != cudaSuccess) { cudaGetLastError(); return 1; }
  std::lock_guard<std::mutex> lock(mu);
  for (int s = kRowsMaxSplit; s > 1; --s) {
    if (2 * s > k_blocks) continue;
    const std::tuple<int, const void*, int> key(device, reinterpret_cast<const void*>(kernel), smem * 16 + s);
    auto hit = most.find(key);
    if (hit == most.end()) {
      cudaLaunchConfig_t cfg = {};
      cfg.gridDim = dim3(s);
      cfg.blockDim = dim3(threads);
      cfg.dynamicSmemBytes = smem;
      cudaLaunchAttribute attr[1];
      attr[0].id = cudaLaunchAttributeClusterDimension;
      attr[0].val.clusterDim.x = s;
      attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
      cfg.attrs = attr;
      cfg.numAttrs = 1;
      int n = 0;
      if (cudaOccupancyMaxActiveClusters(&n, kernel, &cfg) != cudaSuccess) { cudaGetLastError(); n = 0; }
      hit = most.emplace(key, n).first;
    }
    if (tiles <= hit->second) return s;
  }
  return 1;
}
template <typename Kernel, typename... Args>
static int rows_launch(Kernel kernel, int grid, int threads, int smem, int splits, cudaStream_t stream, const Args&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  cfg.attrs = attr;
  if (splits > 1) {
    attr[cfg.numAttrs].id = cudaLaunchAttributeClusterDimension;
    attr[cfg.numAttrs].val.clusterDim.x = splits;
    attr[cfg.numAttrs].val.clusterDim.y = attr[cfg.numAttrs].val.clusterDim.z = 1;
    ++cfg.numAttrs;
  }
  if (launch_overlap()) {
    attr[cfg.numAttrs].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[cfg.numAttrs].val.programmaticStreamSerializationAllowed = 1;
    ++cfg.numAttrs;
  }
  return static_cast<int>(cudaLaunchKernelEx(&cfg, kernel, args...));
}

// The iterations [it0, it1) of a CTA, tile by tile: the tile it shares with the CTA before it, the one it shares with the CTA after it,
// then the whole ones.
struct RowsSegs {
  long long it0, it1, first_end, last_begin, mid;
  int k_blocks, state = 0;
  OGB_DEVICE RowsSegs(const RowsGemmParams& p) : k_blocks(p.k_blocks) {
    if (p.splits > 0) {
      const long long base = static_cast<long long>(blockIdx.x / p.splits) * k_blocks;
      const int rank = blockIdx.x % p.splits;
      it0 = base + k_blocks * rank / p.splits;
      it1 = base + k_blocks * (rank + 1) / p.splits;
    } else {
      const long long total = static_cast<long long>(p.n_tiles) * k_blocks;
      it0 = GemmWork::range_begin(total, gridDim.x, blockIdx.x);
      it1 = GemmWork::range_begin(total, gridDim.x, blockIdx.x + 1);
    }
    first_end = it0 % k_blocks != 0 ? min(it1, (it0 / k_blocks + 1) * k_blocks) : it0;
    last_begin = it1 % k_blocks != 0 ? max(first_end, it1 / k_blocks * k_blocks) : it1;
    mid = first_end;
  }
  OGB_DEVICE bool next(int& tile, int& kb0, int& kb1) {
    long long a = 0, b = 0;
    if (state == 0) { a = it0; b = first_end; state = 1; }
    if (state == 1 && a >= b) { a = last_begin; b = it1; state = 2; }
    if (state == 2 && a >= b) {
      if (mid >= last_begin) return false;
      a = mid;
      b = mid = mid + k_blocks;
    }
    tile = static_cast<int>(a / k_blocks);
    kb0 = static_cast<int>(a - static_cast<long long>(tile) * k_blocks);
    kb1 = static_cast<int>(b - static_cast<long long>(tile) * k_blocks);
    return true;
  }
};

// The k-blocks of a CTA one by one.
struct RowsCursor {
  RowsSegs segs;
  int tile = 0, kb = 0, kb1 = 0;
  bool more;
  OGB_DEVICE explicit RowsCursor(const RowsGemmParams& p) : segs(p) { more = segs.next(tile, kb, kb1); }
  OGB_DEVICE void step() {
    if (more && ++kb == kb1) more = segs.next(tile, kb, kb1);
  }
};

// Four neighbouring columns n .. n + 3 of row m: sums (and the up half's, when gated) -> the stored result.
template <int EPI>
OGB_DEVICE void rows_store(const RowsGemmParams& p, const ActArgs& act, int m, int n, const float4& a, const float4& b) {
  const int n_out = (EPI == kEpiSwiGLU) ? p.N / 2 : p.N;
  if (n >= n_out) return;
  float v[4] = {a.x, a.y, a.z, a.w};
  const bool full = n + 4 <= n_out;
  if constexpr (EPI == kEpiSwiGLU) {
    const float u[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) v[i] = gated_act(act, v[i], u[i]);
  } else {
    if (p.has_bias != 0) {
#pragma unroll
      for (int i = 0; i < 4; ++i) v[i] += __bfloat162float(p.bias[min(n + i, p.N - 1)]);
    }
    if constexpr (EPI == kEpiResidual) {
      const __nv_bfloat16* rs = p.residual + static_cast<size_t>(m) * p.ldr + n;
      if (full) {
        const uint2 r = *reinterpret_cast<const uint2*>(rs);
        const float2 r0 = unpack_bf16(r.x), r1 = unpack_bf16(r.y);
        v[0] += r0.x; v[1] += r0.y; v[2] += r1.x; v[3] += r1.y;
      } else {
        for (int i = 0; i < n_out - n; ++i) v[i] += __bfloat162float(rs[i]);
      }
    } else {
#pragma unroll
      for (int i = 0; i < 4; ++i) v[i] = plain_act(act, v[i]);
    }
  }
  const size_t at = static_cast<size_t>(m) * p.ldc + n;
  if (p.C_f32 != nullptr) {
#pragma unroll
    for (int i = 0; i < 4; ++i)
      if (n + i < n_out) p.C_f32[at + i] = v[i];
  } else if (full) {
    *reinterpret_cast<uint2*>(p.C + at) = make_uint2(pack_bf16(v[0], v[1]), pack_bf16(v[2], v[3]));
  } else {
#pragma unroll
    for (int i = 0; i < 4; ++i)
      if (n + i < n_out) p.C[at + i] = __float2bfloat16(v[i]);
  }
}
OGB_DEVICE void rows_epi_sync() { asm volatile("bar.sync 1, 128;" ::: "memory"); }

// Ranges: the four epilogue warps (warp index mod 4 = TMEM lane quarter = columns 32 q .. 32 q + 31 of a tile).  stage: TW * kRowsStage
// bytes, shared_last: one word.
template <int TW, int EPI>
OGB_DEVICE void rows_epilogue(const RowsGemmParams& p, const ActArgs& act, uint32_t tmem_base, int bufs, int acc_cols, uint64_t* tmem_full,
                              uint64_t* tmem_empty, volatile int* abort_flag, float* stage, volatile uint32_t* shared_last) {
  const int q = (threadIdx.x >> 5) & 3, lane = threadIdx.x & 31;
  const int k_blocks = p.k_blocks;
  const long long total = static_cast<long long>(p.n_tiles) * k_blocks;
  const int slot_floats = TW * 4 * acc_cols * 32;
  const int rows = p.M;
  pdl_wait();
  bool ok = true;
  RowsSegs segs(p);
  int tile, kb0, kb1;
  for (int seg = 0; segs.next(tile, kb0, kb1); ++seg) {
    const bool head = kb0 == 0, whole = head && kb1 == k_blocks;
    const int buf = bufs == 2 ? (seg & 1) : 0;
    const uint32_t buf_phase = (bufs == 2 ? seg >> 1 : seg) & 1;
    // every lane polls (each needs the acquire); the vote keeps the warp converged for tcgen05.ld.  After a wait that ran out
    // the warps go on to arrive on the counters of their shared tiles, so that they still wrap to zero.
    if (ok && !__all_sync(0xffffffffu, mbar_wait(&tmem_full[buf], buf_phase))) {
      ok = false;
      if (lane == 0) { atomicOr(p.status, kStatusWaitTimeout); *abort_flag = 1; }
    }
    tc_fence_after();
    const uint32_t t_addr = tmem_base + (static_cast<uint32_t>(q * 32) << 16) + buf * TW * acc_cols;
    int c_lo = 0, c_hi = 0;                                   // the CTAs that share the tile
    if (!whole) {
      c_lo = GemmWork::owner(total, gridDim.x, static_cast<long long>(tile) * k_blocks);
      c_hi = GemmWork::owner(total, gridDim.x, static_cast<long long>(tile + 1) * k_blocks - 1) + 1;
      if (ok) {
        float4* dst = reinterpret_cast<float4*>(p.ws + static_cast<size_t>(blockIdx.x * 2 + (head ? 1 : 0)) * slot_floats) + q * acc_cols * 8 + lane;
#pragma unroll
        for (int w = 0; w < TW; ++w) {
#pragma unroll 1
          for (int c = 0; c < rows; c += 32) {
            uint32_t r[32];
            tmem_ld_32x32(t_addr + w * acc_cols + c, r);
            tmem_ld_wait();
#pragma unroll
            for (int j = 0; j < 32; j += 4)
              if (c + j < rows)
                __stcg(dst + (w * 4 * acc_cols + c + j) * 8, make_float4(__uint_as_float(r[j]), __uint_as_float(r[j + 1]), __uint_as_float(r[j + 2]),
                                                                        __uint_as_float(r[j + 3])));
          }
        }
      }
      tc_fence_before();
      __threadfence();
      rows_epi_sync();
      if (lane == 0) mbar_arrive(&tmem_empty[buf]);
      if (q == 0 && lane == 0) {
        *shared_last = atomicInc(p.counters + c_lo, static_cast<unsigned int>(c_hi - c_lo - 1)) == static_cast<unsigned int>(c_hi - c_lo - 1);
        __threadfence();
      }
      rows_epi_sync();
      const bool last = *shared_last != 0;
      rows_epi_sync();
      if (!__all_sync(0xffffffffu, ok && last)) continue;
    } else if (!ok) {
      continue;
    }
    // 32 rows of accumulator w from row c on: from TMEM, or the partials of all CTAs of the tile in their order
    auto gather = [&](int w, int c, float (&v)[32]) {
      if (whole) {
        uint32_t r[32];
        tmem_ld_32x32(t_addr + w * acc_cols + c, r);
        tmem_ld_wait();
#pragma unroll
        for (int j = 0; j < 32; ++j) v[j] = __uint_as_float(r[j]);
        return;
      }
#pragma unroll
      for (int j = 0; j < 32; ++j) v[j] = 0.f;
      // two CTAs at a time: 64 values in flight per thread
#pragma unroll 1
      for (int x = c_lo; x < c_hi; x += 2) {
        float4 t[2][8];
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          // the first CTA of a tile holds its head (slot 1), the others a later part (slot 0)
          const int from = min(x + i, c_hi - 1);
          const float4* src = reinterpret_cast<const float4*>(p.ws + static_cast<size_t>(from * 2 + (from == c_lo ? 1 : 0)) * slot_floats) +
                              ((w * 4 + q) * acc_cols + c) * 8 + lane;
#pragma unroll
          for (int j = 0; j < 8; ++j) t[i][j] = __ldcg(src + j * 32);
        }
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          if (x + i < c_hi) {
#pragma unroll
            for (int j = 0; j < 8; ++j) { v[4 * j] += t[i][j].x; v[4 * j + 1] += t[i][j].y; v[4 * j + 2] += t[i][j].z; v[4 * j + 3] += t[i][j].w; }
          }
        }
      }
    };
#pragma unroll 1
    for (int c = 0; c < rows; c += 32) {
#pragma unroll
      for (int w = 0; w < TW; ++w) {
        float v[32];
        gather(w, c, v);
#pragma unroll
        for (int j = 0; j < 32; ++j) stage[(w * 32 + j) * 128 + q * 32 + lane] = v[j];
      }
      rows_epi_sync();
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const int m = q * 8 + j;
        if (c + m < rows) {
          const float4 a = *reinterpret_cast<const float4*>(stage + m * 128 + 4 * lane);
          const float4 b = *reinterpret_cast<const float4*>(stage + ((TW - 1) * 32 + m) * 128 + 4 * lane);
          rows_store<EPI>(p, act, c + m, tile * 128 + 4 * lane, a, b);
        }
      }
      rows_epi_sync();
    }
    if (whole) {
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&tmem_empty[buf]);
    }
  }
}

// A cluster per tile.  Epilogue warps lay the accumulator's rows [r0, r0 + count) into `stage` [TW][count][128] ...
template <int TW>
OGB_DEVICE void rows_lay_out(uint32_t tmem_base, int acc_cols, int r0, int count, float* stage) {
  const int q = (threadIdx.x >> 5) & 3, lane = threadIdx.x & 31;
#pragma unroll
  for (int w = 0; w < TW; ++w) {
#pragma unroll 1
    for (int c = 0; c < count; c += 32) {
      uint32_t r[32];
      tmem_ld_32x32(tmem_base + (static_cast<uint32_t>(q * 32) << 16) + w * acc_cols + r0 + c, r);
      tmem_ld_wait();
      float* dst = stage + (static_cast<size_t>(w) * count + c) * 128 + q * 32 + lane;
#pragma unroll
      for (int j = 0; j < 32; ++j)
        if (c + j < count) dst[j * 128] = __uint_as_float(r[j]);
    }
  }
}
// ... and all warps of the cluster's CTA `rank` sum every splits-th row of them over the CTAs.
template <int TW, int EPI>
OGB_DEVICE void rows_sum_cluster(const RowsGemmParams& p, const ActArgs& act, int tile, int rank, int r0, int count, float* stage) {
  const cooperative_groups::cluster_group cluster = cooperative_groups::this_cluster();
  const int warps = blockDim.x >> 5, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int m = rank + p.splits * warp; m < count && r0 + m < p.M; m += p.splits * warps) {
    float4 s[TW];
#pragma unroll
    for (int w = 0; w < TW; ++w) {
      float4 t[kRowsMaxSplit];
      const float* src = stage + (static_cast<size_t>(w) * count + m) * 128 + 4 * lane;
#pragma unroll
      for (int x = 0; x < kRowsMaxSplit; ++x)
        if (x < p.splits) t[x] = *reinterpret_cast<const float4*>(p.splits > 1 ? cluster.map_shared_rank(src, x) : src);
      s[w] = t[0];
#pragma unroll
      for (int x = 1; x < kRowsMaxSplit; ++x)
        if (x < p.splits) { s[w].x += t[x].x; s[w].y += t[x].y; s[w].z += t[x].z; s[w].w += t[x].w; }
    }
    rows_store<EPI>(p, act, r0 + m, tile * 128 + 4 * lane, s[0], s[TW - 1]);
  }
}
// All threads of a CTA, after their parts of the main loop: the whole epilogue of a tile that a cluster shares.  smem: the ring.
template <int TW, int EPI>
OGB_DEVICE void rows_finish_cluster(const RowsGemmParams& p, const ActArgs& act, uint32_t tmem_base, int acc_cols, uint64_t* tmem_full,
                                    volatile int* abort_flag, uint8_t* smem, int ring_bytes) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  float* stage = reinterpret_cast<float*>(smem);
  bool ok = true;
  pdl_wait();
  if (warp >= 2 && warp < 6) {
    ok = __all_sync(0xffffffffu, mbar_wait(&tmem_full[0], 0));      // every product has retired: the ring is free
    if (!ok && lane == 0) { atomicOr(p.status, kStatusWaitTimeout); *abort_flag = 1; }
    tc_fence_after();
  }
  const int most = ring_bytes / (TW * 512) / 32 * 32;
  for (int r0 = 0; r0 < p.M; r0 += most) {
    const int count = min(most, (p.M - r0 + 31) / 32 * 32);
    if (warp >= 2 && warp < 6 && ok) rows_lay_out<TW>(tmem_base, acc_cols, r0, count, stage);
    if (p.splits > 1) cooperative_groups::this_cluster().sync();
    else __syncthreads();
    rows_sum_cluster<TW, EPI>(p, act, blockIdx.x / p.splits, blockIdx.x % p.splits, r0, count, stage);
    // nobody overwrites or leaves what is being read
    if (p.splits > 1) cooperative_groups::this_cluster().sync();
    else __syncthreads();
  }
}

// The MMA issuer (one lane): every stage holds TW tiles of 128 rows of W and then the activation tile.  False: a wait ran out.
template <int TW>
OGB_DEVICE bool rows_issue_mma(const RowsGemmParams& p, uint8_t* smem, int stage_bytes, uint32_t tmem_base, int bufs, int acc_cols, uint64_t* full_bar,
                               uint64_t* empty_bar, uint64_t* tmem_full, uint64_t* tmem_empty) {
  const uint32_t idesc = make_idesc_bf16(128, p.mn);
  int stage = 0;
  uint32_t phase = 0;
  RowsSegs segs(p);
  int tile, kb0, kb1;
  for (int seg = 0; segs.next(tile, kb0, kb1); ++seg) {
    const int buf = bufs == 2 ? (seg & 1) : 0;
    const uint32_t buf_phase = (bufs == 2 ? seg >> 1 : seg) & 1;
    if (!mbar_wait(&tmem_empty[buf], buf_phase ^ 1)) return false;
    tc_fence_after();
    const uint32_t d_addr = tmem_base + buf * TW * acc_cols;
    for (int kb = kb0; kb < kb1; ++kb) {
      if (!mbar_wait(&full_bar[stage], phase)) return false;
      tc_fence_after();
      const uint32_t sw = smem_u32(smem + stage * stage_bytes);
      const uint64_t db = make_kmajor_sw128_desc(sw + TW * 128 * kBK * 2);
#pragma unroll
      for (int w = 0; w < TW; ++w) {
        const uint64_t da = make_kmajor_sw128_desc(sw + w * 128 * kBK * 2);
#pragma unroll
        for (int k = 0; k < kBK / 16; ++k) umma_f16(d_addr + w * acc_cols, da + 2 * k, db + 2 * k, idesc, (kb > kb0 || k > 0) ? 1u : 0u);
      }
      umma_commit(&empty_bar[stage]);
      if (++stage == p.stages) { stage = 0; phase ^= 1; }
    }
    umma_commit(&tmem_full[buf]);
  }
  return true;
}

struct RowsBars {
  uint64_t full[kRowsMaxStages], empty[kRowsMaxStages], tmem_full[2], tmem_empty[2];
  uint32_t tmem_slot, shared_last;
  int abort_flag;
};
static_assert(sizeof(RowsBars) <= kRowsBarBytes, "barriers");

// Barriers and TMEM of a block; full_arrivals: what completes a stage besides its bytes.  Returns the TMEM address.
OGB_DEVICE uint32_t rows_setup(RowsBars* bars, int stages, uint32_t full_arrivals, uint32_t tmem_cols) {
  if (threadIdx.x == 0) {
    for (int i = 0; i < stages; ++i) {
      mbar_init(&bars->full[i], full_arrivals);
      mbar_init(&bars->empty[i], 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(&bars->tmem_full[i], 1);
      mbar_init(&bars->tmem_empty[i], 4);
    }
    bars->abort_flag = 0;
    mbar_fence_init();
  }
  if ((threadIdx.x >> 5) == 1) {
    tmem_alloc(&bars->tmem_slot, tmem_cols);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  return bars->tmem_slot;
}
OGB_DEVICE void rows_teardown(RowsBars* bars, uint32_t tmem_base, uint32_t tmem_cols) {
  tc_fence_before();
  __syncthreads();
  if (*reinterpret_cast<volatile int*>(&bars->abort_flag) != 0 && threadIdx.x == 0) {
    // A wait ran out: give copies that may still be in flight a bounded time to land.
    const uint64_t t0 = global_timer_ns();
    while (global_timer_ns() - t0 < 200000ull) { __nanosleep(1000); }
  }
  __syncthreads();
  if ((threadIdx.x >> 5) == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, tmem_cols);
  }
}
// TMEM of a launch: ranges keep two accumulator sets where they fit, a cluster's tile needs one.
template <int TW>
OGB_DEVICE void rows_tmem(const RowsGemmParams& p, int& acc_cols, int& bufs, uint32_t& cols) {
  acc_cols = (p.mn + 31) / 32 * 32;                           // the reads take 32 columns at a time
  bufs = p.splits == 0 && 2 * TW * acc_cols <= 512 ? 2 : 1;
  cols = 32;
  while (static_cast<int>(cols) < bufs * TW * acc_cols) cols *= 2;
}

template <int TW, int EPI>
__global__ void __launch_bounds__(kRowsThreads, 1)
gemm_rows_kernel(const __grid_constant__ CUtensorMap tmap_w, const __grid_constant__ CUtensorMap tmap_a, const RowsGemmParams p, const ActArgs act) {
  extern __shared__ __align__(1024) uint8_t smem[];
  constexpr int kStageW = TW * 128 * kBK * 2;
  const int stage_bytes = kStageW + p.mn * kBK * 2;
  const int ring_bytes = p.stages * stage_bytes;
  RowsBars* bars = reinterpret_cast<RowsBars*>(smem + ring_bytes);
  float* staging = reinterpret_cast<float*>(smem + ring_bytes + kRowsBarBytes);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  int acc_cols, bufs;
  uint32_t tmem_cols;
  rows_tmem<TW>(p, acc_cols, bufs, tmem_cols);
  if (threadIdx.x == 0) {
    tma_prefetch_desc(&tmap_w);
    tma_prefetch_desc(&tmap_a);
  }
  const uint32_t tmem_base = rows_setup(bars, p.stages, 1, tmem_cols);
  pdl_trigger();

  if (warp == 0) {
    // ------------------------------ TMA producer ------------------------------
    if (lane == 0) {
      int stage = 0;
      uint32_t phase = 0;
      bool ok = true;
      auto load_w = [&](const RowsCursor& c, int st) {
        mbar_expect_tx(&bars->full[st], stage_bytes);
#pragma unroll
        for (int w = 0; w < TW; ++w)
          tma_load_2d(smem + st * stage_bytes + w * 128 * kBK * 2, &tmap_w, &bars->full[st], c.kb * kBK, (c.tile * TW + w) * 128);
      };
      // the first ring of W is on its way before the kernel ahead has ended; its activations follow
      int ahead = 0;
      for (RowsCursor c(p); c.more && ahead < p.stages; c.step()) load_w(c, ahead++);
      pdl_wait();
      for (RowsCursor c(p); c.more; c.step()) {
        if (ahead > 0) {
          --ahead;
        } else {
          if (!mbar_wait(&bars->empty[stage], phase ^ 1)) { ok = false; break; }
          load_w(c, stage);
        }
        tma_load_2d(smem + stage * stage_bytes + kStageW, &tmap_a, &bars->full[stage], c.kb * kBK, 0);
        if (++stage == p.stages) { stage = 0; phase ^= 1; }
      }
      if (!ok) { atomicOr(p.status, kStatusWaitTimeout); bars->abort_flag = 1; }
    }
    __syncwarp();
  } else if (warp == 1) {
    // ------------------------------ MMA issuer ------------------------------
    if (lane == 0 && !rows_issue_mma<TW>(p, smem, stage_bytes, tmem_base, bufs, acc_cols, bars->full, bars->empty, bars->tmem_full, bars->tmem_empty)) {
      atomicOr(p.status, kStatusWaitTimeout);
      bars->abort_flag = 1;
    }
    __syncwarp();
  } else if (p.splits == 0) {
    rows_epilogue<TW, EPI>(p, act, tmem_base, bufs, acc_cols, bars->tmem_full, bars->tmem_empty, &bars->abort_flag, staging, &bars->shared_last);
  }
  if (p.splits > 0) rows_finish_cluster<TW, EPI>(p, act, tmem_base, acc_cols, bars->tmem_full, &bars->abort_flag, smem, ring_bytes);
  rows_teardown(bars, tmem_base, tmem_cols);
}

}  // namespace ogb
