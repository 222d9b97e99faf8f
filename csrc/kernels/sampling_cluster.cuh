// The fused sampler with a row spread over a cluster: eight CTAs keep a row's bf16 logits in their shared memory, so the row crosses
// HBM once and every later pass reads it on chip.  Same integer weights, thresholds and draw as sample_kernel (sampling.cu).
//
// What bounded the one-CTA kernels was their own traffic: 32-bit weights written to memory (608 KB per row of 152 k logits, more
// than L2 for 256 rows) and read again by five radix passes per filter, 1024 threads at a time.  Here a weight is recomputed from
// its logit where it is needed, and a threshold takes one histogram: 1024 buckets of the logit's distance from the maximum (a
// weight's logarithm, so buckets hold similar shares of ordinary rows), kept as two 32-bit sums of the weights' low 16 and high
// bits; the many weights below 2^16 of 2^30 are only summed.  The bucket in which the target falls holds a few hundred logits as a rule; they are listed and the threshold
// is picked among them exactly.  A bucket with more than fit the list (equal or nearly equal logits) is cut again, by weight, until
// they fit or are all equal: each cut narrows the range of 30-bit weights a thousandfold.
// 256 rows of 152064 (temperature, top-k, top-p and min-p mixed): 665 -> 260 us; inside a decode step of 256 rows (top-p 0.9, sure of a
// few tokens) 292 -> 152, of 40 rows 194 -> 32.  What is left is a CTA's chain of passes and cluster barriers, seven times per SM.
#pragma once
#include <cooperative_groups.h>

#include "common.cuh"

namespace ogb {

constexpr int kClCtas = 8;                   // the portable cluster size
constexpr int kClThreads = 512;
constexpr int kClWarps = kClThreads / 32;
constexpr int kClBuckets = 1024;
constexpr int kClList = 1024;
constexpr int kClMaxCuts = 3;                // a cut leaves a 1024th of the range of weights: 2^30 values, 2^20, 2^10, 1
constexpr uint32_t kClLow = 1u << 16;        // smaller weights are summed, and looked at one by one only where a threshold falls among them
constexpr int kClMaxSlice = 65536;           // logits per CTA: 2^16 low halves of weights still sum below 2^32

struct ClShared {
  uint32_t cnt[kClBuckets], lo[kClBuckets], hi[kClBuckets];      // this CTA's share of the row
  uint32_t row_cnt[kClBuckets];                                  // the row's
  unsigned long long row_mass[kClBuckets];
  uint32_t list[kClList], cand[kClList];
  float high[kClWarps], low[kClWarps];
  unsigned long long sums[kClWarps], scan[kClWarps];             // cl_block_sum's; find's, written while a slower warp may still read the other
  // one slot per exchange with the other CTAs that can be under way while a slower CTA still reads the last one
  float best, lowest;
  int first;
  uint32_t n, w_min, w_max, thr;
  uint32_t rest_cnt;
  unsigned long long rest_mass, mass[2], above;
  int bucket;
};

OGB_DEVICE __nv_bfloat162 as_bf162(uint32_t u) { return *reinterpret_cast<__nv_bfloat162*>(&u); }
OGB_DEVICE unsigned long long cl_block_sum(unsigned long long v, unsigned long long* sh) {
  v = warp_sum_u64(v);
  __syncthreads();
  if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = v;
  __syncthreads();
  unsigned long long r = 0;
#pragma unroll
  for (int i = 0; i < kClWarps; ++i) r += sh[i];
  return r;
}

__global__ void __cluster_dims__(kClCtas, 1, 1) __launch_bounds__(kClThreads, 2)
sample_cluster_kernel(const __nv_bfloat16* __restrict__ logits, int* __restrict__ out, const float* __restrict__ temperature,
                      const int* __restrict__ top_k, const float* __restrict__ top_p, const float* __restrict__ min_p,
                      const float* __restrict__ uniform, int vocab, int ld, int slice) {
  namespace cg = cooperative_groups;
  extern __shared__ __align__(16) uint8_t cl_smem[];
  ClShared& sh = *reinterpret_cast<ClShared*>(cl_smem);
  uint4* row_sh = reinterpret_cast<uint4*>(cl_smem + (sizeof(ClShared) + 15) / 16 * 16);
  const cg::cluster_group cluster = cg::this_cluster();
  const int rank = static_cast<int>(cluster.block_rank());
  const int rowi = blockIdx.x / kClCtas;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int begin = rank * slice;                                  // slice and vocab are multiples of 8
  const int nvec = max(0, min(vocab, begin + slice) - begin) / 8;
  const uint4* src = reinterpret_cast<const uint4*>(logits + static_cast<size_t>(rowi) * ld + begin);
  auto peer = [&](int r) -> const ClShared& { return *cluster.map_shared_rank(&sh, r); };

  // ---- the row comes in; its largest and its smallest logit, two values at a time ----
  const __nv_bfloat162 ninf = as_bf162(0xff80ff80u), pinf = as_bf162(0x7f807f80u);
  __nv_bfloat162 hi2 = ninf, lo2 = pinf;                           // a NaN never replaces a number
  for (int vi = tid; vi < nvec; vi += kClThreads) {
    const uint4 q = __ldcs(src + vi);
    row_sh[vi] = q;
    hi2 = __hmax2(hi2, __hmax2(__hmax2(as_bf162(q.x), as_bf162(q.y)), __hmax2(as_bf162(q.z), as_bf162(q.w))));
    lo2 = __hmin2(lo2, __hmin2(__hmin2(as_bf162(q.x), as_bf162(q.y)), __hmin2(as_bf162(q.z), as_bf162(q.w))));
  }
  float best = warp_max(fmaxf(__low2float(hi2), __high2float(hi2)));
  float low = -warp_max(-fminf(__low2float(lo2), __high2float(lo2)));
  if (lane == 0) { sh.high[warp] = best; sh.low[warp] = low; }
  __syncthreads();
  if (warp == 0) {
    best = warp_max(sh.high[lane & (kClWarps - 1)]);
    low = -warp_max(-sh.low[lane & (kClWarps - 1)]);
    if (lane == 0) { sh.best = best; sh.lowest = low; sh.first = 0x7fffffff; }
  }
  cluster.sync();
  for (int r = 0; r < kClCtas; ++r) {
    best = r == 0 ? peer(0).best : fmaxf(best, peer(r).best);
    low = r == 0 ? peer(0).lowest : fminf(low, peer(r).lowest);
  }
  // the lowest token with the largest logit; 0 where there is none above -inf
  auto take_largest = [&]() {
    int at = 0x7fffffff;
    for (int vi = tid; vi < nvec; vi += kClThreads) {
      const uint4 q = row_sh[vi];
      const uint32_t ws[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
      for (int e = 3; e >= 0; --e) {
        const float2 f = unpack_bf16(ws[e]);
        if (f.y == best) at = min(at, begin + vi * 8 + 2 * e + 1);
        if (f.x == best) at = min(at, begin + vi * 8 + 2 * e);
      }
    }
    at = __reduce_min_sync(0xffffffffu, at);
    if (lane == 0) atomicMin(&sh.first, at);
    cluster.sync();
    if (rank == 0 && tid == 0) {
      for (int r = 0; r < kClCtas; ++r) at = min(at, peer(r).first);
      out[rowi] = best > -INFINITY ? at : 0;
    }
    cluster.sync();                                                // nobody leaves while its shared memory is being read
  };
  const float temp = temperature[rowi];
  const float inv_t = 1.f / temp;
  if (!(temp > 0.f) || !(best > -INFINITY)) {
    take_largest();
    return;
  }
  // Weights of at least kClLow (the largest 2^14-fold) are told apart by distance: ln 2^14 = 9.704.
  const float range = fminf(9.75f, (best - low) * inv_t);
  const float scale = range > 1e-6f ? kClBuckets / range : 0.f;
  auto weight = [&](float l) -> uint32_t {                         // 0 (a NaN's too): the token cannot be drawn
    return min(__float2uint_rz(__expf((l - best) * inv_t) * 1073741824.f + 0.5f), 1073741823u);
  };
  auto bucket_of = [&](float l) { return min(kClBuckets - 1, static_cast<int>((best - l) * inv_t * scale)); };
  float l_from = best - 21.6f / inv_t;                             // weights below 2^-31 of the largest round to zero
  l_from -= fabsf(l_from) * 1e-6f;
  // f(weight, logit, index) of a vector's logits in [from, to] that can be drawn; a vector without one costs its maximum only
  auto each = [&](int vi, float from, float to, auto&& f) {
    const uint4 q = row_sh[vi];
    const uint32_t ws[4] = {q.x, q.y, q.z, q.w};
    const __nv_bfloat162 m = __hmax2(__hmax2(as_bf162(q.x), as_bf162(q.y)), __hmax2(as_bf162(q.z), as_bf162(q.w)));
    if (!(fmaxf(__low2float(m), __high2float(m)) >= from)) return;
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const float2 p = unpack_bf16(ws[e]);
      if (p.x >= from && p.x <= to) {
        const uint32_t w = weight(p.x);
        if (w != 0) f(w, p.x, 2 * e);
      }
      if (p.y >= from && p.y <= to) {
        const uint32_t w = weight(p.y);
        if (w != 0) f(w, p.y, 2 * e + 1);
      }
    }
  };
  const int k = top_k[rowi];
  const bool use_k = k > 0 && k < vocab;
  const float p = top_p[rowi];
  const bool use_p = p > 0.f && p < 1.f;

  // ---- histograms: clear, count (one of the two below), sum over the cluster ----
  uint32_t rest_cnt;
  unsigned long long rest_mass;
  auto clear = [&]() {
    for (int i = tid; i < kClBuckets; i += kClThreads) sh.cnt[i] = sh.lo[i] = sh.hi[i] = 0u;
    __syncthreads();
  };
  auto count = [&](uint32_t w, int b) {
    atomicAdd(&sh.lo[b], w & 0xffffu);
    if (w >> 16) atomicAdd(&sh.hi[b], w >> 16);
    if (use_k) atomicAdd(&sh.cnt[b], 1u);
  };
  auto sum_up = [&](uint32_t out_cnt, unsigned long long out_mass) {
    out_mass = cl_block_sum(out_mass, sh.sums);
    const unsigned long long oc = use_k ? cl_block_sum(out_cnt, sh.sums) : 0ull;
    if (tid == 0) { sh.rest_mass = out_mass; sh.rest_cnt = static_cast<uint32_t>(oc); }
    cluster.sync();
    // every CTA sums an eighth of the buckets over the cluster and hands the sums to all: four threads to a bucket, two CTAs each
    constexpr int kShare = kClBuckets / kClCtas;
    static_assert(kShare * 4 == kClThreads, "four threads per bucket");
    const int b = rank * kShare + tid / 4, r0 = (tid & 3) * 2;
    const ClShared &s0 = peer(r0), &s1 = peer(r0 + 1);
    uint32_t c = s0.cnt[b] + s1.cnt[b];
    unsigned long long m = static_cast<unsigned long long>(s0.lo[b]) + s1.lo[b] + ((static_cast<unsigned long long>(s0.hi[b]) + s1.hi[b]) << 16);
#pragma unroll
    for (int o = 1; o < 4; o <<= 1) {
      c += __shfl_xor_sync(0xffffffffu, c, o);
      m += __shfl_xor_sync(0xffffffffu, m, o);
    }
    for (int r = r0; r < r0 + 2; ++r) {
      ClShared* d = cluster.map_shared_rank(&sh, r);
      d->row_cnt[b] = c;
      d->row_mass[b] = m;
    }
    rest_cnt = 0;
    rest_mass = 0;
    for (int r = 0; r < kClCtas; ++r) {
      rest_cnt += peer(r).rest_cnt;
      rest_mass += peer(r).rest_mass;
    }
    cluster.sync();
  };
  // The first bucket in which `above` plus the measure of all buckets up to it reaches the target; -1: none.  sh.above: what lies before it.
  auto find = [&](bool by_mass, unsigned long long above, unsigned long long target) -> int {
    const unsigned long long a = by_mass ? sh.row_mass[2 * tid] : sh.row_cnt[2 * tid], b = by_mass ? sh.row_mass[2 * tid + 1] : sh.row_cnt[2 * tid + 1];
    unsigned long long incl = a + b;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const unsigned long long n = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += n;
    }
    if (tid == 0) sh.bucket = -1;
    if (lane == 31) sh.scan[warp] = incl;
    __syncthreads();
    unsigned long long run = above + incl - a - b;
    for (int i = 0; i < warp; ++i) run += sh.scan[i];
    if (run < target && run + a >= target) { sh.bucket = 2 * tid; sh.above = run; }
    run += a;
    if (run < target && run + b >= target) { sh.bucket = 2 * tid + 1; sh.above = run; }
    __syncthreads();
    const int r = sh.bucket;
    return r;
  };

  bool row_known = false;                                          // the histogram is that of the distances
  auto by_distance = [&]() {
    if (row_known) return;
    row_known = true;
    clear();
    uint32_t out_cnt = 0, out_mass = 0;                            // a thread has at most 128 weights below 2^16
    for (int vi = tid; vi < nvec; vi += kClThreads) {
      const uint4 q = row_sh[vi];
      const uint32_t ws[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        const float2 p = unpack_bf16(ws[e / 2]);
        const float l = (e & 1) ? p.y : p.x;
        const uint32_t w = weight(l);
        if (w >= kClLow) {
          count(w, bucket_of(l));
        } else {
          out_mass += w;
          if (use_k) out_cnt += w != 0;
        }
      }
    }
    sum_up(out_cnt, out_mass);
  };
  // No survivor has a logit below it.  The margin covers the roundings of bucket_of.
  auto bucket_from = [&](int bucket) {
    const float d = (bucket + 1) / (scale * inv_t);
    return best - d - (d + fabsf(best)) * 1e-5f;
  };
  // The largest threshold T with measure(w >= T) >= target among weights of at least `floor_w`; floor_w when there is none.
  auto select = [&](bool by_mass, unsigned long long target, uint32_t floor_w) -> uint32_t {
    by_distance();
    int bucket = find(by_mass, 0, target);
    unsigned long long above;
    uint32_t from = floor_w, to = 0xffffffffu;
    float l_lo = l_from, l_hi = INFINITY;
    if (bucket >= 0) {
      above = sh.above;
      if (scale * inv_t > 0.f) {
        l_lo = fmaxf(l_lo, bucket_from(bucket));
        const float d = bucket / (scale * inv_t);
        l_hi = best - d + (d + fabsf(best)) * 1e-5f;
        l_from = l_lo;
      }
      if (from < kClLow) from = kClLow;
    } else {
      // the target lies among the weights below kClLow, or nowhere
      above = cl_block_sum(by_mass ? sh.row_mass[2 * tid] + sh.row_mass[2 * tid + 1] : sh.row_cnt[2 * tid] + sh.row_cnt[2 * tid + 1], sh.sums);
      if (above + (by_mass ? rest_mass : rest_cnt) < target) return floor_w;
      to = kClLow - 1;
    }
    for (int cuts = 0; cuts <= kClMaxCuts; ++cuts) {
      if (tid == 0) { sh.n = 0; sh.w_min = 0xffffffffu; sh.w_max = 0u; sh.thr = 0u; }
      __syncthreads();
      for (int vi = tid; vi < nvec; vi += kClThreads)
        each(vi, l_lo, l_hi, [&](uint32_t w, float l, int) {
          if (w < from || w > to || (bucket >= 0 && bucket_of(l) != bucket)) return;
          const uint32_t at = atomicAdd(&sh.n, 1u);
          if (at < kClList) sh.list[at] = w;
          else { atomicMin(&sh.w_min, w); atomicMax(&sh.w_max, w); }
        });
      __syncthreads();
      for (int i = tid; i < min(static_cast<int>(sh.n), kClList); i += kClThreads) { atomicMin(&sh.w_min, sh.list[i]); atomicMax(&sh.w_max, sh.list[i]); }
      cluster.sync();
      uint32_t n = 0, w_min = 0xffffffffu, w_max = 0u;
      for (int r = 0; r < kClCtas; ++r) {
        n += peer(r).n;
        w_min = min(w_min, peer(r).w_min);
        w_max = max(w_max, peer(r).w_max);
      }
      if (n == 0) { cluster.sync(); return floor_w; }
      if (w_min == w_max) { cluster.sync(); return w_min; }
      if (n <= kClList) {
        uint32_t off = 0;
        for (int r = 0; r < kClCtas; ++r) {
          const uint32_t m = peer(r).n;
          for (uint32_t i = tid; i < m; i += kClThreads) sh.cand[off + i] = peer(r).list[i];
          off += m;
        }
        cluster.sync();                                            // also: the lists may be written again from here on
        // every eighth candidate is this CTA's; four threads share the sum of one
        uint32_t t = 0;
        for (uint32_t i0 = rank + kClCtas * warp * 8; i0 < n; i0 += kClCtas * kClWarps * 8) {
          const uint32_t i = i0 + kClCtas * (lane / 4);
          const uint32_t w = sh.cand[min(i, n - 1)];
          unsigned long long sum = 0;
          for (uint32_t j = tid & 3; j < n; j += 4) { const uint32_t v = sh.cand[j]; sum += v >= w ? (by_mass ? v : 1u) : 0u; }
          sum += __shfl_xor_sync(0xffffffffu, sum, 1);
          sum += __shfl_xor_sync(0xffffffffu, sum, 2);
          if (i < n && above + sum >= target) t = max(t, w);
        }
        if (t != 0) atomicMax(&sh.thr, t);
        cluster.sync();
        for (int r = 0; r < kClCtas; ++r) t = max(t, peer(r).thr);
        t = __reduce_max_sync(0xffffffffu, t);
        cluster.sync();
        return max(t, floor_w);
      }
      // too many for the list: cut [w_min, w_max] into buckets, largest weights first
      const unsigned long long width = static_cast<unsigned long long>(w_max - w_min) + 1;
      row_known = false;
      clear();
      for (int vi = tid; vi < nvec; vi += kClThreads)
        each(vi, l_lo, l_hi, [&](uint32_t w, float l, int) {
          if (w >= from && w <= to && (bucket < 0 || bucket_of(l) == bucket))
            count(w, static_cast<int>(kClBuckets - 1 - static_cast<unsigned long long>(w - w_min) * kClBuckets / width));
        });
      sum_up(0, 0);
      const int cut = find(by_mass, above, target);
      if (cut < 0) return floor_w;
      above = sh.above;
      const unsigned long long c = kClBuckets - 1 - cut;
      from = w_min + static_cast<uint32_t>((c * width + kClBuckets - 1) / kClBuckets);
      to = w_min + static_cast<uint32_t>(((c + 1) * width + kClBuckets - 1) / kClBuckets) - 1;
    }
    return from;                                                   // not reached: after kClMaxCuts one weight is left
  };
  // summed weight of this thread's tokens in vectors [v0, v1), v0 + step, ... with weights of at least thr
  auto mass_of = [&](int v0, int v1, int step, uint32_t thr) {
    unsigned long long s = 0;
    for (int vi = v0; vi < v1; vi += step) each(vi, l_from, INFINITY, [&](uint32_t w, float, int) { s += w >= thr ? w : 0u; });
    return s;
  };

  uint32_t thr = 1;                                                // zero-weight tokens never survive
  if (use_k) thr = select(false, static_cast<unsigned long long>(k), thr);
  if (use_p) {
    // smallest set of largest weights whose mass reaches p * total (mass renormalised over survivors)
    unsigned long long total;
    if (!use_k) {                                                  // all of the row
      by_distance();
      total = rest_mass + cl_block_sum(sh.row_mass[2 * tid] + sh.row_mass[2 * tid + 1], sh.sums);
    } else {
      const unsigned long long mine = cl_block_sum(mass_of(tid, nvec, kClThreads, thr), sh.sums);
      if (tid == 0) sh.mass[0] = mine;
      cluster.sync();
      total = 0;
      for (int r = 0; r < kClCtas; ++r) total += peer(r).mass[0];
    }
    unsigned long long target = static_cast<unsigned long long>(static_cast<double>(total) * static_cast<double>(p));
    if (target < 1ull) target = 1ull;
    thr = select(true, target, thr);
  }
  const float mp = min_p[rowi];
  if (mp > 0.f) {
    const uint32_t floor_mp = static_cast<uint32_t>(fminf(mp, 1.f) * 1073741824.f);
    if (floor_mp > thr) thr = floor_mp;
  }

  // ---- the draw, in token order: masses of the warps' neighbouring ranges, of the CTAs' slices, then a walk ----
  const int per_warp = (nvec + kClWarps - 1) / kClWarps;
  const int v0 = min(nvec, warp * per_warp), v1 = min(nvec, v0 + per_warp);
  const unsigned long long mine = warp_sum_u64(mass_of(v0 + lane, v1, 32, thr));
  __syncthreads();
  if (lane == 0) sh.sums[warp] = mine;
  __syncthreads();
  unsigned long long before = 0, cta = 0;
  for (int i = 0; i < kClWarps; ++i) {
    if (i < warp) before += sh.sums[i];
    cta += sh.sums[i];
  }
  if (tid == 0) sh.mass[1] = cta;
  cluster.sync();
  unsigned long long total = 0;
  for (int r = 0; r < kClCtas; ++r) {
    const unsigned long long m = peer(r).mass[1];
    if (r < rank) before += m;
    total += m;
  }
  float u = uniform[rowi];
  u = fminf(fmaxf(u, 0.f), 0.99999994f);
  unsigned long long target = static_cast<unsigned long long>(static_cast<double>(u) * static_cast<double>(total));
  if (total > 0 && target >= total) target = total - 1;
  if (total == 0) {
    take_largest();
    return;
  } else if (target >= before && target < before + mine) {
    unsigned long long run = before;
    for (int base = v0; base < v1; base += 32) {
      const int vi = base + lane;
      const unsigned long long own = vi < v1 ? mass_of(vi, vi + 1, 1, thr) : 0ull;
      unsigned long long incl = own;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const unsigned long long n = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += n;
      }
      const unsigned long long end = run + incl;
      const bool hit = own > 0 && target >= end - own && target < end;
      if (hit) {
        unsigned long long at = end - own;
        int pick = -1;
        each(vi, l_from, INFINITY, [&](uint32_t w, float, int e) {
          if (w < thr) return;
          if (pick < 0 && target < at + w) pick = begin + vi * 8 + e;
          at += w;
        });
        out[rowi] = pick;
      }
      if (__any_sync(0xffffffffu, hit)) break;
      run += __shfl_sync(0xffffffffu, incl, 31);
    }
  }
  cluster.sync();                                                  // nobody leaves while its shared memory is being read
}

// False: a row does not fit the cluster's shared memory, or is not made of aligned 16-byte vectors.
inline bool sample_cluster_applies(const void* logits, int vocab, int ld) {
  const int slice = ((vocab + kClCtas - 1) / kClCtas + 7) / 8 * 8;
  return vocab % 8 == 0 && ld % 8 == 0 && (reinterpret_cast<uintptr_t>(logits) & 15) == 0 && slice <= kClMaxSlice;
}

inline int launch_sample_cluster(const void* logits, int* out, const float* temperature, const int* top_k, const float* top_p, const float* min_p,
                                 const float* uniform, int rows, int vocab, int ld, cudaStream_t stream) {
  const int slice = ((vocab + kClCtas - 1) / kClCtas + 7) / 8 * 8;
  const int smem = static_cast<int>((sizeof(ClShared) + 15) / 16 * 16) + slice * 2;
  static OncePerDevice allowed;
  const int rc = allow_smem(allowed, sample_cluster_kernel, static_cast<int>((sizeof(ClShared) + 15) / 16 * 16) + kClMaxSlice * 2);
  if (rc != 0) return rc;
  sample_cluster_kernel<<<rows * kClCtas, kClThreads, smem, stream>>>(static_cast<const __nv_bfloat16*>(logits), out, temperature, top_k, top_p, min_p,
                                                                      uniform, vocab, ld, slice);
  return static_cast<int>(cudaGetLastError());
}

}  // namespace ogb
