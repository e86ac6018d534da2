// Per-tensor symmetric int8 quantisation on the device: the step the reference project performs on
// the host before the attention call (abs_max + float_quant2_int8, inc/utils.hpp:23-39, driven by
// test_fmha_i8.cpp:95-110).  The scale is known only when every element has been seen, so the tensor is needed twice;
// ONE launch does both passes and keeps as much of it on the chip in between as fits:
//   quant_cluster_kernel  up to 524,288 elements: one cluster of 1..16 CTAs holds the whole tensor in registers, the
//                         CTAs exchange their maxima through distributed shared memory.  5 bytes moved per element.
//   quant_grid_kernel     larger: one CTA per SM (cooperative launch), every warp streams its tiles through a private
//                         ring of bulk copies.  At the end of pass 1 the ring still holds each warp's last tiles and its
//                         registers the first ones (53 MB over the chip); pass 2 takes those from there and walks the
//                         others from the last to the first, so that it meets what the L2 still has.
// Two launches over 65,536-element chunks, which these replace, took 16.5 us for 255,749 elements (four CTAs) and 107 us
// for 67,108,864; these take 5.5 and 90 us.  The large case is bound by DRAM: pass 1 reads all 268 MB from there, pass 2
// what neither the SMs (50 MB) nor the L2 kept.
#pragma once
#include <cooperative_groups.h>
#include <cuda_runtime.h>
#include <cstdint>
#include "fmha_fwd_sm100.cuh"
#include "ptx.cuh"
#include "../../include/fmha_i8_c.h"

namespace fmha {

__device__ __forceinline__ float abs_max4(float m, const float4& v) {
  return fmaxf(m, fmaxf(fmaxf(fabsf(v.x), fabsf(v.y)), fmaxf(fabsf(v.z), fabsf(v.w))));
}
__device__ __forceinline__ int quant_one(float v, float scale) {
  // float_quant2_int8: floorf(x*scale + 0.5) with the sum rounded once to float, clamp to +-127
  const float f = floorf(__fadd_rn(__fmul_rn(v, scale), 0.5f));
  return static_cast<int>(fminf(fmaxf(f, -127.f), 127.f));
}
__device__ __forceinline__ uint32_t quant_four(const float4& v, float scale) {
  return (static_cast<uint32_t>(quant_one(v.x, scale)) & 0xFFu) | ((static_cast<uint32_t>(quant_one(v.y, scale)) & 0xFFu) << 8) |
         ((static_cast<uint32_t>(quant_one(v.z, scale)) & 0xFFu) << 16) | (static_cast<uint32_t>(quant_one(v.w, scale)) << 24);
}
__device__ __forceinline__ float quant_scale(float amax) {
  return (amax > 0.f) ? __fdiv_rn(127.0f, amax) : 0.f;     // an all-zero tensor quantises to zeros
}
// Largest of a block's values; `scratch` holds one float per warp.
template <int kThreads>
__device__ __forceinline__ float block_max(float m, float* scratch) {
  // magnitudes are non-negative: they order like their bit patterns
  m = __uint_as_float(__reduce_max_sync(0xFFFFFFFFu, __float_as_uint(m)));
  if ((threadIdx.x & 31) == 0) scratch[threadIdx.x >> 5] = m;
  __syncthreads();
  m = (threadIdx.x & 31) < kThreads / 32 ? scratch[threadIdx.x & 31] : 0.f;
  return __uint_as_float(__reduce_max_sync(0xFFFFFFFFu, __float_as_uint(m)));
}

// ------------------------------------------------------------------------------------------ up to 524,288 elements
constexpr int kQuantClusterThreads = 1024;
constexpr int kQuantClusterVec = 8;            // float4 per thread, all loads in flight at once
constexpr int kQuantClusterMax = 16, kQuantClusterPortable = 8;
constexpr long long kQuantPerCta = 4LL * kQuantClusterThreads * kQuantClusterVec;    // 32,768 elements

// CTAs for n elements: two float4 per thread are enough to cover the latency of memory, more CTAs than that only make
// the exchange longer; beyond 8 CTAs (the portable cluster size) only what the registers of 8 cannot hold.
inline int quant_cluster_size(long long n) {
  int c = 1;
  while (c < kQuantClusterPortable && n > c * (kQuantPerCta / 4)) c *= 2;
  return n > kQuantClusterPortable * kQuantPerCta ? kQuantClusterMax : c;
}

__global__ void __launch_bounds__(kQuantClusterThreads, 1)
quant_cluster_kernel(const float* x, int n, int8_t* out, float* amax_out) {
  __shared__ float warp_max[kQuantClusterThreads / 32];
  __shared__ float cta_max[kQuantClusterMax];
  grid_launch_dependents();
  const uint32_t ctas = cluster_ctas(), rank = cluster_rank();
  cluster_arrive();                                   // every CTA of the cluster runs before its memory is written
  grid_dependency_wait();
  const int n4 = n / 4, per_cta = (n4 + static_cast<int>(ctas) - 1) / static_cast<int>(ctas);
  const int begin = static_cast<int>(rank) * per_cta, end = min(begin + per_cta, n4);
  const float4* x4 = reinterpret_cast<const float4*>(x);
  float4 v[kQuantClusterVec];
#pragma unroll
  for (int k = 0; k < kQuantClusterVec; ++k) {
    const int i = begin + k * kQuantClusterThreads + static_cast<int>(threadIdx.x);
    v[k] = i < end ? x4[i] : make_float4(0.f, 0.f, 0.f, 0.f);
  }
  // up to three elements behind the last float4
  const int tail = n4 * 4 + static_cast<int>(threadIdx.x);
  const bool has_tail = rank == 0 && tail < n;
  const float t = has_tail ? x[tail] : 0.f;
  float m = fabsf(t);
#pragma unroll
  for (int k = 0; k < kQuantClusterVec; ++k) m = abs_max4(m, v[k]);
  m = block_max<kQuantClusterThreads>(m, warp_max);
  cluster_wait();
  if (threadIdx.x < ctas) st_cluster_f32(smem_u32(&cta_max[rank]), threadIdx.x, m);
  cluster_arrive();
  cluster_wait();
  float amax = 0.f;
  for (uint32_t i = 0; i < ctas; ++i) amax = fmaxf(amax, cta_max[i]);
  if (rank == 0 && threadIdx.x == 0 && amax_out) *amax_out = amax;
  const float scale = quant_scale(amax);
  uint32_t* o4 = reinterpret_cast<uint32_t*>(out);
#pragma unroll
  for (int k = 0; k < kQuantClusterVec; ++k) {
    const int i = begin + k * kQuantClusterThreads + static_cast<int>(threadIdx.x);
    if (i < end) o4[i] = quant_four(v[k], scale);
  }
  if (has_tail) out[tail] = static_cast<int8_t>(quant_one(t, scale));
}

// ------------------------------------------------------------------------------------------ larger tensors
constexpr int kQuantThreads = 256;
constexpr int kQuantWarps = kQuantThreads / 32;
constexpr int kQuantTile = 1024;               // elements per tile: 8 float4 per lane
constexpr int kQuantVec = kQuantTile / 128;
constexpr int kQuantStages = 7;                // ring of 7 x 4 KB per warp: all of shared memory
constexpr int kQuantKeep = 4;                  // tiles a warp keeps in registers (128 of them)
constexpr long long kQuantHoldBytes = 50000000;
constexpr size_t kQuantGridSmem = static_cast<size_t>(kQuantWarps) * kQuantStages * kQuantTile * sizeof(float);

// What the CTAs of one call exchange, their maxima, lies in the call's own output until the result goes there: nothing is shared with
// another call, however many are in flight and whether they are captured or not.  The first 4 bytes x CTAs of a CTA's first tile are its
// copy of the list; every CTA writes its entry into all copies, and reads and later overwrites only its own.
constexpr int kQuantMaxCtas = kQuantTile / 4;  // the list fits into a tile of output
static_assert(kQuantMaxCtas <= kQuantThreads, "one thread per entry");

__global__ void __launch_bounds__(kQuantThreads, 1)
quant_grid_kernel(const float* __restrict__ x, long long n, int8_t* __restrict__ out, float* __restrict__ amax_out, unsigned* __restrict__ status) {
  extern __shared__ __align__(128) uint8_t ring_raw[];
  __shared__ uint64_t bars[kQuantWarps][kQuantStages];
  __shared__ float warp_max[kQuantWarps];
  __shared__ int s_abort;
  const int lane = threadIdx.x & 31, warp = warp_index();
  float* ring = reinterpret_cast<float*>(ring_raw) + warp * (kQuantStages * kQuantTile);
  uint64_t* bar = bars[warp];

  // warp w of CTA c takes tiles w * CTAs + c, then every (warps * CTAs)-th: the whole chip reads one stretch of memory
  // at a time, and the last stretch is the one that pass 2 begins with
  const int n_tiles = static_cast<int>(n / kQuantTile);
  const int stride = static_cast<int>(gridDim.x) * kQuantWarps, first = warp * static_cast<int>(gridDim.x) + static_cast<int>(blockIdx.x);
  const int mine = first < n_tiles ? (n_tiles - first + stride - 1) / stride : 0;
  auto tile_at = [&](int i) { return (static_cast<long long>(first) + static_cast<long long>(i) * stride) * kQuantTile; };

  if (threadIdx.x == 0) s_abort = 0;
  if (lane == 0) {
    for (int s = 0; s < kQuantStages; ++s) mbar_init(smem_u32(&bar[s]), 1);
    mbar_init_fence();
  }
  __syncthreads();
  volatile int* abort_flag = &s_abort;
  // The L2 is asked to hold on to the stretch that pass 2 meets first and to nothing else: what pass 2 reads or writes is
  // not used again.  67,108,864 elements: 94.7 us with nothing held, 91.9 with 40 MB, 89.4 with 49, 89.3 with 52 or 58, 90.1 with
  // 70 (the L2 is two halves, and what is read from the other half takes room in both); 33,554,432: 45.2, 46.4, 47.1, 47.1, 47.2, 47.6.
  const uint64_t evict_first = l2_evict_first(), evict_last = l2_evict_last();
  const int hold_from = mine - kQuantStages - static_cast<int>(kQuantHoldBytes / (static_cast<long long>(kQuantTile) * 4 * stride));
  auto load = [&](int i, int s, bool first_pass) {
    mbar_arrive_expect_tx(smem_u32(&bar[s]), kQuantTile * sizeof(float));
    bulk_load(smem_u32(ring + s * kQuantTile), x + tile_at(i), kQuantTile * sizeof(float), smem_u32(&bar[s]),
              first_pass && i >= hold_from ? evict_last : evict_first);
  };
  bool ok = true;
  uint32_t parity_bits = 0u;                   // bit s: parity of the next completion of ring slot s
  auto landed = [&](int s) {
    ok = ok && __all_sync(0xFFFFFFFFu, mbar_wait(smem_u32(&bar[s]), (parity_bits >> s) & 1u, abort_flag));
    parity_bits ^= 1u << s;
    return reinterpret_cast<const float4*>(ring + s * kQuantTile);
  };

  // ---- pass 1: the largest magnitude
  if (lane == 0)
    for (int i = 0; i < kQuantStages && i < mine; ++i) load(i, i, true);
  float m = 0.f;
  float4 keep[kQuantKeep][kQuantVec];
#pragma unroll
  for (int i = 0; i < kQuantKeep; ++i) {
#pragma unroll
    for (int k = 0; k < kQuantVec; ++k) keep[i][k] = make_float4(0.f, 0.f, 0.f, 0.f);
    if (i < mine) {
      const float4* t = landed(i);
#pragma unroll
      for (int k = 0; k < kQuantVec; ++k) {
        keep[i][k] = t[lane + 32 * k];
        m = abs_max4(m, keep[i][k]);
      }
      __syncwarp();
      if (lane == 0 && i + kQuantStages < mine) load(i + kQuantStages, i, true);
    }
  }
  for (int i = kQuantKeep, s = kQuantKeep; i < mine; ++i) {
    const float4* t = landed(s);
#pragma unroll
    for (int k = 0; k < kQuantVec; ++k) m = abs_max4(m, t[lane + 32 * k]);
    __syncwarp();
    if (lane == 0 && i + kQuantStages < mine) load(i + kQuantStages, s, true);
    if (++s == kQuantStages) s = 0;
  }
  // what is left behind the last whole tile: the last CTA reads it, twice
  const long long rest = static_cast<long long>(n_tiles) * kQuantTile;
  const bool has_rest = blockIdx.x == gridDim.x - 1;
  if (has_rest)
    for (long long i = rest + threadIdx.x; i < n; i += kQuantThreads) m = fmaxf(m, fabsf(x[i]));

  // ---- the largest of all CTAs.  The grid's barrier is the one of the cooperative launch, whose CTAs are all resident and all come
  // here: no wait above is longer than its limit.
  m = block_max<kQuantThreads>(m, warp_max);
  const int ctas = static_cast<int>(gridDim.x), t = static_cast<int>(threadIdx.x);
  if (t < ctas) __stcg(reinterpret_cast<float*>(out + static_cast<long long>(t) * kQuantTile) + blockIdx.x, m);
  cooperative_groups::this_grid().sync();
  m = t < ctas ? __ldcg(reinterpret_cast<const float*>(out + static_cast<long long>(blockIdx.x) * kQuantTile) + t) : 0.f;
  const float amax = block_max<kQuantThreads>(m, warp_max);      // (its barrier: the list has been read before the tile is written)
  if (blockIdx.x == 0 && t == 0 && amax_out) *amax_out = amax;
  const float scale = quant_scale(amax);

  // ---- pass 2: quantise, from the last tile to the first
  auto store = [&](int i, int k, const float4& v) { __stcs(reinterpret_cast<uint32_t*>(out + tile_at(i)) + lane + 32 * k, quant_four(v, scale)); };
  auto from_ring = [&](int i, int s, const float4* t) {
#pragma unroll
    for (int k = 0; k < kQuantVec; ++k) store(i, k, t[lane + 32 * k]);
    __syncwarp();
    if (lane == 0 && i - kQuantStages >= kQuantKeep) load(i - kQuantStages, s, false);
  };
  const int still_there = max(mine - kQuantStages, kQuantKeep);    // tiles [still_there, mine) are still in the ring
  for (int i = mine - 1; i >= still_there; --i) {
    const int s = i % kQuantStages;
    from_ring(i, s, reinterpret_cast<const float4*>(ring + s * kQuantTile));
  }
#pragma unroll
  for (int i = 0; i < kQuantKeep; ++i)
    if (i < mine) {
#pragma unroll
      for (int k = 0; k < kQuantVec; ++k) store(i, k, keep[i][k]);
    }
  for (int i = still_there - 1; i >= kQuantKeep; --i) {
    const int s = i % kQuantStages;
    from_ring(i, s, landed(s));
  }
  if (has_rest)
    for (long long i = rest + threadIdx.x; i < n; i += kQuantThreads) out[i] = static_cast<int8_t>(quant_one(x[i], scale));
  if (!ok && lane == 0) {
    raise_status(abort_flag, status, FMHA_I8_DEV_WAIT_QUANT, blockIdx.x);
    const long long t0 = clock64();
    while (clock64() - t0 < 2000000LL) { /* copies still in flight land before the CTA may exit */ }
  }
}

}  // namespace fmha
