// Per-tensor symmetric int8 quantisation on the device: the step the reference project performs on
// the host before the attention call (abs_max + float_quant2_int8, inc/utils.hpp:23-39, driven by
// test_fmha_i8.cpp:95-110).  The scale is known only when every element has been seen, so the tensor is needed twice;
// ONE launch does both passes and keeps as much of it on the chip in between as fits:
//   quant_cluster_kernel  up to 524,288 elements: one cluster of 1..16 CTAs holds the whole tensor in registers, the
//                         CTAs exchange their maxima through distributed shared memory.  5 bytes moved per element.
//   quant_grid_kernel     larger: one CTA per SM (cooperative launch), every warp streams its tiles through a private
//                         ring of bulk copies.  At the end of pass 1 the ring still holds each warp's last tiles, its
//                         registers the first ones and its part of tensor memory the next (97 MB over the chip); pass 2
//                         takes those from there and reads the others again, as far as it can from the L2.
// 255,749 elements take 4.1 us, 67,108,864 take 74 to 80: DRAM, since pass 1 reads all 268 MB from there and pass 2 what neither the SMs
// (97 MB) nor the L2 (some 50) kept, 121 MB.  Without tensor memory the latter take 7 % longer, 33,554,432 elements 6 %.
#pragma once
#include <cooperative_groups.h>
#include <cuda_runtime.h>
#include <cstdint>
#include "fmha_fwd_sm100.cuh"
#include "ptx.cuh"
#include "../../include/fmha_i8_c.h"

namespace fmha {

__device__ __forceinline__ float abs_max4(float m, const float4& v) { return max3_abs(max3_abs(m, v.x, v.y), v.z, v.w); }
__device__ __forceinline__ int quant_one(float v, float scale) {
  // float_quant2_int8: floorf(x*scale + 0.5) with the sum rounded once to float, clamp to +-127
  const float f = floorf(__fadd_rn(__fmul_rn(v, scale), 0.5f));
  return static_cast<int>(fminf(fmaxf(f, -127.f), 127.f));
}
// The same for N float4, a word of bytes each.  floorf and the conversion to an integer are instructions of the unit that also
// has the exponentials, 16 lanes a cycle on an SM; with them it, not memory, was what quantising waited for (67,108,864 elements: 29
// us of that unit; 89.5 -> 84.2 us in all, 33,554,432 elements 47.2 -> 37.7, 255,749 5.6 -> 4.2).  Here the floor comes from an addition to 1.5 * 2^23 that
// rounds down.  That needs x*scale + 0.5 to be a number in [-127, 128), which it is unless x is not a number or the scale is not
// finite: false is returned if it may not be, and the words are then quant_one's to make.
template <int N>
__device__ __forceinline__ bool quant_words(const float4 (&v)[N], float scale, uint32_t (&words)[N]) {
  const float2 s2 = make_float2(scale, scale), half = make_float2(0.5f, 0.5f), magic = make_float2(kMagic, kMagic);
  float most = 0.f;
#pragma unroll
  for (int i = 0; i < N; ++i) {
    const float2 y01 = __fadd2_rn(__fmul2_rn(make_float2(v[i].x, v[i].y), s2), half), y23 = __fadd2_rn(__fmul2_rn(make_float2(v[i].z, v[i].w), s2), half);
    most = max3_abs_nan(max3_abs_nan(most, y01.x, y01.y), y23.x, y23.y);
    const float2 n01 = __fadd2_rd(y01, magic), n23 = __fadd2_rd(y23, magic);
    words[i] = __byte_perm(__byte_perm(__float_as_uint(n01.x), __float_as_uint(n01.y), 0x0040),
                           __byte_perm(__float_as_uint(n23.x), __float_as_uint(n23.y), 0x0040), 0x5410);
  }
  return most < 127.75f;
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
  uint32_t words[kQuantClusterVec];
  if (!quant_words(v, scale, words)) {
#pragma unroll
    for (int k = 0; k < kQuantClusterVec; ++k) words[k] = quant_four(v[k], scale);
  }
#pragma unroll
  for (int k = 0; k < kQuantClusterVec; ++k) {
    const int i = begin + k * kQuantClusterThreads + static_cast<int>(threadIdx.x);
    if (i < end) o4[i] = words[k];
  }
  if (has_tail) out[tail] = static_cast<int8_t>(quant_one(t, scale));
}

// ------------------------------------------------------------------------------------------ larger tensors
constexpr int kQuantThreads = 256;
constexpr int kQuantWarps = kQuantThreads / 32;
constexpr int kQuantTile = 1024;               // elements per tile: 8 float4 per lane
constexpr int kQuantVec = kQuantTile / 128;
constexpr int kQuantStages = 7;                // ring of 7 x 4 KB per warp: all of shared memory
// Tiles a warp keeps in registers (32 each): its first.  231 of the 255 that a thread can have are in use then.  4 -> 5: 12,000,000 elements 16.1
// -> 15.7 us, 24,000,000 25.3 -> 25.0, 67,108,864 1 % or less (75.0 -> 74.2, on another box 79.3 -> 78.6); 6: 33,554,432 elements 32.7 -> 34.8.
constexpr int kQuantKeep = 5;
static_assert(kQuantKeep < kQuantStages, "the first tiles are taken from the slots of their first loads, and the next one from the slot behind");
constexpr int kQuantTmem = 8;                  // tiles a warp keeps in tensor memory, 32 columns each: the next
constexpr uint32_t kQuantTmemCols = 32 * kQuantTmem * kQuantWarps / 4;      // two warps to a lane quarter
static_assert(kQuantTmemCols <= 512, "tensor memory has 512 columns");
constexpr long long kQuantHoldBytes = 50000000;
constexpr size_t kQuantGridSmem = static_cast<size_t>(kQuantWarps) * kQuantStages * kQuantTile * sizeof(float);

// What the CTAs of one call exchange, their maxima, lies in the call's own output until the result goes there: nothing is shared with
// another call, however many are in flight and whether they are captured or not.  The first 4 bytes x CTAs of a CTA's first tile are its
// copy of the list; every CTA writes its entry into all copies, and reads and later overwrites only its own.
constexpr int kQuantMaxCtas = kQuantTile / 4;  // the list fits into a tile of output
static_assert(kQuantMaxCtas <= kQuantThreads, "one thread per entry");

// kTmem: some warp has more tiles than its registers and its ring hold (quant_needs_tmem).
inline bool quant_needs_tmem(long long n, int ctas) { return n / kQuantTile > static_cast<long long>(kQuantKeep + kQuantStages) * kQuantWarps * ctas; }
template <bool kTmem>
__global__ void __launch_bounds__(kQuantThreads, 1)
quant_grid_kernel(const float* __restrict__ x, long long n, int8_t* __restrict__ out, float* __restrict__ amax_out, unsigned* __restrict__ status) {
  extern __shared__ __align__(128) uint8_t ring_raw[];
  __shared__ uint64_t bars[kQuantWarps][kQuantStages];
  __shared__ float warp_max[kQuantWarps];
  __shared__ int s_abort;
  __shared__ uint32_t s_tmem;
  const int lane = threadIdx.x & 31, warp = warp_index();
  float* ring = reinterpret_cast<float*>(ring_raw) + warp * (kQuantStages * kQuantTile);
  uint64_t* bar = bars[warp];

  // warp w of CTA c takes tiles w * CTAs + c, then every (warps * CTAs)-th: the whole chip reads one stretch of memory
  // at a time
  const int n_tiles = static_cast<int>(n / kQuantTile);
  const int stride = static_cast<int>(gridDim.x) * kQuantWarps, first = warp * static_cast<int>(gridDim.x) + static_cast<int>(blockIdx.x);
  const int mine = first < n_tiles ? (n_tiles - first + stride - 1) / stride : 0;
  auto tile_at = [&](int i) { return (static_cast<long long>(first) + static_cast<long long>(i) * stride) * kQuantTile; };

  if (threadIdx.x == 0) s_abort = 0;
  if (lane == 0) {
    for (int s = 0; s < kQuantStages; ++s) mbar_init(smem_u32(&bar[s]), 1);
    mbar_init_fence();
  }
  // The L2 is asked to hold on to the last of the tiles that are read again and to nothing else: what pass 2 reads or writes is
  // not used again.  67,108,864 elements: 79.5 us with 30 MB held, 78.9 with 45, 78.4 with 50, 78.0 with 58 or 64 (the L2 is two halves,
  // and what is read from the other half takes room in both); 33,554,432: 34.7, 35.4, 35.6, 35.6, 35.6.  Tiles for pass 2 asked into the
  // L2 before the grid's barrier: 2 a warp 78.0 and 35.9, 8 a warp 80.7 and 36.2.
  const uint64_t evict_first = l2_evict_first(), evict_last = l2_evict_last();
  // Pass 2 finds tiles [still_there, mine) in the ring, the first on_chip in registers and tensor memory, and reads the others
  // again: those from `held` on from the L2, those below from DRAM.
  const int on_chip = min(mine, kTmem ? kQuantKeep + kQuantTmem : kQuantKeep), still_there = max(mine - kQuantStages, on_chip);
  const int hold = static_cast<int>(kQuantHoldBytes / (static_cast<long long>(kQuantTile) * 4 * stride));
  const int held = max(still_there - hold, on_chip);
  auto load = [&](int i, int s, bool first_pass) {
    mbar_arrive_expect_tx(smem_u32(&bar[s]), kQuantTile * sizeof(float));
    bulk_load(smem_u32(ring + s * kQuantTile), x + tile_at(i), kQuantTile * sizeof(float), smem_u32(&bar[s]),
              first_pass && i >= held && i < still_there ? evict_last : evict_first);
  };
  if (lane == 0)
    for (int i = 0; i < kQuantStages && i < mine; ++i) load(i, i, true);
  if (kTmem && warp == 0) {
    __syncwarp();
    tmem_alloc(smem_u32(&s_tmem), kQuantTmemCols);
    tmem_relinquish();
  }
  if (kTmem) tc_fence_before();
  __syncthreads();
  if (kTmem) tc_fence_after();
  const uint32_t tmem_base = kTmem ? *reinterpret_cast<volatile uint32_t*>(&s_tmem) : 0u;
  const uint32_t my_tmem = tmem_base + (static_cast<uint32_t>(warp & 3) << 21) + static_cast<uint32_t>((warp >> 2) * 32 * kQuantTmem);
  // What is left behind the last whole tile is the last CTA's, asked for here: after the tiles its latency would be seen (600,001
  // elements 8.3 -> 6.2 us).
  constexpr int kQuantRest = kQuantTile / kQuantThreads;
  const long long rest_end = blockIdx.x == gridDim.x - 1 ? n : 0;
  auto rest_at = [&](int k) { return static_cast<long long>(n_tiles) * kQuantTile + k * kQuantThreads + static_cast<int>(threadIdx.x); };
  float rest[kQuantRest];
#pragma unroll
  for (int k = 0; k < kQuantRest; ++k) rest[k] = rest_at(k) < rest_end ? x[rest_at(k)] : 0.f;
  volatile int* abort_flag = &s_abort;
  bool ok = true;
  uint32_t parity_bits = 0u;                   // bit s: parity of the next completion of ring slot s
  auto landed = [&](int s) {
    ok = ok && __all_sync(0xFFFFFFFFu, mbar_wait_timed(smem_u32(&bar[s]), (parity_bits >> s) & 1u, abort_flag));
    parity_bits ^= 1u << s;
    return reinterpret_cast<const float4*>(ring + s * kQuantTile);
  };

  // ---- pass 1: the largest magnitude
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
  int slot = kQuantKeep;
  auto next_slot = [&]() { if (++slot == kQuantStages) slot = 0; };
#pragma unroll 1
  for (int i = kQuantKeep; kTmem && i < on_chip; ++i, next_slot()) {
    const float4* t = landed(slot);
    float4 v[kQuantVec];
#pragma unroll
    for (int k = 0; k < kQuantVec; ++k) {
      v[k] = t[lane + 32 * k];
      m = abs_max4(m, v[k]);
    }
    tmem_st_tile(my_tmem + static_cast<uint32_t>((i - kQuantKeep) * 32), v);
    __syncwarp();
    if (lane == 0 && i + kQuantStages < mine) load(i + kQuantStages, slot, true);
  }
  for (int i = max(on_chip, kQuantKeep); i < mine; ++i, next_slot()) {
    const float4* t = landed(slot);
#pragma unroll
    for (int k = 0; k < kQuantVec; ++k) m = abs_max4(m, t[lane + 32 * k]);
    __syncwarp();
    if (lane == 0 && i + kQuantStages < mine) load(i + kQuantStages, slot, true);
  }
  if (kTmem) {
    __syncwarp();
    tmem_wait_st();
  }
#pragma unroll
  for (int k = 0; k < kQuantRest; ++k) m = fmaxf(m, fabsf(rest[k]));

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

  // ---- pass 2: quantise.  First what the ring holds; every slot that gets free takes one of the tiles that are read again, DRAM's and
  // the L2's in turn, in proportion to their numbers, so that DRAM is busy from the first to the last.
  auto store = [&](int i, const float4 (&v)[kQuantVec]) {
    uint32_t words[kQuantVec];
    const bool good = quant_words(v, scale, words);
    uint32_t* to = reinterpret_cast<uint32_t*>(out + tile_at(i)) + lane;
#pragma unroll
    for (int k = 0; k < kQuantVec; ++k) __stcs(to + 32 * k, words[k]);
    if (!good) {
      const float4* from = reinterpret_cast<const float4*>(x + tile_at(i)) + lane;
#pragma unroll 1
      for (int k = 0; k < kQuantVec; ++k) to[32 * k] = quant_four(from[32 * k], scale);
    }
  };
  const int again = still_there - on_chip, from_dram = held - on_chip;
  int next_l2 = still_there - 1, next_dram = held - 1, asked = 0, turn = again - 1;
  int in_slot = 0;                             // lane s: the tile that is on its way into ring slot s
  auto ask = [&](int s) {
    if (!kTmem || asked == again) return;
    ++asked;
    turn += from_dram;
    const bool dram = turn >= again;
    if (dram) turn -= again;
    const int i = dram ? next_dram-- : next_l2--;
    if (lane == s) in_slot = i;
    if (lane == 0) load(i, s, false);
  };
  auto from_ring = [&](int i, int s, const float4* t) {
    float4 v[kQuantVec];
#pragma unroll
    for (int k = 0; k < kQuantVec; ++k) v[k] = t[lane + 32 * k];
    __syncwarp();
    ask(s);
    store(i, v);
  };
  int s = mine > 0 ? (mine - 1) % kQuantStages : 0;
  auto slot_before = [&]() { s = s == 0 ? kQuantStages - 1 : s - 1; };
  const int first_again = s;
  for (int i = mine - 1; i >= still_there; --i, slot_before()) from_ring(i, s, reinterpret_cast<const float4*>(ring + s * kQuantTile));
#pragma unroll
  for (int i = 0; i < kQuantKeep; ++i)
    if (i < mine) store(i, keep[i]);
#pragma unroll 1
  for (int i = kQuantKeep; kTmem && i < on_chip; ++i) {
    float4 v[kQuantVec];
    tmem_ld_tile(my_tmem + static_cast<uint32_t>((i - kQuantKeep) * 32), v);
    store(i, v);
  }
  s = first_again;
  for (int i = 0; kTmem && i < again; ++i, slot_before()) from_ring(__shfl_sync(0xFFFFFFFFu, in_slot, s), s, landed(s));
#pragma unroll
  for (int k = 0; k < kQuantRest; ++k)
    if (rest_at(k) < rest_end) out[rest_at(k)] = static_cast<int8_t>(quant_one(rest[k], scale));
  if (!ok && lane == 0) {
    raise_status(abort_flag, status, FMHA_I8_DEV_WAIT_QUANT, blockIdx.x);
    const long long t0 = clock64();
    while (clock64() - t0 < 2000000LL) { /* copies still in flight land before the CTA may exit */ }
  }
  if (kTmem) {
    tc_fence_before();
    __syncthreads();
    if (warp == 0) {
      tc_fence_after();
      tmem_dealloc(tmem_base, kQuantTmemCols);
    }
  }
}

}  // namespace fmha
