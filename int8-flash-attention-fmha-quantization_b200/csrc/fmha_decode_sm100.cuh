// Attention of a few query rows per head (decoding against a cache): fmha_i8_sm100_infer_cross with up to four rows, at head_dim 64
// up to kDecodeMaxRows (few_rows() in fmha_api.cu draws the line).  Same arithmetic as the forward kernel (fmha_fwd_sm100.cuh): key tiles of 128 starting at key 0, P
// quantised to 8 bits against each tile's own row maximum, tiles merged in fp32; key tiles without an unmasked key are
// skipped.
//
// What bounds it: every byte of K and V is used once or a few times, so HBM does.  The tensor-core kernel spends a 128-row
// tile on the few rows and leaves one SM to walk all keys of a head; here
//   * a head is split over the CTAs of a cluster (1..8) and over the warps of a CTA; every warp owns whole key tiles, keeps
//     its running maximum, sum and output row, and the partial results meet in the first CTA's shared memory at the end;
//   * a key tile is one contiguous piece of K and one of V, brought in by one bulk copy each; a warp has one tile of
//     both, and asks for the next K as soon as it has formed its scores, for the next V after P.V.  Three CTAs of 64 KB
//     share an SM, so about 100 KB per SM are in flight, enough to cover the latency of HBM at full bandwidth;
//   * dot products on the integer cores (dp4a).  Scores: one lane = four neighbouring keys, whose 16-byte chunks it reads
//     in an order rotated by its lane number (no bank conflicts).  P.V: one lane = four neighbouring output columns, the
//     bytes of four keys transposed with eight byte permutations.  About 770 warp instructions per tile of 32 KB and one
//     row, an eighth of what the SM can issue while that tile arrives.
// Measured against the general kernel, cross attention B16 H32 D128, 1025..4096 keys of 4096 per sequence, one row per head
// (340 MB on average): 82.9 -> 55.3 us, 94 % of the measured copy bandwidth.
#pragma once
#include <cuda_runtime.h>
#include <cstdint>
#include "fmha_fwd_sm100.cuh"
#include "ptx.cuh"
#include "../../include/fmha_i8_c.h"

namespace fmha {

constexpr int kDecodeMaxRows = 8;
constexpr int kDecodeMaxCluster = 8;
template <int D> struct DecodeCfg {
  static constexpr int kWarps = (D == 128) ? 2 : 4;              // 64 KB of tiles per CTA at either head_dim
  static constexpr int kThreads = kWarps * 32;
  static constexpr int kTileBytes = kTile * D;
  static constexpr int kRingBytes = 2 * kWarps * kTileBytes;     // per warp: one K tile, one V tile
  static constexpr int kPartFloats = D + 2;                      // one row of a partial result: output, maximum, sum
};
template <int D, int R> struct DecodeSmem {
  alignas(128) uint8_t ring[DecodeCfg<D>::kRingBytes];           // at the end, in the cluster's first CTA: the partial results
  alignas(16) uint32_t q[R][D / 4];
  alignas(16) uint32_t p[DecodeCfg<D>::kWarps][R][32];           // the 8-bit P row of a tile, four keys per word
  uint64_t k_full[DecodeCfg<D>::kWarps], v_full[DecodeCfg<D>::kWarps];
  uint32_t live_bits[kMaxTiles / 32];
  uint8_t live[kMaxTiles];
  int n_live, abort;
};

// acc + the dot product of four unsigned bytes with four signed ones
__device__ __forceinline__ int dot4(uint32_t p, uint32_t v, int acc) {
  int d;
  asm("dp4a.u32.s32 %0, %1, %2, %3;" : "=r"(d) : "r"(p), "r"(v), "r"(acc));
  return d;
}

// grid = (clusters of c CTAs) x (bh_count * row groups); R = query rows per group (rows past Sq are computed and dropped).
template <int D, int R>
__global__ void __launch_bounds__(DecodeCfg<D>::kThreads, 3)
fmha_decode_kernel(const int8_t* q, const int8_t* k, const int8_t* v, const FwdParams p) {
  using Cfg = DecodeCfg<D>;
  using Smem = DecodeSmem<D, R>;
  constexpr int W = Cfg::kWarps;
  extern __shared__ __align__(128) uint8_t smem_raw[];
  Smem& sm = *reinterpret_cast<Smem*>(smem_raw);
  grid_launch_dependents();
  const int lane = threadIdx.x & 31, warp = warp_index();
  const int ctas = static_cast<int>(cluster_ctas()), rank = static_cast<int>(cluster_rank());
  const int unit = static_cast<int>(blockIdx.x) / ctas;
  const int bh = unit / p.q_tiles, row0 = (unit - bh * p.q_tiles) * R;
  const int batch = (p.bh_begin + bh) / p.H;
  const int n_tiles = (p.S + kTile - 1) / kTile;
  const uint32_t* mask4 = reinterpret_cast<const uint32_t*>(p.mask + static_cast<int64_t>(batch) * p.S);
  const int8_t* k_head = k + static_cast<int64_t>(bh) * p.S * D;
  const int8_t* v_head = v + static_cast<int64_t>(bh) * p.S * D;

  if (threadIdx.x == 0) sm.abort = 0;
  if (lane == 0) {
    mbar_init(smem_u32(&sm.k_full[warp]), 1);
    mbar_init(smem_u32(&sm.v_full[warp]), 1);
    mbar_init_fence();
  }
  if (threadIdx.x < kMaxTiles / 32) sm.live_bits[threadIdx.x] = 0u;
  __syncthreads();
  grid_dependency_wait();

  // ---- query rows; key tiles with at least one unmasked key (a word of the mask = four keys; S is a multiple of 64)
  for (int i = threadIdx.x; i < R * (D / 4); i += Cfg::kThreads) {
    const int r = i / (D / 4);
    sm.q[r][i % (D / 4)] = (row0 + r < p.Sq) ? reinterpret_cast<const uint32_t*>(q + (static_cast<int64_t>(bh) * p.Sq + row0) * D)[i] : 0u;
  }
  auto mask_word = [&](int t) -> uint32_t {
    const int key = t * kTile + 4 * lane;
    return key < p.S ? mask4[key >> 2] : 0xFFFFFFFFu;
  };
  auto has_key = [&](uint32_t m4) -> bool { return __any_sync(0xFFFFFFFFu, __vcmpeq4(m4, 0u) != 0u); };      // a mask byte that is zero
  if (n_tiles <= 2 * W) {
#pragma unroll 1
    for (int t = warp; t < n_tiles; t += W)
      if (has_key(mask_word(t)) && lane == 0) atomicOr(&sm.live_bits[0], 1u << t);
  } else {
    // A warp takes a run of tiles inside one 32-bit word of the list, with eight loads in flight: one tile after the other,
    // which is what a CTA would wait for before its first copy, took 6 us of the call above.
    const int words = (n_tiles + 31) / 32, run = words == 1 ? (n_tiles + W - 1) / W : words >= W ? 32 : 16;
    for (int t0 = warp * run; t0 < n_tiles; t0 += W * run) {
      const int t1 = min(t0 + run, n_tiles);
      uint32_t bits = 0u;
#pragma unroll 1
      for (int t = t0; t < t1; t += 8) {
        uint32_t m4[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) m4[i] = mask_word(t + i);
#pragma unroll
        for (int i = 0; i < 8; ++i)
          if (has_key(m4[i]) && t + i < t1) bits |= 1u << ((t + i) & 31);
      }
      if (lane == 0) atomicOr(&sm.live_bits[t0 >> 5], bits);
    }
  }
  __syncthreads();
  for (int t = threadIdx.x; t < n_tiles; t += Cfg::kThreads) {
    const uint32_t word = sm.live_bits[t >> 5];
    int at = __popc(word & ((1u << (t & 31)) - 1u));
    for (int i = 0; i < (t >> 5); ++i) at += __popc(sm.live_bits[i]);
    if ((word >> (t & 31)) & 1u) sm.live[at] = static_cast<uint8_t>(t);
    if (t == n_tiles - 1) sm.n_live = at + static_cast<int>((word >> (t & 31)) & 1u);
  }
  __syncthreads();
  const int n_live = sm.n_live;
  const int begin = n_live * rank / ctas, end = n_live * (rank + 1) / ctas;      // this CTA's share

  uint8_t* k_tile = sm.ring + warp * 2 * Cfg::kTileBytes;
  uint8_t* v_tile = k_tile + Cfg::kTileBytes;
  const uint32_t bar_k = smem_u32(&sm.k_full[warp]), bar_v = smem_u32(&sm.v_full[warp]);
  volatile int* abort_flag = &sm.abort;
  // K and V pass through once: the L2 need not keep them
  const uint64_t once = l2_evict_first();
  auto fetch = [&](const int8_t* head, uint8_t* dst, uint32_t bar, int i) {
    const int t = sm.live[i];
    const uint32_t bytes = static_cast<uint32_t>(min(kTile, p.S - t * kTile)) * D;
    mbar_arrive_expect_tx(bar, bytes);
    bulk_load(smem_u32(dst), head + static_cast<int64_t>(t) * Cfg::kTileBytes, bytes, bar, once);
  };

  float m_run[R], l_run[R], o[R][4];
#pragma unroll
  for (int r = 0; r < R; ++r) {
    m_run[r] = -INFINITY;
    l_run[r] = 0.f;
#pragma unroll
    for (int c = 0; c < 4; ++c) o[r][c] = 0.f;
  }
  bool ok = true;
  uint32_t n = 0;
  if (lane == 0 && begin + warp < end) {
    fetch(k_head, k_tile, bar_k, begin + warp);
    fetch(v_head, v_tile, bar_v, begin + warp);
  }
  for (int i = begin + warp; i < end; i += W, ++n) {
    const int key0 = sm.live[i] * kTile + 4 * lane;         // my four keys
    const uint32_t masked = key0 < p.S ? ~__vcmpeq4(mask4[key0 >> 2], 0u) : 0xFFFFFFFFu;    // byte = 0xFF: masked

    // ---- scores of my four keys (inc/fmha_i8.cuh:120-172)
    if (!(ok = __all_sync(0xFFFFFFFFu, mbar_wait_timed(bar_k, n & 1u, abort_flag)))) break;
    int s[R][4];
#pragma unroll
    for (int r = 0; r < R; ++r)
#pragma unroll
      for (int j = 0; j < 4; ++j) s[r][j] = 0;
    // Eight lanes read 16 bytes each at a time, without bank conflicts if they hit eight different 16-byte columns of the
    // 128-byte line.  head_dim 128: rotating the chunk by the lane does it.  head_dim 64: a line holds two keys; rotating
    // covers one half of it, and every other group of four lanes takes its keys in the order 1 0 3 2 for the other half.
    constexpr int kChunks = D / 16;
    const int swap = (D == 64) ? (lane >> 2) & 1 : 0;
#pragma unroll
    for (int c = 0; c < kChunks; ++c) {
      const int at = (c + lane) & (kChunks - 1);
      uint4 qc[R];
#pragma unroll
      for (int r = 0; r < R; ++r) qc[r] = reinterpret_cast<const uint4*>(sm.q[r])[at];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const uint4 kc = reinterpret_cast<const uint4*>(k_tile)[(4 * lane + (j ^ swap)) * kChunks + at];
#pragma unroll
        for (int r = 0; r < R; ++r) {
          s[r][j] = __dp4a(static_cast<int>(qc[r].x), static_cast<int>(kc.x), s[r][j]);
          s[r][j] = __dp4a(static_cast<int>(qc[r].y), static_cast<int>(kc.y), s[r][j]);
          s[r][j] = __dp4a(static_cast<int>(qc[r].z), static_cast<int>(kc.z), s[r][j]);
          s[r][j] = __dp4a(static_cast<int>(qc[r].w), static_cast<int>(kc.w), s[r][j]);
        }
      }
    }
    __syncwarp();
    if (lane == 0 && i + W < end) fetch(k_head, k_tile, bar_k, i + W);

    // ---- tile maximum, P, row sum (inc/fmha_i8.cuh:183-253), merge of the statistics (:301-304)
    float e_old[R], e_cur[R];
    __syncwarp();                                           // P of the tile before has been read by all lanes
#pragma unroll
    for (int r = 0; r < R; ++r) {
      if (D == 64 && swap) {
        int t = s[r][0]; s[r][0] = s[r][1]; s[r][1] = t;
        t = s[r][2]; s[r][2] = s[r][3]; s[r][3] = t;
      }
      int mx = INT_MIN;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        s[r][j] += static_cast<int>(kMagicBits);            // the bits of the float 1.5*2^23 + s
        if (!((masked >> (8 * j)) & 1u)) mx = max(mx, s[r][j]);
      }
      mx = __reduce_max_sync(0xFFFFFFFFu, mx);              // a live tile has an unmasked key
      const RowConsts rc = row_consts(mx, p.c2, p.row_scale, p.scale_qk, p.p_mul);
      float sum = 0.f;
      uint32_t word = 0u;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float x = ((masked >> (8 * j)) & 1u) ? -INFINITY : __int_as_float(s[r][j]);
        const float e = ex2_approx(fmaf(x, rc.c2.x, rc.neg_hi.x));
        sum += e;
        word |= (__float_as_uint(fmaf(e, rc.p_mul_f.x, kMagic)) & 0xFFu) << (8 * j);
      }
      sm.p[warp][r][lane] = word;
#pragma unroll
      for (int d = 16; d > 0; d >>= 1) sum += __shfl_xor_sync(0xFFFFFFFFu, sum, d);
      const float m_new = fmaxf(m_run[r], rc.m_tile);
      e_old[r] = __expf(m_run[r] - m_new);                  // 0 on the first tile
      e_cur[r] = __expf(rc.m_tile - m_new);
      l_run[r] = fmaf(e_old[r], l_run[r], e_cur[r] * (rc.f * sum));
      m_run[r] = m_new;
    }
    __syncwarp();

    // ---- P.V of my four output columns (inc/fmha_i8.cuh:255-296); at head_dim 64 the two halves of the warp take one half
    //      of the keys each and are added up at the end
    if (!(ok = __all_sync(0xFFFFFFFFu, mbar_wait_timed(bar_v, n & 1u, abort_flag)))) break;
    constexpr int kWords = D / 4, kGroups = 32 * kWords / 32;       // words per row; groups of four keys per lane
    const int col = lane & (kWords - 1), group0 = (D == 64) ? (lane >> 4) * kGroups : 0;
    const uint32_t* vw = reinterpret_cast<const uint32_t*>(v_tile) + 4 * group0 * kWords + col;
    int acc[R][4];
#pragma unroll
    for (int r = 0; r < R; ++r)
#pragma unroll
      for (int c = 0; c < 4; ++c) acc[r][c] = 0;
#pragma unroll 2
    for (int g = 0; g < kGroups; g += 4) {
      uint4 pw[R];
#pragma unroll
      for (int r = 0; r < R; ++r) pw[r] = *reinterpret_cast<const uint4*>(&sm.p[warp][r][group0 + g]);
#pragma unroll
      for (int h = 0; h < 4; ++h) {
        const uint32_t* row = vw + 4 * (g + h) * kWords;
        const uint32_t v0 = row[0], v1 = row[kWords], v2 = row[2 * kWords], v3 = row[3 * kWords];
        const uint32_t a = __byte_perm(v0, v1, 0x5140), b = __byte_perm(v2, v3, 0x5140);
        const uint32_t c = __byte_perm(v0, v1, 0x7362), d = __byte_perm(v2, v3, 0x7362);
        const uint32_t w0 = __byte_perm(a, b, 0x5410), w1 = __byte_perm(a, b, 0x7632);
        const uint32_t w2 = __byte_perm(c, d, 0x5410), w3 = __byte_perm(c, d, 0x7632);
#pragma unroll
        for (int r = 0; r < R; ++r) {
          const uint32_t pr = h == 0 ? pw[r].x : h == 1 ? pw[r].y : h == 2 ? pw[r].z : pw[r].w;
          acc[r][0] = dot4(pr, w0, acc[r][0]);
          acc[r][1] = dot4(pr, w1, acc[r][1]);
          acc[r][2] = dot4(pr, w2, acc[r][2]);
          acc[r][3] = dot4(pr, w3, acc[r][3]);
        }
      }
    }
    __syncwarp();
    if (lane == 0 && i + W < end) fetch(v_head, v_tile, bar_v, i + W);
#pragma unroll
    for (int r = 0; r < R; ++r)
#pragma unroll
      for (int c = 0; c < 4; ++c) o[r][c] = fmaf(o[r][c], e_old[r], e_cur[r] * static_cast<float>(acc[r][c]));
  }
  if (!ok) {
    if (lane == 0) {
      raise_status(abort_flag, p.status, FMHA_I8_DEV_WAIT_K_LOAD, n);
      const long long t0 = clock64();
      while (clock64() - t0 < 2000000LL) { /* copies still in flight land before their memory is used again */ }
    }
    __syncwarp();
  }

  // ---- partial results into the first CTA's tiles, which nobody needs any more once all warps have come here
  cluster_arrive();
  cluster_wait();
  const uint32_t part0 = map_to_rank(smem_u32(sm.ring), 0);
  auto part_at = [&](int index, int r) { return part0 + static_cast<uint32_t>((index * R + r) * Cfg::kPartFloats * 4); };
#pragma unroll
  for (int r = 0; r < R; ++r) {
    if (D == 64)
#pragma unroll
      for (int c = 0; c < 4; ++c) o[r][c] += __shfl_xor_sync(0xFFFFFFFFu, o[r][c], 16);
    const uint32_t part = part_at(rank * W + warp, r);
    if (lane < D / 4) {
      st_cluster_v2(part + lane * 16, o[r][0], o[r][1]);
      st_cluster_v2(part + lane * 16 + 8, o[r][2], o[r][3]);
    }
    if (lane == 0) st_cluster_v2(part + D * 4, m_run[r], l_run[r]);
  }
  cluster_arrive();
  cluster_wait();
  if (rank != 0) return;

  // ---- merge, normalise, requantise, store (inc/fmha_i8.cuh:298-332): one thread = four output columns of one row
  for (int i = threadIdx.x; i < R * (D / 4); i += Cfg::kThreads) {
    const int r = i / (D / 4), col = i % (D / 4);
    if (row0 + r >= p.Sq) break;
    const float* parts = reinterpret_cast<const float*>(sm.ring) + r * Cfg::kPartFloats;
    float m = -INFINITY;
    for (int x = 0; x < ctas * W; ++x) m = fmaxf(m, parts[x * R * Cfg::kPartFloats + D]);
    float l = 0.f, a[4] = {0.f, 0.f, 0.f, 0.f};
    if (m > -INFINITY)
      for (int x = 0; x < ctas * W; ++x) {
        const float* part = parts + x * R * Cfg::kPartFloats;
        const float e = __expf(part[D] - m);
        l = fmaf(e, part[D + 1], l);
#pragma unroll
        for (int c = 0; c < 4; ++c) a[c] = fmaf(e, part[4 * col + c], a[c]);
      }
    const float inv = l > 0.f ? 1.0f / l : 0.f;
    uint32_t word = 0u;
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      const float y = fminf(fmaxf(p.scale_v_out * (a[c] * inv), -127.f), 127.f) + kMagic;
      word |= (__float_as_uint(y) & 0xFFu) << (8 * c);
    }
    reinterpret_cast<uint32_t*>(p.o + (static_cast<int64_t>(bh) * p.Sq + row0 + r) * D)[col] = word;
  }
}

}  // namespace fmha
