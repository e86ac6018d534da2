// The INT8 flash-attention forward kernel for sm_100a.
//
// Replaces the reference project's FMHAInferKernel (inc/fmha_i8.cuh:43-334).  Same arithmetic
// contract -- key tiles of 128 starting at key 0, P quantised to 8 bits against each tile's own row
// maximum, tiles merged in fp32 -- on a different machine model:
//
//   work unit  = (batch*head, one 128-row query tile).  The kernel is persistent: min(units, SMs)
//                CTAs, one per SM, CTA c walks units c, c + grid, ...  A CTA's whole life is ONE
//                sequence of steps g = 0, 1, 2, ... (step = one live key tile of one unit); barrier
//                phases, the K/V ring and tensor memory carry on from one unit to the next, so no role
//                drains at a unit boundary.
//   two chains = the softmax warps form two teams; steps alternate between them (chain = g & 1).
//   S buffers  = S = Q.K^T of step g lands in accumulator g % n of tensor memory (n = 3 at head_dim 128, 4 at
//                head_dim 64), issued as soon as that accumulator is free, i.e. several steps ahead of the
//                softmax warps.  The same accumulator then carries the step through the rest of its life: once the
//                softmax threads have consumed S, P.V of the step writes its partial output there.  The 8-bit P row
//                goes into a 32-column annex of the accumulator (head_dim 128) or over the two ends of the
//                accumulator itself (head_dim 64, where the partial output needs only 64 columns in between).  So
//                every step in flight owns its whole set of buffers and no role ever waits for another STEP's
//                buffer, only for its own step's previous stage.
//
//   warp 0       loader: TMA brings Q (once per unit, in a small ring) and rings of K and of V tiles into
//                swizzled shared memory, running ahead into the next units.
//   warp 1       S issuer:  S_b = bias + Q . K_g^T  (tcgen05.mma smem x smem -> int32 in tensor memory).
//   warp 2       scanner: turns the coming units' padding-mask rows into the list of key tiles that hold at least
//                one unmasked key, each marked if it has masked keys too (ring of four).
//   warp 3       P.V issuer:  O~ = bias + P_b . V_g  (tcgen05.mma tmem x smem -> int32 in tensor memory) when the
//                softmax warps have written P_b.
//                These four run warp-wide -- every lane waits and counts, one elected lane issues -- so that
//                descriptors and addresses are warp-uniform values; issued from a single divergent lane an MMA
//                cost about 100 cycles of issue time, this way about 70.
//   warps 4-11   merge: two threads per query row, each holding one half (D/2 columns) of the fp32 running
//                output row.  After P.V of a step they drain the partial output from tensor memory, rescale
//                and add it; at the end of a unit they normalise, requantise and store the row.  This keeps
//                the per-tile drain and the epilogue off the softmax warps.
//   warps 12-27  softmax: warps 12-19 serve chain 0, warps 20-27 chain 1.  TWO threads share one query row:
//                thread `half` owns keys [64*half, 64*half+64) of the tile.  Each reads its part of S twice
//                (integer max, then exp + requantise), the two exchange their maxima through shared memory,
//                and each writes its 8-bit P values into the annex or, at head_dim 64, over columns it has already
//                consumed (the lower half row walks up and leaves P in columns [0,16), the upper one walks down
//                and leaves it in [112,128)).
//                These threads hold no output row, so they are light (64 registers).
//
// What bounds it: issue slots (62 % busy; 4180 warp instructions for a step of 128 x 128 scores at head_dim 128, 2450 of them
// arithmetic) and the exponential unit (64 %), on a chain of hand-offs that the sets of buffers overlap; in units of one or two
// steps the merge warps, which spend more on a unit's epilogue than on a step.  B8 H32 S2048 D128: 405 us while the chip is cool enough
// for 1965 MHz, 430 to 440 back to back, where the power limit holds it at 1820 to 1860.
//
// The bias: every accumulator is first written by a one-step bf16 MMA whose operands hold 4096 and
// 3072, i.e. the fp32 value 1.5*2^23 (bits 0x4B400000); the int8 MMAs then add their integer result
// to that bit pattern.  Read back as a float the accumulator is exactly 1.5*2^23 + s, so no thread
// ever converts integers to floats: one fused multiply-add turns the raw accumulator into the
// exponent argument (or into the rescaled partial output).
//
// The padding mask goes the same way: where a key tile has masked keys, the issuer of S presets their columns to -2^127
// instead (a second product, 2^100 * -2^27, that swallows the first).  The scores added to that bit pattern leave a float
// of the same size (-2^126 at the least), below every real score as an integer and as a float.  Its exponential is zero,
// or 2^-126 where the workers of fmha_fwd64_sm100.cuh compute it on the multiply-add pipe: nothing beside the row maximum's, which is 2^-32 at the least, and
// quantised to zero.  (As long as 2^126 * c2 is large: kMinC2.)  The softmax threads treat every tile alike.  Before, they tested a mask bit per score in a loop that was not pipelined: B256 H16 S256
// D64 with lengths 64..256 took 132 us instead of 115, B24 H16 S576 D64 with lengths 300..576 66 instead of 59, and the
// smaller code makes unmasked head_dim-64 calls faster too (B8 H32 S2048: 430 -> 400 us).
//
// Tensor memory (512 columns x 128 lanes x 32 bit): accumulator b at columns [128 b, 128 b + 128).
// head_dim 128: annex b at [384 + 32 b, 384 + 32 b + 32) holds P (four int8 per column, keys in order), the partial
// output fills the accumulator.  head_dim 64: inside the accumulator, P of keys 0-63 in columns [0,16), P of keys
// 64-127 in columns [112,128), partial output in [16,80).
//
// Numerics kept equal to the reference kernel within the test tolerance: the running output is kept
// unnormalised (divided by the row sum once at the end) instead of renormalised after every tile,
// exp() is ex2.approx on an argument formed exactly from the integer accumulator, and masked keys
// contribute exactly zero (the reference adds a large negative number before scaling,
// inc/fmha_i8.cuh:191-193).  Key tiles with no unmasked key are skipped.
#pragma once
#include <cuda.h>
#include <cuda_runtime.h>
#include <cstdint>
#include "ptx.cuh"
#include "../../include/fmha_i8_c.h"

namespace fmha {

// Optional timeline tracing for performance work: with -DFMHA_TRACE the first CTA records clock64()
// stamps of its phase boundaries.  Compiled out of the product build.
#ifdef FMHA_TRACE
__device__ long long g_trace[48][512];
#define FMHA_STAMP(slot, idx) do { if (blockIdx.x == 0 && (threadIdx.x & 31) == 0 && (idx) < 512u) g_trace[slot][idx] = clock64(); } while (0)
#else
#define FMHA_STAMP(slot, idx) do { } while (0)
#endif

constexpr int kTile = 128;           // query rows per tile == keys per tile
constexpr int kHalf = 64;            // keys per softmax thread
constexpr int kMaxSeq = 32768;
constexpr int kMaxTiles = kMaxSeq / kTile;
constexpr int kSoftmaxWarps = 16;    // 2 chains x 2 key halves x 4 lane quarters
constexpr int kMergeWarps = 8;       // 2 column halves x 4 lane quarters
constexpr int kFwdWarps = kSoftmaxWarps + kMergeWarps + 4;
constexpr int kFwdThreads = kFwdWarps * 32;          // 896
// Warp numbering: the one-warp roles first, then the merge warps, then the softmax warps (a role's lane quarter of
// tensor memory is its warp number modulo 4; register targets are set per group of four warps).
constexpr int kWarpLoad = 0;
constexpr int kWarpMmaS = 1;
constexpr int kWarpScan = 2;
constexpr int kWarpMmaO = 3;
constexpr int kWarpMerge0 = 4;
constexpr int kWarpSoftmax0 = kWarpMerge0 + kMergeWarps;
// Tensor memory.  A buffer set is one 128-column accumulator that first holds S of a step and then, once the softmax
// threads have consumed it, the partial output P.V of the same step.
//   head_dim 128: three sets (384 columns) plus three 32-column annexes that take the P bytes of the step (480 columns);
//                 the partial output covers the whole accumulator, so P.V is one group of MMAs with N = 128.
//   head_dim 64:  four sets (512 columns); the P bytes stay inside the accumulator, keys 0-63 in its first 16 columns and
//                 keys 64-127 in its last 16, and the 64-column partial output sits between them from column 16 on.
//                 (Three sets with annexes, as at head_dim 128, run 5 % faster on sequences of 2048 and more and 5 %
//                 slower at sequence length 512, where the S issuer works several units ahead.)
template <int D> struct SBufs { static constexpr int n = (D == 128) ? 3 : 4; };
constexpr int kSBufsMax = 4;
template <int D> struct PLayout {
  static constexpr bool kAnnex = (D == 128);
  static constexpr int kOOff = kAnnex ? 0 : 16;        // first column of the partial output inside its accumulator
  static constexpr int kAnnexCols = 32;                // 128 keys x 1 byte
  // column (relative to the accumulator of the set, or to the set's annex) of the P bytes of keys [32 kk, 32 kk + 32)
  __host__ __device__ static constexpr int p_col(int kk) { return kAnnex ? 8 * kk : (kk >> 1) * 112 + (kk & 1) * 8; }
};
constexpr int kInfoBufs = 4;         // units whose mask information is resident at once
constexpr int kInfoConsumers = 3 + kSoftmaxWarps + kMergeWarps;   // loader, two issuers, softmax and merge warps release an info buffer once each
// setmaxnreg moves registers inside the CTA's own launch allocation (registers per thread at launch x
// threads), not inside the SM's whole register file: a request that does not fit blocks forever.  With
// 896 threads the launch allocation is 72 registers per thread (the host checks this before the first
// launch and refuses otherwise); the targets per role (FwdRegs) add up to 28 x 72.
constexpr int kLaunchRegs = 72;
template <int D> struct FwdRegs {
  // head_dim 128: the merge threads hold a 64-register half output row (B8 H32 S2048 at 1965 MHz: 104/40 takes 405 us,
  // 96/56 410, 88/72 427).  head_dim 64: the output row is 32 registers; 88/72 is the split at which
  // ptxas reports no spills at all, and C5 runs 5 % faster with it than with 80/88 or 96/56, which both spill.
  static constexpr int kSoftmax = 64, kMerge = (D == 128) ? 104 : 88, kOther = (D == 128) ? 40 : 72;
  static_assert(kSoftmaxWarps * kSoftmax + kMergeWarps * kMerge + 4 * kOther <= kFwdWarps * kLaunchRegs,
                "setmaxnreg targets exceed the CTA's register allocation: the kernel would hang");
  static_assert(kSoftmax <= kLaunchRegs && kMerge >= kLaunchRegs, "the softmax warps give registers, the merge warps gain");
};

constexpr uint32_t kTmemCols = 512;
constexpr float kMagic = 12582912.0f;          // 1.5 * 2^23: float whose ulp is 1 over [2^23, 2^24)
constexpr uint32_t kMagicBits = 0x4B400000u;
// Smallest factor from scores to exponents that the kernels work with, far from both of its limits.  A masked key's score is -2^126
// or less, and its exponent has to be below -150 for the exponential to be zero: 2^126 * 2^-100 = 2^26.  The scores of a row differ by
// at most 2 * 128 * 128 * head_dim = 2^22, and 2^22 * 2^-100 = 2^-78 is far below half an ulp of 1 (2^-25): the exponentials of a
// call whose own factor is smaller are all 1, and they are with this one.
constexpr float kMinC2 = 0x1p-100f;
// Largest one.  Scores are whole numbers: from here on a key whose score is not the row's maximum has an exponential of 2^-64 or less, which
// changes no sum and quantises to zero, and with this factor it has the same.  What it is for: the residue of row_consts, at most 32
// here, grows with the factor.
constexpr float kMaxC2 = 64.0f;
// Up to this factor 2^-residue is 1 - residue ln 2 to 2^-22, the accuracy of the exponentials (the residue is 2^-10 at the most).
constexpr float kLinearC2 = 0x1p-9f;
constexpr int kBiasBytes = 4096;               // 128 rows x 16 bf16, unswizzled core-matrix layout
template <int D> __host__ __device__ constexpr int bias_bytes() { return (2 + SBufs<D>::n) * kBiasBytes; }

template <int D> struct FwdCfg {
  static_assert(D == 64 || D == 128, "head_dim must be 64 or 128");
  static constexpr int kStagesK = (D == 128) ? 3 : 4;   // ring depth of K
  // ring depth of V: one thread loads K(g), V(g), K(g+1), ... in order, and V(g) is consumed a few steps (the number of S accumulators) after
  // K(g), so the V ring has to be that much deeper than the K ring
  static constexpr int kStagesV = (D == 128) ? 6 : 8;
  static_assert(kStagesV >= kStagesK + SBufs<D>::n, "V ring too shallow for the in-order loader");
  // Q tiles resident at once: the S cursor runs three steps ahead, which with one-tile units means three
  // units ahead, so short-sequence shapes want more than two (head_dim 128 has no shared memory to spare)
  static constexpr int kQBufs = (D == 128) ? 2 : 4;
  static constexpr int kTileBytes = kTile * D;              // one 128-row tile of int8
  static constexpr int kTilesBytesTotal = (kQBufs + kStagesK + kStagesV) * kTileBytes;
};

// u / d = u * mul >> shift for every u < 2^31, without a division's twenty instructions: all roles take units apart, and short
// units wait for it (B64 H32 S256 D128 81.9 -> 78.2 us).
struct FastDiv {
  uint32_t mul;
  int shift;
};
__device__ __forceinline__ int fast_div(int u, const FastDiv d) {
  return static_cast<int>((static_cast<uint64_t>(static_cast<uint32_t>(u)) * d.mul) >> d.shift);
}

struct FwdParams {
  const int8_t* mask;   // [B,S] whole mask
  int8_t* o;            // first head of the slice
  int o_wide;           // o is 32-byte aligned: the epilogue may use 32-byte stores
  int S;                // keys per head (seq_len; seq_len_k when queries and keys differ in number)
  int Sq;               // query rows per head (== S for self-attention)
  int H, bh_begin, bh_count, q_tiles;
  FastDiv by_q_tiles, by_heads;
  int n_units;          // bh_count * q_tiles work units
  int own_rounds;       // units [0, own_rounds * CTAs) are taken round-robin by the CTAs, one CTA each; the others ...
  int parts;            // ... by clusters of this many CTAs, each CTA a part of the unit's key tiles (1: no clusters, all units are round-robin)
  float row_scale;      // 1/sqrt(D), the reference's constant (inc/fmha_i8.cuh:71)
  float scale_qk;       // q_amax*k_amax/127^2 (inc/fmha_i8.cuh:72)
  float scale_v_out;    // v_amax/(o_amax*128) (inc/fmha_i8.cuh:318)
  float c2;             // row_scale*scale_qk*log2(e)
  float p_mul;          // 128: P8 = rn(128 p), the reference's quantisation (inc/fmha_i8.cuh:241-250, which keeps -rn(128 p) in a
                        // signed byte); 255: P8 = rn(255 p) (the reference README's planned UINT8 x INT8 variant).  P8 is an unsigned
                        // byte in all kernels.
  float* amax_out;      // calibration mode when not null: nothing is stored to o; instead the largest |output|
                        // in real units, max |O~ / l| * amax_scale, is folded into this device float
  float amax_scale;     // v_amax / (127 * 128)  (127 * 255 with unsigned P)
  unsigned* status;     // eight device status words
  // (Whole-row P scaling policies, fmha_policy_sm100.cuh: P8 = rn(p_mul * exp(score - row max)), or with the static scale
  // rn(127 min(p_mul * exp(score - row max) / l, 1)); scale_v_out is the factor that turns sum_j P8 v8 [/ l] into int8 output units.)
  unsigned char unused[32];            // see kParamBytes
};

// The size of a launch's parameters matters beyond what it holds, for reasons that were not found: B1 H2 S64 D64 takes 4.1 to 4.4 us a call with 536 or
// 600 bytes (24 modulo 64) and 4.4 to 4.8 with 504, 520, 528, 552, 568 or 760, in calls in a row, where the host is what they wait for; at head_dim
// 128 it makes no difference to short calls, but B8 H32 S2048 takes 405 us with 520 or more and 415 with 504 or 512 (what the compiler keeps in registers
// changes).
constexpr size_t kParamBytes = 3 * sizeof(CUtensorMap) + sizeof(FwdParams);
static_assert(kParamBytes == 536, "another size: measure the smallest and the long calls again");

// Kinds of live key tiles.  Tiles with unmasked keys in one half only -- the last one of a sequence, every other time -- are
// processed as the 64 keys of that half by the workers of fmha_fwd64_sm100.cuh: the other half's probabilities are zero and change
// no maximum, no sum and no product.  Here they are tiles with masked keys, of which the threads of a half without an unmasked one skip the
// exponentials: a second, shorter way through the whole step with the softmax threads' 64 registers costs the first one more than it saves (B64 H32
// S192 D128 72 -> 79 us, B8 H32 S2048 D128 415 -> 434).
constexpr uint8_t kTileMixed = 1;      // (the half in use of) the tile has masked keys too
constexpr uint8_t kTileLower = 2;      // keys 64..127 are all masked
constexpr uint8_t kTileUpper = 4;      // keys 0..63 are all masked
constexpr uint8_t kTileHalf = kTileLower | kTileUpper;

// What every role needs to know about one work unit's padding mask.  kInfoBufs of these live in shared
// memory: the scanner warp fills the ones of coming units while the current unit is being processed.
struct UnitInfo {
  int n_live;                         // key tiles with at least one unmasked key (of this CTA's part of them)
  int begin;                          // this CTA's part begins here in the lists below
  uint8_t live[kMaxTiles];            // indices of the live key tiles, ascending
  uint8_t kind[kMaxTiles];            // their kinds
};

template <int NK, int NV> struct FwdCtl {
  uint64_t q_full[4], q_empty[4];      // Q ring (kQBufs used): rows have landed / the unit's last S = Q.K^T has completed
  uint64_t k_full[NK], k_empty[NK], v_full[NV], v_empty[NV];
  uint64_t early_full;                 // the first unit's Q rows and its likely first K tile, asked for before its mask is known
  uint64_t s_full[kSBufsMax];          // per S accumulator: S = Q.K^T has completed
  uint64_t s_free[kSBufsMax];          // per S accumulator: the merge threads have drained the partial output that lived in it
  uint64_t o_full[kSBufsMax];          // per S accumulator: P.V of the step that owns it has completed
  uint64_t p_ready[4];                 // per step slot (g & 3): P written, row statistics published
  uint64_t xch[2][4];                  // per chain and lane quarter: the two half-row threads have published their maxima
  uint64_t info_full[kInfoBufs], info_empty[kInfoBufs];
  uint32_t tmem_base;
  int abort;
  // row statistics of a step, written by the softmax threads and read by the merge threads (slot = g & 3)
  float st_m[4][kTile], st_f[4][kTile], st_s0[4][kTile], st_s1[4][kTile];
  int xmax[2][2][2][kTile];            // [chain][step parity][half][row]: biased integer maximum of that half row
  float2 part[kTile];                  // row maximum and sum of a partial result (a unit shared by a cluster)
  UnitInfo info[kInfoBufs];
};

// Device view of one word of mapped host memory (set by the host once per device; null until then).
// A wait that gives up writes 1 to it so that the next host call sees the failure without a synchronisation.
__device__ unsigned* g_host_flag_ptr;

__device__ __noinline__ void raise_status(volatile int* abort_flag, unsigned* status, unsigned code, unsigned tile) {
  *abort_flag = 1;
  if (atomicCAS(&status[0], 0u, code) == 0u) {
    status[1] = blockIdx.x;
    status[2] = threadIdx.x >> 5;
    status[3] = tile;
    unsigned* host_word = g_host_flag_ptr;
    if (host_word != nullptr) {
      *reinterpret_cast<volatile unsigned*>(host_word) = 1u;
      __threadfence_system();
    }
  }
}

__device__ __forceinline__ float clear_low2(float x) { return __uint_as_float(__float_as_uint(x) & 0xFFFFFFFCu); }

__device__ __forceinline__ float ex2_approx(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// Builds one unit's view of its batch's padding mask: the list of live tiles and whether each has masked keys too.
// Executed by ONE warp; a lane looks at 32 keys, four lanes make a tile.  kGroups: groups of eight tiles whose loads are in
// flight together (for masks of more than 32 tiles, kLong: 128 tiles one group after the other take 5 us; in the workers, which feel the 7 KB of
// code that four take, two: B1 H16 S8192 348 -> 338 us, one 347).  kHalves: tiles with one open half are told apart.
template <int kGroups, bool kHalves, typename Info>
__device__ __forceinline__ int scan_mask_groups(Info* info, const uint32_t* words, int S, int n_tiles) {
  const int lane = threadIdx.x & 31;
  int n = 0;
#pragma unroll 1
  for (int base0 = 0; base0 < n_tiles; base0 += 8 * kGroups) {
    uint32_t open[kGroups], masked[kGroups];                     // any unmasked key; any masked key (keys beyond S count as masked)
#pragma unroll
    for (int q = 0; q < kGroups; ++q) {
      const int key0 = (base0 + 8 * q) * kTile + lane * 32;
      open[q] = 0u;
      masked[q] = 0xFFFFFFFFu;
      if (key0 < S) {  // S is a multiple of 64, so a 32-key group is entirely inside or outside
        masked[q] = 0u;
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const uint32_t wv = words[(key0 >> 2) + i];
          masked[q] |= wv;
          open[q] |= __vcmpeq4(wv, 0u);
        }
      }
    }
#pragma unroll
    for (int q = 0; q < kGroups; ++q) {
      const uint32_t any_open = __ballot_sync(0xFFFFFFFFu, open[q] != 0u), any_masked = __ballot_sync(0xFFFFFFFFu, masked[q] != 0u);
      const bool is_live = lane < 8 && ((any_open >> (4 * lane)) & 0xFu) != 0u;
      const uint32_t ballot = __ballot_sync(0xFFFFFFFFu, is_live);
      if (is_live) {
        const int pos = n + __popc(ballot & ((1u << lane) - 1u));
        info->live[pos] = static_cast<uint8_t>(base0 + 8 * q + lane);
        const uint32_t tile_masked = (any_masked >> (4 * lane)) & 0xFu, tile_open = (any_open >> (4 * lane)) & 0xFu;
        // (without kHalves they count as masked keys: one request of S320 waits for this, 6.5 -> 6.8 us)
        if (kHalves && (tile_open & 0xCu) == 0u) info->kind[pos] = kTileLower | ((tile_masked & 0x3u) != 0u ? kTileMixed : 0);
        else if (kHalves && (tile_open & 0x3u) == 0u) info->kind[pos] = kTileUpper | ((tile_masked & 0xCu) != 0u ? kTileMixed : 0);
        else info->kind[pos] = tile_masked != 0u ? kTileMixed : 0;
      }
      n += __popc(ballot);
    }
  }
  return n;
}
template <bool kHalves, int kLong, typename Info>
__device__ __forceinline__ void scan_mask_warp(Info* info, const int8_t* mask_row, int S, int n_tiles) {
  const uint32_t* words = reinterpret_cast<const uint32_t*>(mask_row);
  const int n = n_tiles <= 32 ? scan_mask_groups<1, kHalves>(info, words, S, n_tiles) : scan_mask_groups<kLong, kHalves>(info, words, S, n_tiles);
  if ((threadIdx.x & 31) == 0) info->n_live = n;
  __syncwarp();
}

// The same for up to kTiles key tiles, less code and shorter: a lane looks at four keys of each.  In the workers the scan stands between a step's S
// and its P.V, 2300 cycles in the general form, which P.V of half tiles waits for: B256 H16 S256 D64 (64..256 keys) 85.5 -> 84.3 us, B64 H16 S64 8.75
// -> 8.56; in the general kernel B64 H32 S256 D128 73.9 -> 73.0.  (For up to eight tiles, in the workers: B32 H12 S512 (256..512) 34.9 -> 35.5.)
template <int kTiles, bool kHalves, typename Info>
__device__ __forceinline__ void scan_few_tiles(Info* info, const int8_t* mask_row, int S) {
  const uint32_t* words = reinterpret_cast<const uint32_t*>(mask_row);
  const int lane = threadIdx.x & 31;
  uint32_t w[kTiles];
#pragma unroll
  for (int t = 0; t < kTiles; ++t) w[t] = t * kTile + lane * 4 < S ? words[t * 32 + lane] : 0xFFFFFFFFu;
  int n = 0;
#pragma unroll
  for (int t = 0; t < kTiles; ++t) {
    const uint32_t open = __ballot_sync(0xFFFFFFFFu, __vcmpeq4(w[t], 0u) != 0u), masked = __ballot_sync(0xFFFFFFFFu, w[t] != 0u);
    const bool no_upper = kHalves && (open >> 16) == 0u, no_lower = kHalves && (open & 0xFFFFu) == 0u;
    const uint32_t in_use = no_upper ? masked & 0xFFFFu : no_lower ? masked >> 16 : masked;
    if (open != 0u) {
      if (lane == 0) {
        info->live[n] = static_cast<uint8_t>(t);
        info->kind[n] = static_cast<uint8_t>((no_upper ? kTileLower : no_lower ? kTileUpper : 0) | (in_use != 0u ? kTileMixed : 0));
      }
      ++n;
    }
  }
  if (lane == 0) info->n_live = n;
  __syncwarp();
}

// The bf16 operands of the bias MMA in the unswizzled K-major layout (core matrix = 8 rows x 16 bytes, the two K halves
// of a row group 128 bytes apart, row groups 256 bytes apart).  A: every row holds 4096 and 2^100.  B: row n = key n holds
// 3072 and 0, or 3072 and -2^27 where the key is masked; one B for tiles without masked keys, one per S accumulator for the others.
constexpr uint32_t kBiasA = 0x71804580u;         // {4096, 2^100}
constexpr uint32_t kBiasB = 0x00004540u;         // {3072, 0}
constexpr uint32_t kBiasBMasked = 0xCD004540u;   // {3072, -2^27}
__device__ __forceinline__ void fill_bias_operands(uint8_t* bias_a, int n_b) {
  for (int i = threadIdx.x; i < (1 + n_b) * kBiasBytes / 16; i += blockDim.x)      // the B operands follow A
    reinterpret_cast<uint4*>(bias_a)[i] = make_uint4((i & 8) ? 0u : i < kBiasBytes / 16 ? kBiasA : kBiasB, 0u, 0u, 0u);
  fence_proxy_async_smem();
}
// Executed by one warp, lane l for keys l, 32 + l, 64 + l and 96 + l: the B operand of a tile with masked keys.
__device__ __forceinline__ void fill_mask_operand(uint8_t* bias_b, const bool (&masked)[4], const int group_bytes = 256) {
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int row = 32 * i + static_cast<int>(threadIdx.x & 31);
    *reinterpret_cast<uint32_t*>(bias_b + (row >> 3) * group_bytes + (row & 7) * 16) = masked[i] ? kBiasBMasked : kBiasB;
  }
  fence_proxy_async_smem();
  __syncwarp();
}

// Row maximum over N raw accumulator words (biased integers compare like the integers themselves).
template <int N>
__device__ __forceinline__ void chunk_max(const uint32_t (&r)[N], int& max_a, int& max_b) {
#pragma unroll
  for (int i = 0; i < N; i += 4) {
    max_a = max(max_a, max(static_cast<int>(r[i]), static_cast<int>(r[i + 1])));
    max_b = max(max_b, max(static_cast<int>(r[i + 2]), static_cast<int>(r[i + 3])));
  }
}

// 2^a for two values a <= 32 on the multiply-add pipe: a = n + f with |f| <= 1/2, a degree-5 minimax polynomial for 2^f (fitted by
// exchange; 2.1e-7 in fp32 arithmetic, the error bound of ex2.approx is 2^-22 = 2.4e-7), n added to the exponent.
__device__ __forceinline__ float2 exp2_poly(float2 a) {
  const float2 magic = make_float2(kMagic, kMagic), neg_magic = make_float2(-kMagic, -kMagic);
  a.x = fmaxf(a.x, -126.f);
  a.y = fmaxf(a.y, -126.f);
  const float2 t = __fadd2_rn(a, magic);                    // n in the low bits
  const float2 n = __fadd2_rn(t, neg_magic);
  const float2 f = __fadd2_rn(a, make_float2(-n.x, -n.y));
  float2 q = __ffma2_rn(f, make_float2(0.0013276472f, 0.0013276472f), make_float2(0.0096755410f, 0.0096755410f));
  q = __ffma2_rn(q, f, make_float2(0.0555071309f, 0.0555071309f));
  q = __ffma2_rn(q, f, make_float2(0.2402212024f, 0.2402212024f));
  q = __ffma2_rn(q, f, make_float2(0.6931469440f, 0.6931469440f));
  q = __ffma2_rn(q, f, make_float2(1.f, 1.f));
  return make_float2(__uint_as_float(__float_as_uint(q.x) + (__float_as_uint(t.x) << 23)), __uint_as_float(__float_as_uint(q.y) + (__float_as_uint(t.y) << 23)));
}

// N scores -> N probabilities (summed into two independent packed accumulators) -> N/4 words of
// packed bytes holding rn(128 p) (or rn(255 p)).  x = raw accumulator read as float = kMagic + s.
// A word's bytes are put together in pairs by the arithmetic that rounds them: kMagic + n1, times 256 and less 255 kMagic, is
// kMagic + 256 n1, all exact, and adding 128 p0 to that rounds to kMagic + 256 n1 + n0, where 128 p0 alone would round (256 n1 is
// even).  The two low bytes are the pair, as long as no byte is negative.  One byte permutation then makes a word of two pairs:
// four instructions per word against two multiply-adds and three permutations, which run at half rate.  (Long head_dim-128 sequences -1.4 to
// -2.6 % in one run, within the power limit's noise in others; B256 H16 S256 D64, 64..256 keys, -0.8 %.)
// kCap: p is multiplied by `share` and limited to one before it is quantised (the static policy clips at its top level,
// fmha_i8_quant_deviation.py:38-43): multiplications that saturate, where a minimum has half their rate.
// kPolyPairs: that many pairs of values per eight are computed by exp2_poly.  kPack = false: only the sums are wanted.
template <int N, bool kCap = false, int kPolyPairs = 0, bool kPack = true>
__device__ __forceinline__ void chunk_exp_pack(const uint32_t (&r)[N], const float2 c2, const float2 neg_hi,
                                               const float2 p_mul_f, float2 (&sum)[2], uint32_t (&packed)[N / 4], const float share = 0.f) {
  const float2 magic2 = make_float2(kMagic, kMagic);
#pragma unroll
  for (int g = 0; g < N / 4; ++g) {
    const float2 x01 = make_float2(__uint_as_float(r[4 * g]), __uint_as_float(r[4 * g + 1]));
    const float2 x23 = make_float2(__uint_as_float(r[4 * g + 2]), __uint_as_float(r[4 * g + 3]));
    const float2 a01 = __ffma2_rn(x01, c2, neg_hi);
    const float2 a23 = __ffma2_rn(x23, c2, neg_hi);
    float2 p01 = make_float2(ex2_approx(a01.x), ex2_approx(a01.y));
    float2 p23 = (g & 1) < kPolyPairs ? exp2_poly(a23) : make_float2(ex2_approx(a23.x), ex2_approx(a23.y));
    if (kCap) {
      p01.x = __saturatef(p01.x * share); p01.y = __saturatef(p01.y * share);
      p23.x = __saturatef(p23.x * share); p23.y = __saturatef(p23.y * share);
    }
    const float2 even = make_float2(p01.x, p23.x), odd = make_float2(p01.y, p23.y);
    sum[0] = __fadd2_rn(sum[0], even);
    sum[1] = __fadd2_rn(sum[1], odd);
    if (!kPack) continue;
    const float2 high = __ffma2_rn(__ffma2_rn(odd, p_mul_f, magic2), make_float2(256.f, 256.f), make_float2(-255.f * kMagic, -255.f * kMagic));
    const float2 y = __ffma2_rn(even, p_mul_f, high);
    packed[g] = __byte_perm(__float_as_uint(y.x), __float_as_uint(y.y), 0x5410);
  }
}

// Constants of one row of one tile, derived from the biased integer row maximum.
struct RowConsts {
  float2 c2, neg_hi, p_mul_f;
  float f, m_tile;
};
__device__ __forceinline__ RowConsts row_consts(const int imax, const float c2s, const float row_scale, const float scale_qk, const float p_mul) {
  // exponent argument (s - smax) * c2 = x * c2 - M * c2 with x = kMagic + s and M = kMagic + smax.
  // M * c2 = hi + lo exactly (lo is the rounding residual, half an ulp of hi or less: 2^-14 for c2 = 1e-4, 1/2 for 1, 32 for
  // 64); the factor 2^-lo is folded into the quantisation constant and the row sum, so nothing is lost and nothing is paid per element.
  RowConsts k;
  const float M = __uint_as_float(static_cast<uint32_t>(imax));
  const float hi = M * c2s;
  const float lo = fmaf(M, c2s, -hi);
  k.f = c2s < kLinearC2 ? fmaf(-lo, 0.6931471805599453f, 1.0f) : ex2_approx(-lo);
  k.c2 = make_float2(c2s, c2s);
  k.neg_hi = make_float2(-hi, -hi);
  k.p_mul_f = make_float2(p_mul * k.f, p_mul * k.f);        // 128 f (or 255 f): quantisation multiplier
  // the value the reference computes for the maximal element (inc/fmha_i8.cuh:196); rounded by itself, since what is wanted of it are
  // differences, and one of a rounded product and a fused multiply-add is not zero where the maxima are equal
  k.m_tile = __fmul_rn(row_scale * static_cast<float>(imax - static_cast<int>(kMagicBits)), scale_qk);
  return k;
}

// Does any of N pairs of the unnormalised output leave [-127, 127] when it is multiplied by `scale` and rounded?
template <int N> __device__ __forceinline__ bool needs_clamp(const float2* o2, const float scale) {
  float m0 = 0.f, m1 = 0.f;
#pragma unroll
  for (int i = 0; i < N; i += 2) { m0 = max3_abs(m0, o2[i].x, o2[i].y); m1 = max3_abs(m1, o2[i + 1].x, o2[i + 1].y); }
  return !(fmaxf(m0, m1) * scale < 127.25f);
}
// Eight pairs to sixteen bytes: rn(clamp(x * scale)) through the magic number (x + 1.5*2^23 has the integer nearest to x in its
// low bits, the low byte is the two's-complement integer), bytes gathered with PRMT.
__device__ __forceinline__ void requantise16(const float2* o2, const float2 scale, const bool clamp, uint32_t* words) {
  float2 v[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) v[i] = __ffma2_rn(o2[i], scale, make_float2(kMagic, kMagic));
  if (clamp) {      // (clamping commutes with the addition)
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      v[i].x = fminf(fmaxf(v[i].x, kMagic - 127.f), kMagic + 127.f);
      v[i].y = fminf(fmaxf(v[i].y, kMagic - 127.f), kMagic + 127.f);
    }
  }
#pragma unroll
  for (int i = 0; i < 4; ++i)
    words[i] = __byte_perm(__byte_perm(__float_as_uint(v[2 * i].x), __float_as_uint(v[2 * i].y), 0x0040),
                           __byte_perm(__float_as_uint(v[2 * i + 1].x), __float_as_uint(v[2 * i + 1].y), 0x0040), 0x5410);
}

// o2 = e_old * o2 + e_cur * (P8 . V) for N output columns.  r = accumulator, preset by the bias MMA, so that it reads as the float
// kMagic + (P8 . V).
template <int N>
__device__ __forceinline__ void drain_chunk(const uint32_t (&r)[N], float2* o2, const float2 e_cur, const float2 e_bias, const float2 e_old) {
#pragma unroll
  for (int i = 0; i < N / 2; ++i) {
    const float2 x = make_float2(__uint_as_float(r[2 * i]), __uint_as_float(r[2 * i + 1]));
    const float2 t = __ffma2_rn(x, e_cur, e_bias);          // e_cur * (P8 . V), exact product before rounding
    o2[i] = __ffma2_rn(o2[i], e_old, t);
  }
}

// The units of one CTA in order: `own` round-robin ones, then perhaps one that it shares with its cluster.
struct UnitWalk {
  int own, count, shared;
  __device__ __forceinline__ int unit(int it) const { return it < own ? static_cast<int>(blockIdx.x + it * gridDim.x) : shared; }
};
template <bool kFull>
__device__ __forceinline__ UnitWalk unit_walk(const FwdParams& p) {
  const int b = static_cast<int>(blockIdx.x), ctas = static_cast<int>(gridDim.x);
  UnitWalk w;
  if (!kFull || p.parts == 1) {
    w.own = w.count = (p.n_units - b + ctas - 1) / ctas;
    w.shared = 0;
  } else {
    w.own = p.own_rounds;
    w.shared = p.own_rounds * ctas + b / p.parts;           // a cluster's CTAs have consecutive numbers
    w.count = w.own + (w.shared < p.n_units ? 1 : 0);
  }
  return w;
}

// Geometry of work unit u.
struct UnitGeom {
  int bh_local, batch, q_row0;
};
__device__ __forceinline__ UnitGeom unit_geom(const FwdParams& p, int u) {
  UnitGeom g;
  g.bh_local = fast_div(u, p.by_q_tiles);
  g.batch = fast_div(p.bh_begin + g.bh_local, p.by_heads);
  g.q_row0 = (u - g.bh_local * p.q_tiles) * kTile;
  return g;
}

// ---------------------------------------------------------------------------------------------- softmax role
// One thread = one half (64 keys) of one query row of one chain.  Walks the CTA's step sequence and
// handles the steps of its chain.
template <int D>
__device__ __forceinline__ void softmax_role(const FwdParams& p, FwdCtl<FwdCfg<D>::kStagesK, FwdCfg<D>::kStagesV>* ctl, const uint32_t tmem_base,
                                             const UnitWalk walk) {
  const int warp = warp_index() - kWarpSoftmax0, lane = threadIdx.x & 31;
  const int chain = warp >> 3, half = (warp >> 2) & 1, quad = warp & 3;
  const int row = quad * 32 + lane;
  // my 64 columns of S buffer 0; my P bytes go over their first 16 columns
  const uint32_t tS0 = tmem_base + (static_cast<uint32_t>(quad * 32) << 16) + static_cast<uint32_t>(half * kHalf);
  const uint32_t bar_x = smem_u32(&ctl->xch[chain][quad]);
  volatile int* abort_flag = &ctl->abort;
  const float c2s = p.c2, row_scale = p.row_scale, scale_qk = p.scale_qk, p_mul = p.p_mul;

  uint32_t n = 0;     // steps this chain has processed so far (phase of xch)
  uint32_t g0 = 0;    // global index of the current unit's first step
  for (int it = 0; it < walk.count; ++it) {
    const int buf = it % kInfoBufs;
    if (!__all_sync(0xFFFFFFFFu, mbar_wait(smem_u32(&ctl->info_full[buf]), static_cast<uint32_t>((it / kInfoBufs) & 1), abort_flag))) {
      raise_status(abort_flag, p.status, FMHA_I8_DEV_WAIT_INFO, it);
      return;
    }
    const int n_live = ctl->info[buf].n_live;
    __syncwarp();
    if (lane == 0) mbar_arrive(smem_u32(&ctl->info_empty[buf]));     // only the tile count is needed here
#pragma unroll 1
    for (int j = (chain ^ static_cast<int>(g0)) & 1; j < n_live; j += 2, ++n) {
      const uint32_t g = g0 + static_cast<uint32_t>(j);
      const uint32_t sb = g % SBufs<D>::n;                       // S accumulator of this step
      const uint32_t tS = tS0 + sb * kTile;
      if (!__all_sync(0xFFFFFFFFu, mbar_wait(smem_u32(&ctl->s_full[sb]), (g / SBufs<D>::n) & 1u, abort_flag))) {
        raise_status(abort_flag, p.status, FMHA_I8_DEV_WAIT_S_READY, g);
        return;
      }
      tc_fence_after();
      if (half == 0 && quad == 0) FMHA_STAMP(chain * 4 + 0, n);

      // Order of my four 16-column chunks: at head_dim 64 the lower half row walks up, the upper half row walks DOWN, which
      // lets each leave its P bytes over columns it has already consumed (the first 16 and the last 16 of the
      // accumulator); columns [16,112) stay untouched, and P.V of this step puts the partial output there.
      const int c0 = !PLayout<D>::kAnnex && half ? 3 : 0, cs = !PLayout<D>::kAnnex && half ? -1 : 1;      // first chunk and direction
      // my 16 columns of P: inside the accumulator (head_dim 64) or in the annex of the buffer set (head_dim 128)
      const uint32_t tP = PLayout<D>::kAnnex
          ? tS0 - static_cast<uint32_t>(half * kHalf) + SBufs<D>::n * kTile + sb * PLayout<D>::kAnnexCols + static_cast<uint32_t>(half * 16)
          : tS + (half ? 48u : 0u);

      uint32_t ra[16], rb[16];
      // ---- pass 1: biased integer maximum of my 64 columns (inc/fmha_i8.cuh:183-206)
      int max_a = INT_MIN, max_b = INT_MIN;
      // two tensor-memory round trips (a round trip costs about as much as the whole arithmetic of this pass), two
      // 16-column loads in flight each time: 32 registers of data live instead of the 48 that one 32-column load
      // plus the prefetch for pass 2 would need
      tmem_ld16_issue(tS, ra);
      tmem_ld16_issue(tS + 16, rb);
      tmem_ld_fence(ra); tmem_ld_fence(rb);
      chunk_max<16>(ra, max_a, max_b);
      tmem_ld16_issue(tS + 32, ra);
      chunk_max<16>(rb, max_a, max_b);
      tmem_ld16_issue(tS + 48, rb);
      tmem_ld_fence(ra); tmem_ld_fence(rb);
      chunk_max<16>(ra, max_a, max_b);
      tmem_ld16_issue(tS + c0 * 16, ra);     // first chunk of pass 2, in flight during the exchange
      chunk_max<16>(rb, max_a, max_b);
      const int mine = max(max_a, max_b);
      // ---- exchange with the thread that owns the other half of this row
      int* xrow = &ctl->xmax[chain][n & 1u][0][row];
      xrow[half * kTile] = mine;
      mbar_arrive(bar_x);
      if (!__all_sync(0xFFFFFFFFu, mbar_wait(bar_x, n & 1u, abort_flag))) {
        tmem_ld_fence(ra);
        raise_status(abort_flag, p.status, FMHA_I8_DEV_WAIT_S_READY, g);
        return;
      }
      const int imax = max(mine, xrow[(half ^ 1) * kTile]);
      const RowConsts k = row_consts(imax, c2s, row_scale, scale_qk, p_mul);
      if (half == 0 && quad == 0) FMHA_STAMP(chain * 4 + 1, n);
      // Half a tile without an unmasked key (the last one of a sequence, every other time): no exponentials, all P are zero.  (The mask is the same
      // for all rows, and scores of unmasked keys are positive as biased integers.  B128 H16 S192 D128 66.7 -> 64.2 us, B128 H16 S64 23.2 -> 21.9, one
      // request of S320 5.77 -> 5.60 and at head_dim 128 6.36 -> 6.11; long sequences without such halves up to +0.3 %.)
      const bool none = __all_sync(0xFFFFFFFFu, mine < 0);

      // ---- pass 2: exp, row sum, requantise, P over columns already consumed (inc/fmha_i8.cuh:208-253)
      float2 sum[2] = {make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
      uint32_t packed[4];
      auto sixteen = [&](const uint32_t (&r)[16], int c) {
        chunk_exp_pack<16>(r, k.c2, k.neg_hi, k.p_mul_f, sum, packed);
        tmem_st4(tP + (c0 + c * cs) * 4, packed);
      };
      if (none) {
        tmem_ld_fence(ra);
#pragma unroll
        for (int c = 0; c < 4; ++c) packed[c] = 0u;
#pragma unroll
        for (int c = 0; c < 4; ++c) tmem_st4(tP + c * 4, packed);
      } else {
        tmem_ld_fence(ra); tmem_ld16_issue(tS + (c0 + cs) * 16, rb);
        sixteen(ra, 0);
        tmem_ld_fence(rb); tmem_ld16_issue(tS + (c0 + 2 * cs) * 16, ra);
        sixteen(rb, 1);
        tmem_ld_fence(ra); tmem_ld16_issue(tS + (c0 + 3 * cs) * 16, rb);
        sixteen(ra, 2);
        tmem_ld_fence(rb);
        sixteen(rb, 3);
      }
      // ---- publish the row statistics of this step for the merge threads
      const int slot = static_cast<int>(g & 3u);
      const float part = (sum[0].x + sum[0].y) + (sum[1].x + sum[1].y);
      if (half == 0) {
        ctl->st_m[slot][row] = k.m_tile;
        ctl->st_f[slot][row] = k.f;
        ctl->st_s0[slot][row] = part;
      } else {
        ctl->st_s1[slot][row] = part;
      }
      tmem_wait_st();
      tc_fence_before();
      mbar_arrive(smem_u32(&ctl->p_ready[slot]));
      if (half == 0 && quad == 0) FMHA_STAMP(chain * 4 + 2, n);
      FMHA_STAMP(16 + warp, n);
    }
    g0 += static_cast<uint32_t>(n_live);
  }
}

// ---------------------------------------------------------------------------------------------- merge role
// One thread = one half (D/2 columns) of the fp32 running output row of one query row, plus the running
// maximum and the running sum of that row (kept by both threads of the row).
template <int D, bool kFull>
__device__ __forceinline__ void merge_role(const FwdParams& p, FwdCtl<FwdCfg<D>::kStagesK, FwdCfg<D>::kStagesV>* ctl, const uint32_t tmem_base, uint8_t* tiles,
                                           const UnitWalk walk) {
  constexpr int DH = D / 2;
  const int warp = warp_index(), lane = threadIdx.x & 31;
  const int quad = warp & 3, ch = (warp - kWarpMerge0) >> 2;       // ch = which half of the output columns
  const int row = quad * 32 + lane;
  const uint32_t t_lane = tmem_base + (static_cast<uint32_t>(quad * 32) << 16);
  volatile int* abort_flag = &ctl->abort;

  // The running row is never cleared: the first tile of a unit multiplies what the unit before has left by zero.
  float2 o2[DH / 2];
#pragma unroll
  for (int i = 0; i < DH / 2; ++i) o2[i] = make_float2(0.f, 0.f);
  uint32_t g0 = 0;
  for (int it = 0; it < walk.count; ++it) {
    const int u = walk.unit(it);
    const int buf = it % kInfoBufs;
    if (!__all_sync(0xFFFFFFFFu, mbar_wait(smem_u32(&ctl->info_full[buf]), static_cast<uint32_t>((it / kInfoBufs) & 1), abort_flag))) {
      raise_status(abort_flag, p.status, FMHA_I8_DEV_WAIT_INFO, it);
      return;
    }
    const int n_live = ctl->info[buf].n_live;
    __syncwarp();
    if (lane == 0) mbar_arrive(smem_u32(&ctl->info_empty[buf]));     // only the tile count is needed here
    float m_run = -INFINITY, l_run = 0.f;

#pragma unroll 1
    for (int j = 0; j < n_live; ++j) {
      const uint32_t g = g0 + static_cast<uint32_t>(j);
      const int slot = static_cast<int>(g & 3u);
      const uint32_t sb = g % SBufs<D>::n;
      if (!__all_sync(0xFFFFFFFFu, mbar_wait(smem_u32(&ctl->p_ready[slot]), (g >> 2) & 1u, abort_flag))) {
        raise_status(abort_flag, p.status, FMHA_I8_DEV_WAIT_P_READY, g);
        return;
      }
      // ---- merge of tile statistics (inc/fmha_i8.cuh:301-304)
      const float m_tile = ctl->st_m[slot][row];
      const float l_tile = ctl->st_f[slot][row] * (ctl->st_s0[slot][row] + ctl->st_s1[slot][row]);
      const float m_new = fmaxf(m_run, m_tile);
      const float e_old = __expf(m_run - m_new);                       // 0 on the first tile (m_run = -inf)
      const float e_cur = clear_low2(__expf(m_tile - m_new));          // 22 significant bits: kMagic*e_cur is exact
      l_run = fmaf(e_old, l_run, e_cur * l_tile);
      m_run = m_new;
      const float2 e_cur2 = make_float2(e_cur, e_cur), e_bias = make_float2(-e_cur * kMagic, -e_cur * kMagic);
      const float2 e_old2 = make_float2(e_old, e_old);

      // ---- drain my half of O~ = bias + P8 . V into the fp32 running row.  The partial output of step g lives in
      //      the accumulator S(g) came from: all of it at head_dim 128, columns [16,80) at head_dim 64.
      if (!__all_sync(0xFFFFFFFFu, mbar_wait(smem_u32(&ctl->o_full[sb]), (g / SBufs<D>::n) & 1u, abort_flag))) {
        raise_status(abort_flag, p.status, FMHA_I8_DEV_WAIT_O_READY, g);
        return;
      }
      tc_fence_after();
      if (quad == 0) FMHA_STAMP(8 + 2 * ch, g);
      {
        // output column c of this step: tensor-memory column of 16-column chunk i of MY half
        auto chunk_col = [&](int i) -> uint32_t { return t_lane + sb * kTile + PLayout<D>::kOOff + ch * DH + i * 16; };
        // two loads in flight at a time: a round trip to tensor memory costs more than folding a chunk in
        uint32_t ra[16], rb[16];
        tmem_ld16_issue(chunk_col(0), ra);
        tmem_ld16_issue(chunk_col(1), rb);
#pragma unroll
        for (int c = 0; c < DH / 16; c += 2) {
          tmem_ld_fence(ra); tmem_ld_fence(rb);
          if (c + 2 >= DH / 16) {
            // the last two chunks are in registers: the accumulator can go back to the S issuer before they are folded in
            tc_fence_before();
            mbar_arrive(smem_u32(&ctl->s_free[sb]));
          }
          drain_chunk<16>(ra, o2 + c * 8, e_cur2, e_bias, e_old2);
          if (c + 2 < DH / 16) tmem_ld16_issue(chunk_col(c + 2), ra);
          drain_chunk<16>(rb, o2 + (c + 1) * 8, e_cur2, e_bias, e_old2);
          if (c + 3 < DH / 16) tmem_ld16_issue(chunk_col(c + 3), rb);
        }
      }
      if (quad == 0) FMHA_STAMP(9 + 2 * ch, g);
    }
    g0 += static_cast<uint32_t>(n_live);

    // (the unit's place is worked out here and not where it begins: nothing of it stays in registers over its steps)
    const UnitGeom geo = unit_geom(p, u);
    const int q_row = geo.q_row0 + row;

    // ---- calibration mode: only the largest magnitude of the unquantised output is wanted (the reference
    //      takes o_amax from its fp32 CPU result, test_fmha_i8.cpp:161)
    if (kFull && p.amax_out != nullptr) {
      float mx = 0.f;
      if (q_row < p.Sq && n_live > 0 && l_run > 0.f) {
        const float inv = 1.0f / l_run;
#pragma unroll
        for (int i = 0; i < DH / 2; ++i) mx = fmaxf(mx, fmaxf(fabsf(o2[i].x * inv), fabsf(o2[i].y * inv)));
      }
      // non-negative floats order like their bit patterns
      const unsigned bits = __reduce_max_sync(0xFFFFFFFFu, __float_as_uint(mx * p.amax_scale));
      if (lane == 0 && bits != 0u) atomicMax(reinterpret_cast<unsigned*>(p.amax_out), bits);
      continue;
    }

    // ---- a partial result: fp32 half row into the tiles, which nothing uses any more (16-byte chunk c of row r at chunk
    //      c ^ (r & 15): neither these stores nor the merge's loads meet in a bank), maximum and sum beside it
    if (kFull && it >= walk.own) {
      float4* dst = reinterpret_cast<float4*>(tiles) + row * (D / 4);
#pragma unroll
      for (int c = 0; c < DH / 4; ++c) dst[(ch * (DH / 4) + c) ^ (row & 15)] = make_float4(o2[2 * c].x, o2[2 * c].y, o2[2 * c + 1].x, o2[2 * c + 1].y);
      if (ch == 0) ctl->part[row] = make_float2(m_run, l_run);
      continue;
    }

    // ---- epilogue (inc/fmha_i8.cuh:318-332): normalise, requantise, store.  With units of one or two tiles the merge warps
    //      are what the CTA waits for (the epilogue took 3200 of a two-tile unit's 6000 cycles: its minima and maxima go
    //      to the half-rate pipe the softmax warps use most).  So the clamp is applied only where a warp has an output beyond
    //      127, which a calibrated scale makes rare; a row is not cleared for the next unit; no division.  B64 H32 S256
    //      D128: 86.2 -> 78.2 us, B32 H16 S384 46.0 -> 43.2, B128 H16 S128 41.0 -> 38.0.
    const float inv = (n_live > 0 && l_run > 0.f) ? __frcp_rn(l_run) : 0.f;
    const float scale = p.scale_v_out * inv;
    const bool clamp = __any_sync(0xFFFFFFFFu, needs_clamp<DH / 2>(o2, scale));
    if (q_row < p.Sq) {
      int8_t* dst = p.o + (static_cast<int64_t>(geo.bh_local) * p.Sq + q_row) * D + ch * DH;
      uint32_t wide[8];
#pragma unroll
      for (int c = 0; c < DH / 16; ++c) {
        requantise16(o2 + c * 8, make_float2(scale, scale), clamp, wide + (c & 1) * 4);
        // 32-byte stores: a warp's rows are 128 (or 64) bytes apart, so every store touches 32 lines whatever its
        // width, and the 16-byte version of this loop cost 5 % of the whole kernel at head_dim 128
        if (c & 1) {
          if (p.o_wide) {
            st_global_v8(dst + (c - 1) * 16, wide);
          } else {
            *reinterpret_cast<uint4*>(dst + (c - 1) * 16) = make_uint4(wide[0], wide[1], wide[2], wide[3]);
            *reinterpret_cast<uint4*>(dst + c * 16) = make_uint4(wide[4], wide[5], wide[6], wide[7]);
          }
        }
      }
    }
  }
}

template <int N> struct Flight { static constexpr int value = N; };

// The CTAs of a cluster have a part of one unit each: their warps merge some of the rows each, normalise, requantise and store
// them (inc/fmha_i8.cuh:298-332).  A lane holds four columns.
template <int D>
__device__ __forceinline__ void merge_parts(const FwdParams& p, const uint32_t part_smem, const uint32_t tiles_smem, const int unit) {
  const int lane = threadIdx.x & 31, warp = warp_index(), parts = p.parts, rank = static_cast<int>(blockIdx.x) % parts;
  const UnitGeom geo = unit_geom(p, unit);
  const int rows = min(kTile, p.Sq - geo.q_row0);
  constexpr int kLanes = D / 4, kRowsPerWarp = 32 / kLanes;
  const int c = lane & (kLanes - 1);
#pragma unroll 1
  for (int row = (rank * kFwdWarps + warp) * kRowsPerWarp + lane / kLanes; row < rows; row += parts * kFwdWarps * kRowsPerWarp) {
    float m = -INFINITY, l = 0.f;
    float4 o = make_float4(0.f, 0.f, 0.f, 0.f);
    // two parts (of a pair) or four in flight at a time: a load from another SM takes a good part of a microsecond
    auto fold = [&](auto flight, int r0) {
      constexpr int N = decltype(flight)::value;
      float2 ml[N];
      float4 x[N];
#pragma unroll
      for (int i = 0; i < N; ++i) {
        ml[i] = ld_cluster_v2(map_to_rank(part_smem + row * 8, r0 + i));
        x[i] = ld_cluster_v4(map_to_rank(tiles_smem + (row * kLanes + (c ^ (row & 15))) * 16, r0 + i));
      }
#pragma unroll
      for (int i = 0; i < N; ++i) {
        if (ml[i].y > 0.f) {
          const float m_new = fmaxf(m, ml[i].x), e = __expf(m - m_new), f = __expf(ml[i].x - m_new);
          m = m_new;
          l = fmaf(e, l, f * ml[i].y);
          o.x = fmaf(e, o.x, f * x[i].x); o.y = fmaf(e, o.y, f * x[i].y); o.z = fmaf(e, o.z, f * x[i].z); o.w = fmaf(e, o.w, f * x[i].w);
        }
      }
    };
    if (parts == 2) {
      fold(Flight<2>(), 0);
    } else {
#pragma unroll 1
      for (int r0 = 0; r0 < parts; r0 += 4) fold(Flight<4>(), r0);      // four or eight parts
    }
    const float scale = l > 0.f ? p.scale_v_out * __frcp_rn(l) : 0.f;
    const float v[4] = {o.x, o.y, o.z, o.w};
    uint32_t word = 0u;
#pragma unroll
    for (int i = 0; i < 4; ++i)
      word |= (__float_as_uint(fminf(fmaxf(fmaf(v[i], scale, kMagic), kMagic - 127.f), kMagic + 127.f)) & 0xFFu) << (8 * i);
    reinterpret_cast<uint32_t*>(p.o + (static_cast<int64_t>(geo.bh_local) * p.Sq + geo.q_row0 + row) * D)[c] = word;
  }
}

// ---------------------------------------------------------------------------------------------- loader
// One warp, run warp-wide (every lane waits and counts, one elected lane issues the copies): the Q tile of every
// non-empty unit, then per step the K tile and the V tile, in step order.
template <int D>
__device__ __forceinline__ void loader_role(const FwdParams& p, FwdCtl<FwdCfg<D>::kStagesK, FwdCfg<D>::kStagesV>* ctl,
                                            const CUtensorMap* map_q, const CUtensorMap* map_k, const CUtensorMap* map_v,
                                            const uint32_t q_smem, const uint32_t k_smem, const uint32_t v_smem,
                                            const UnitWalk walk) {
  using Cfg = FwdCfg<D>;
  constexpr uint32_t NK = Cfg::kStagesK, NV = Cfg::kStagesV, NQ = Cfg::kQBufs;
  volatile int* abort_flag = &ctl->abort;
  uint32_t g = 0;            // steps loaded so far: ring position and phase continue across units
  uint32_t qn = 0;           // non-empty units so far: Q buffer and phase
  uint32_t fail = 0u, fail_tile = 0u;
  // The first unit's Q rows, and the K tile that its list begins with unless the mask skips tiles, are asked for while the scanner
  // still waits for the mask: a call of one or two rounds is a chain of latencies, and this takes one of them out (B1 H2 S64 D64 4.6 -> 4.4
  // us, B1 H12 S320 6.55 -> 6.4, B1 H16 S576 D128 10.1 -> 9.85).
  int early_tile = -1;
  if (walk.count > 0) {
    const UnitGeom geo = unit_geom(p, walk.unit(0));
    const int parts = walk.own > 0 ? 1 : p.parts;
    early_tile = (p.S + kTile - 1) / kTile * (static_cast<int>(blockIdx.x) % parts) / parts;
    if (elect_one()) {
      const uint32_t bar = smem_u32(&ctl->early_full);
      mbar_arrive_expect_tx(bar, static_cast<uint32_t>(2 * Cfg::kTileBytes));
      tma_load_3d(q_smem, map_q, bar, 0, geo.q_row0, geo.bh_local);
      tma_load_3d(k_smem, map_k, bar, 0, early_tile * kTile, geo.bh_local);
    }
  }
  auto load_unit = [&](const int it, auto is_first) {
    constexpr bool kFirst = decltype(is_first)::value != 0;
    const int u = walk.unit(it);
    const int buf = it % kInfoBufs;
    if (!__all_sync(0xFFFFFFFFu, mbar_wait(smem_u32(&ctl->info_full[buf]), static_cast<uint32_t>((it / kInfoBufs) & 1), abort_flag))) {
      fail = FMHA_I8_DEV_WAIT_INFO; fail_tile = it; return;
    }
    const UnitGeom geo = unit_geom(p, u);
    const UnitInfo* info = &ctl->info[buf];
    const int n_live = info->n_live;
    if (kFirst && !__all_sync(0xFFFFFFFFu, mbar_wait(smem_u32(&ctl->early_full), 0u, abort_flag))) {
      fail = FMHA_I8_DEV_WAIT_Q_LOAD; fail_tile = it; return;
    }
    if (n_live > 0) {
      const uint32_t qb = qn % NQ;
      // the Q buffer is free once the last S = Q.K^T of the unit that used it NQ units ago has completed
      if (qn >= NQ && !__all_sync(0xFFFFFFFFu, mbar_wait(smem_u32(&ctl->q_empty[qb]), ((qn / NQ) - 1) & 1u, abort_flag))) {
        fail = FMHA_I8_DEV_WAIT_K_FREE; fail_tile = it; return;
      }
      if (elect_one()) {
        const uint32_t bar_q = smem_u32(&ctl->q_full[qb]);
        if (kFirst) {
          mbar_arrive(bar_q);
        } else {
          mbar_arrive_expect_tx(bar_q, static_cast<uint32_t>(Cfg::kTileBytes));
          tma_load_3d(q_smem + qb * Cfg::kTileBytes, map_q, bar_q, 0, geo.q_row0, geo.bh_local);
        }
      }
      ++qn;
      for (int j = 0; j < n_live; ++j, ++g) {
        const int t = info->live[info->begin + j];
        const uint32_t sk = g % NK, rk = g / NK, sv = g % NV, rv = g / NV;
        if (rk > 0 && !__all_sync(0xFFFFFFFFu, mbar_wait(smem_u32(&ctl->k_empty[sk]), (rk - 1) & 1u, abort_flag))) {
          fail = FMHA_I8_DEV_WAIT_K_FREE; fail_tile = g; break;
        }
        if (elect_one()) {
          if (kFirst && j == 0 && t == early_tile) {
            mbar_arrive(smem_u32(&ctl->k_full[sk]));
          } else {
            mbar_arrive_expect_tx(smem_u32(&ctl->k_full[sk]), Cfg::kTileBytes);
            tma_load_3d(k_smem + sk * Cfg::kTileBytes, map_k, smem_u32(&ctl->k_full[sk]), 0, t * kTile, geo.bh_local);
          }
        }
        if (rv > 0 && !__all_sync(0xFFFFFFFFu, mbar_wait(smem_u32(&ctl->v_empty[sv]), (rv - 1) & 1u, abort_flag))) {
          fail = FMHA_I8_DEV_WAIT_V_FREE; fail_tile = g; break;
        }
        if (elect_one()) {
          mbar_arrive_expect_tx(smem_u32(&ctl->v_full[sv]), Cfg::kTileBytes);
          tma_load_3d(v_smem + sv * Cfg::kTileBytes, map_v, smem_u32(&ctl->v_full[sv]), 0, t * kTile, geo.bh_local);
        }
      }
    }
    __syncwarp();
    if (fail == 0u && elect_one()) mbar_arrive(smem_u32(&ctl->info_empty[buf]));
  };
  if (walk.count > 0) load_unit(0, Flight<1>());
  for (int it = 1; it < walk.count && fail == 0u; ++it) load_unit(it, Flight<0>());
  if (fail != 0u) {
    if (elect_one()) raise_status(abort_flag, p.status, fail, fail_tile);
    // unwinding: let copies that are still in flight land before the CTA may exit
    const long long t0 = clock64();
    while (clock64() - t0 < 2000000LL) { /* about a millisecond */ }
  }
}

// ---------------------------------------------------------------------------------------------- MMA issuers
// Two warps issue tcgen05.mma: one the S = Q.K^T products, the other the P.V products.  Each runs warp-wide (every
// lane waits and counts, one elected lane issues) and walks the CTA's step sequence on its own; what orders them is the s_free barrier (S(g) may overwrite an accumulator only after
// the P.V that read the P bytes in it has completed) and, through the softmax warps, s_full -> p_ready.
// A wait that gives up only notes which one it was; the status is raised once, after the loop.
struct IssuerErr {
  uint32_t code = 0u, tile = 0u;
};
__device__ __forceinline__ bool issuer_wait(IssuerErr& e, uint32_t bar, uint32_t parity, uint32_t code, uint32_t tile, const volatile int* abort_flag) {
  if (__all_sync(0xFFFFFFFFu, mbar_wait(bar, parity, abort_flag))) return true;
  e.code = code;
  e.tile = tile;
  return false;
}

template <int D>
__device__ __forceinline__ void s_issuer_role(const FwdParams& p, FwdCtl<FwdCfg<D>::kStagesK, FwdCfg<D>::kStagesV>* ctl, const uint32_t tmem_base,
                                              const uint32_t q_smem, const uint32_t k_smem, uint8_t* bias_a,
                                              const UnitWalk walk) {
  using Cfg = FwdCfg<D>;
  constexpr uint32_t NK = Cfg::kStagesK, NQ = Cfg::kQBufs;
  volatile int* abort_flag = &ctl->abort;
  constexpr uint32_t idesc_s = make_idesc_i8(kTile, false);   // S = Q.K^T : N = 128 keys, both K-major
  constexpr uint32_t idesc_bias_s = make_idesc_bf16(kTile);
  const uint64_t d_bias_a = make_smem_desc_noswizzle(smem_u32(bias_a), 128, 256);
  const bool lead = elect_one();
  IssuerErr err;
  uint32_t g = 0, qn = 0;
  bool ok = true;
  for (int it = 0; it < walk.count && ok; ++it) {
    const int u = walk.unit(it);
    const int buf = it % kInfoBufs;
    if (!issuer_wait(err, smem_u32(&ctl->info_full[buf]), static_cast<uint32_t>((it / kInfoBufs) & 1), FMHA_I8_DEV_WAIT_INFO, it, abort_flag)) break;
    const UnitInfo* info = &ctl->info[buf];
    const int n_live = info->n_live;
    const uint32_t qb = qn % NQ;
    if (n_live == 0) {
      __syncwarp();
      if (elect_one()) mbar_arrive(smem_u32(&ctl->info_empty[buf]));
      continue;
    }
    const uint64_t dq = make_smem_desc(q_smem + qb * Cfg::kTileBytes, D);
    const int8_t* mask_row = p.mask + static_cast<int64_t>(unit_geom(p, u).batch) * p.S;
    for (int j = 0; j < n_live; ++j, ++g) {
      const uint32_t sb = g % SBufs<D>::n, stage = g % NK;
      uint32_t tS = tmem_base + sb * kTile;
      const bool mixed = info->kind[info->begin + j] != 0;
      bool masked[4] = {};
      if (mixed) {
        const int key0 = info->live[info->begin + j] * kTile + static_cast<int>(threadIdx.x & 31);
#pragma unroll
        for (int i = 0; i < 4; ++i) masked[i] = key0 + 32 * i >= p.S || mask_row[key0 + 32 * i] != 0;
      }
      // (behind the loads of mask bytes: one request of S320 5.60 -> 5.50 us)
      if (j == 0 && !issuer_wait(err, smem_u32(&ctl->q_full[qb]), (qn / NQ) & 1u, FMHA_I8_DEV_WAIT_Q_LOAD, g, abort_flag)) { ok = false; break; }
      // K first (it has normally been there for a while), then the accumulator: it still holds the partial output of
      // step g - n until the merge warps have drained it, and that hand-off is on the step-to-step critical path
      if (!issuer_wait(err, smem_u32(&ctl->k_full[stage]), (g / NK) & 1u, FMHA_I8_DEV_WAIT_K_LOAD, g, abort_flag)) { ok = false; break; }
      // What the MMAs need is formed and kept in registers before the wait that they follow; the compiler would form it where it is used, a
      // hundred cycles on the step-to-step path (here and for P.V, head_dim 128: B8 H32 S2048 425 -> 417 us, B4 H32 S1024 59.1 -> 58.1, B2 H16 Sq200 Sk1984
      // 15.7 -> 15.4).
      // The tile's preset operand: the common one, or this accumulator's own, which nothing has read since S of step g - n; that has completed,
      // or K of this step would not be there
      static_assert(Cfg::kStagesK <= SBufs<D>::n, "K of a step may land before S of step g - n has completed");
      const uint32_t b_index = mixed ? 1 + sb : 0u;
      if (mixed) fill_mask_operand(bias_a + (1 + b_index) * kBiasBytes, masked);
      uint64_t d_bias_b = make_smem_desc_noswizzle(smem_u32(bias_a) + (1 + b_index) * kBiasBytes, 128, 256);
      uint64_t dk = make_smem_desc(k_smem + stage * Cfg::kTileBytes, D);
      uint32_t bar_s = smem_u32(&ctl->s_full[sb]), bar_k = smem_u32(&ctl->k_empty[stage]), bar_q = j == n_live - 1 ? smem_u32(&ctl->q_empty[qb]) : 0u;
      asm volatile("" : "+l"(d_bias_b), "+l"(dk), "+r"(tS), "+r"(bar_s), "+r"(bar_k), "+r"(bar_q));
      if (g >= SBufs<D>::n && !issuer_wait(err, smem_u32(&ctl->s_free[sb]), ((g / SBufs<D>::n) - 1) & 1u, FMHA_I8_DEV_WAIT_O_FREE, g, abort_flag)) { ok = false; break; }
      FMHA_STAMP(15, g);
      tc_fence_after();
      if (lead) {
        mma_f16_ss(tS, d_bias_a, d_bias_b, idesc_bias_s, 0u);      // accumulator := 0x4B400000, masked keys -2^127
#pragma unroll
        for (int kk = 0; kk < D / 32; ++kk)
          mma_i8_ss(tS, desc_advance(dq, kk * 32), desc_advance(dk, kk * 32), idesc_s, 1u);
        mma_commit(bar_s);
        mma_commit(bar_k);
        if (bar_q != 0u) mma_commit(bar_q);                   // that was the unit's last use of its Q rows
      }
      FMHA_STAMP(12, g);
    }
    if (!ok) break;
    __syncwarp();
    if (elect_one()) mbar_arrive(smem_u32(&ctl->info_empty[buf]));
    ++qn;
  }
  if (err.code != 0u && elect_one()) raise_status(abort_flag, p.status, err.code, err.tile);
}

template <int D>
__device__ __forceinline__ void o_issuer_role(const FwdParams& p, FwdCtl<FwdCfg<D>::kStagesK, FwdCfg<D>::kStagesV>* ctl, const uint32_t tmem_base,
                                              const uint32_t v_smem, const uint32_t bias_a_smem, const uint32_t bias_b_smem,
                                              const UnitWalk walk) {
  using Cfg = FwdCfg<D>;
  constexpr uint32_t NV = Cfg::kStagesV;
  volatile int* abort_flag = &ctl->abort;
  // O = P.V : V is an MN-major operand; one group of MMAs with N = head_dim output columns
  constexpr uint32_t idesc_o = make_idesc_i8(D, true, true);
  constexpr uint32_t idesc_bias = make_idesc_bf16(D);
  const uint64_t d_bias_a = make_smem_desc_noswizzle(bias_a_smem, 128, 256);
  const uint64_t d_bias_b = make_smem_desc_noswizzle(bias_b_smem, 128, 256);
  const bool lead = elect_one();
  IssuerErr err;
  uint32_t g = 0;
  bool ok = true;
  for (int it = 0; it < walk.count && ok; ++it) {
    const int u = walk.unit(it);
    const int buf = it % kInfoBufs;
    if (!issuer_wait(err, smem_u32(&ctl->info_full[buf]), static_cast<uint32_t>((it / kInfoBufs) & 1), FMHA_I8_DEV_WAIT_INFO, it, abort_flag)) break;
    const int n_live = ctl->info[buf].n_live;
    __syncwarp();
    if (elect_one()) mbar_arrive(smem_u32(&ctl->info_empty[buf]));            // only the tile count is needed here
    for (int j = 0; j < n_live; ++j, ++g) {
      const uint32_t sb = g % SBufs<D>::n, stage = g % NV;
      uint64_t dv = make_smem_desc(v_smem + stage * Cfg::kTileBytes, D);
      const uint32_t tS = tmem_base + sb * kTile;
      uint32_t bar_o = smem_u32(&ctl->o_full[sb]), bar_v = smem_u32(&ctl->v_empty[stage]);
      uint32_t tP = PLayout<D>::kAnnex ? tmem_base + SBufs<D>::n * kTile + sb * PLayout<D>::kAnnexCols : tS;
      uint32_t tO = tS + PLayout<D>::kOOff;
      asm volatile("" : "+l"(dv), "+r"(tP), "+r"(tO), "+r"(bar_o), "+r"(bar_v));
      // V first (loaded steps ago), then P: the MMAs go out as soon as the last softmax warp has arrived
      if (!issuer_wait(err, smem_u32(&ctl->v_full[stage]), (g / NV) & 1u, FMHA_I8_DEV_WAIT_V_LOAD, g, abort_flag)) { ok = false; break; }
      if (!issuer_wait(err, smem_u32(&ctl->p_ready[g & 3u]), (g >> 2) & 1u, FMHA_I8_DEV_WAIT_P_READY, g, abort_flag)) { ok = false; break; }
      FMHA_STAMP(13, g);
      tc_fence_after();
      // The accumulator of this step is S(g)'s own buffer (free since the softmax threads have read S(g)), minus the
      // columns that hold P bytes at head_dim 64.
      if (lead) {
        mma_f16_ss(tO, d_bias_a, d_bias_b, idesc_bias, 0u);      // accumulator := 0x4B400000
#pragma unroll
        for (int kk = 0; kk < kTile / 32; ++kk)
          mma_i8_ts(tO, tP + PLayout<D>::p_col(kk), desc_advance(dv, kk * 32 * D), idesc_o, 1u);
        mma_commit(bar_o);
        mma_commit(bar_v);
      }
      FMHA_STAMP(14, g);
    }
  }
  if (err.code != 0u && elect_one()) raise_status(abort_flag, p.status, err.code, err.tile);
}

// Persistent kernel: gridDim.x = min(units, SMs) CTAs; CTA b processes units b, b + gridDim.x, ...  kFull: units shared by clusters and
// calibration too; without them the code is 47 KB instead of 60 (head_dim 128), which all but the longest calls feel, and the merge
// warps spill nothing.  us, with -> without: B64 H32 S256 D128 75.6 -> 71.7, B128 H16 S128 D128 29.5 -> 27.3, B4 H32 S1024 D128 58.4 -> 57.2, B1 H12 S320 D128
// 6.88 -> 6.35 and D64 6.23 -> 5.85, B6 H12 S512 D64 11.0 -> 10.5; B8 H32 S2048 D128 as before.
template <int D, bool kFull>
__global__ void __launch_bounds__(kFwdThreads, 1)
fmha_fwd_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k,
                const __grid_constant__ CUtensorMap map_v, const FwdParams p) {
  using Cfg = FwdCfg<D>;
  constexpr int NK = Cfg::kStagesK, NV = Cfg::kStagesV, NQ = Cfg::kQBufs;
  using Ctl = FwdCtl<NK, NV>;
  extern __shared__ uint8_t smem_raw[];
  // tiles need 1024-byte alignment (swizzle atoms); the launch reserves the slack
  // (pointer arithmetic on the shared array, not a round trip through an integer: the compiler then knows that everything
  // derived from it is shared memory and uses 32-bit shared-space loads and stores instead of generic ones)
  uint8_t* tiles = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
  uint8_t* bias_a = tiles + Cfg::kTilesBytesTotal;
  uint8_t* bias_b = bias_a + kBiasBytes;
  Ctl* ctl = reinterpret_cast<Ctl*>(bias_a + bias_bytes<D>());
  const uint32_t q_smem = smem_u32(tiles);
  const uint32_t k_smem = q_smem + NQ * Cfg::kTileBytes;
  const uint32_t v_smem = k_smem + NK * Cfg::kTileBytes;

  // The next launch of the stream may set itself up (barriers, tensor memory, constant operands: about 1.5 us with the
  // launch latency) on SMs this one leaves free, and waits below for this one to finish before it reads anything.
  grid_launch_dependents();
  const int warp = warp_index(), lane = threadIdx.x & 31;
  const int n_tiles = (p.S + kTile - 1) / kTile;
  const UnitWalk walk = unit_walk<kFull>(p);

  if (threadIdx.x == 0) {
    ctl->abort = 0;
    for (int w = 0; w < NQ; ++w) {
      mbar_init(smem_u32(&ctl->q_full[w]), 1);
      mbar_init(smem_u32(&ctl->q_empty[w]), 1);
    }
    for (int w = 0; w < 2; ++w)
      for (int q = 0; q < 4; ++q) mbar_init(smem_u32(&ctl->xch[w][q]), 64);
    for (int s = 0; s < SBufs<D>::n; ++s) {
      mbar_init(smem_u32(&ctl->s_full[s]), 1);
      mbar_init(smem_u32(&ctl->o_full[s]), 1);
      mbar_init(smem_u32(&ctl->s_free[s]), kMergeWarps * 32);
    }
    for (int s = 0; s < NK; ++s) {
      mbar_init(smem_u32(&ctl->k_full[s]), 1);
      mbar_init(smem_u32(&ctl->k_empty[s]), 1);
    }
    for (int s = 0; s < NV; ++s) {
      mbar_init(smem_u32(&ctl->v_full[s]), 1);
      mbar_init(smem_u32(&ctl->v_empty[s]), 1);
    }
    for (int s = 0; s < 4; ++s) mbar_init(smem_u32(&ctl->p_ready[s]), 8 * 32);
    for (int b = 0; b < kInfoBufs; ++b) {
      mbar_init(smem_u32(&ctl->info_full[b]), 1);
      mbar_init(smem_u32(&ctl->info_empty[b]), kInfoConsumers);
    }
    mbar_init(smem_u32(&ctl->early_full), 1);
    mbar_init_fence();
    tma_prefetch_desc(&map_q);
    tma_prefetch_desc(&map_k);
    tma_prefetch_desc(&map_v);
  }
  if (warp == 0) {
    __syncwarp();
    tmem_alloc(smem_u32(&ctl->tmem_base), kTmemCols);
    tmem_relinquish();
  }
  fill_bias_operands(bias_a, 1 + SBufs<D>::n);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *reinterpret_cast<volatile uint32_t*>(&ctl->tmem_base);
  volatile int* abort_flag = &ctl->abort;
  grid_dependency_wait();      // nothing above touches global memory

  // Every role walks the same unit sequence: `it` counts this CTA's units, info buffer = it % kInfoBufs,
  // phase of an info barrier = (it / kInfoBufs) & 1; `g` counts its steps (live key tiles) across units.
  if (warp >= kWarpSoftmax0) {
    setmaxnreg_dec<FwdRegs<D>::kSoftmax>();
    softmax_role<D>(p, ctl, tmem_base, walk);
  } else if (warp >= kWarpMerge0) {
    setmaxnreg_inc<FwdRegs<D>::kMerge>();
    merge_role<D, kFull>(p, ctl, tmem_base, tiles, walk);
  } else {
    if (FwdRegs<D>::kOther < kLaunchRegs) setmaxnreg_dec<FwdRegs<D>::kOther>();
    else if (FwdRegs<D>::kOther > kLaunchRegs) setmaxnreg_inc<FwdRegs<D>::kOther>();
    if (warp == kWarpLoad) {
      loader_role<D>(p, ctl, &map_q, &map_k, &map_v, q_smem, k_smem, v_smem, walk);
    } else if (warp == kWarpMmaS) {
      s_issuer_role<D>(p, ctl, tmem_base, q_smem, k_smem, bias_a, walk);
    } else if (warp == kWarpMmaO) {
      o_issuer_role<D>(p, ctl, tmem_base, v_smem, smem_u32(bias_a), smem_u32(bias_b), walk);
    } else if (warp == kWarpScan) {
      // ---------------------------------------------------------------- scanner: mask information, units ahead
      bool ok = true;
      for (int it = 0; it < walk.count && ok; ++it) {
        const int u = walk.unit(it);
        const int buf = it % kInfoBufs;
        // the buffer was used by unit it - kInfoBufs: wait until all its consumers have released it
        if (it >= kInfoBufs) {
          ok = __all_sync(0xFFFFFFFFu, mbar_wait(smem_u32(&ctl->info_empty[buf]), static_cast<uint32_t>(((it / kInfoBufs) - 1) & 1), abort_flag));
          if (!ok) { if (lane == 0) raise_status(abort_flag, p.status, FMHA_I8_DEV_WAIT_INFO, it); break; }
        }
        const UnitGeom geo = unit_geom(p, u);
        const int8_t* mask_row = p.mask + static_cast<int64_t>(geo.batch) * p.S;
        if (n_tiles <= 4) scan_few_tiles<4, false>(&ctl->info[buf], mask_row, p.S);
        else scan_mask_warp<false, 4>(&ctl->info[buf], mask_row, p.S, n_tiles);
        if (lane == 0) {
          const int n = ctl->info[buf].n_live, parts = it < walk.own ? 1 : p.parts, rank = static_cast<int>(blockIdx.x) % parts;
          ctl->info[buf].begin = n * rank / parts;
          ctl->info[buf].n_live = n * (rank + 1) / parts - n * rank / parts;
        }
        if (lane == 0) mbar_arrive(smem_u32(&ctl->info_full[buf]));
      }
    }
  }

  // every unit of this CTA has been computed and stored by the time the merge warps leave their loop
  tc_fence_before();
  if (!kFull || walk.count == walk.own) {      // (the same for all CTAs of a cluster)
    __syncthreads();
  } else {
    __syncwarp();
    cluster_arrive();          // every partial result of the unit is in shared memory
    cluster_wait();
    merge_parts<D>(p, smem_u32(ctl->part), smem_u32(tiles), walk.shared);
    __syncwarp();
    cluster_arrive();          // and stays there until everyone has read it
    cluster_wait();
  }
  if (warp == 0) {
    tc_fence_after();
    tmem_dealloc(tmem_base, kTmemCols);
  }
}

}  // namespace fmha
