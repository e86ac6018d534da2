// The forward kernel at head_dim 64 for calls with many query tiles (use_workers() in fmha_api.cu draws the line; the others,
// and head_dim 128, whose output row does not fit beside the scores, run fmha_fwd_sm100.cuh).  Same arithmetic, another
// division of the work:
//
//   worker  = four warps that do everything for a query tile of their own: row maximum, exponentials, the fp32 running row
//             and the epilogue, one thread per query row, nothing handed from thread to thread.  Four workers to a CTA, one CTA to
//             an SM; CTA c's units are c, c + grid, ..., and its workers take them as they finish.
//   driver  = one warp per worker: mask scan, TMA copies, S = Q.K^T, P.V.
//   tensor memory: 128 columns per worker.  S of a step; then its 8-bit P over the first 32 columns and P.V over the last 64.
//   key tiles with unmasked keys in one half only are 64 keys: S has 64 columns, the softmax threads read 64, P.V takes two of its
//             four steps.  B256 H16 S256 (lengths 64..256) -7 %, B64 H16 S320 -9 %, B64 H16 S64 -12 %.
//
// A worker's step is one serial chain -- S, maximum, exponentials, P.V, fold -- of 3600 cycles when it runs alone.  Four of them
// on an SM hide each other's latencies; nobody waits for a stage that other threads own, which is what bounds the other kernel
// on short sequences (its merge warps need 4500 cycles per unit of two steps whatever the other warps do).  What bounds this
// one: issue slots and the exponential unit, 64 % and 69 % busy on long sequences, where a step takes 5300 cycles, i.e. 1330 per
// SM.  An eighth of the exponentials is computed on the multiply-add pipe (all on the exponential unit: 2.5 % slower on
// B8 H32 S2048; a quarter: 3 % slower).  Pass 2 reads eight columns at a time: with sixteen the 104 registers of a softmax
// thread do not suffice, and the spills cost 4 to 9 %.
// Measured against the other kernel: see use_workers().
#pragma once
#include "fmha_fwd_sm100.cuh"

namespace fmha {
namespace w64 {
// kShort: for units of up to kShortTiles key tiles.  The maximum of a half tile branches off that of a whole one behind the first loads, or with
// kShort in front of them.  Behind, the step is faster, and the compiler spills values of the unit (-Xptxas -v: 72 bytes stored, 68 loaded, none in
// front), which short units pay for.  Behind against in front, per cent of the time: one and two tiles +1 to +2 where lengths differ, -1.5
// where they do not (B64 H16 S256); three tiles -1.4 to -3; long sequences -3.  (To be measured again when the step changes: what is spilled is
// the compiler's choice.)
// kCalib: calibration, apart from the forward pass because short units are the faster the smaller the code is.  It is 54 and 62 KB without
// calibration, 25 of it the drivers'; with all of it in one instance, long masks scanned in larger steps and units taken apart by divisions it
// was 74: B256 H16 S256 (64..256) 88.7 -> 85.1 us, B8 H32 S2048 335 -> 330.  (One copy of the driver per worker, 226 KB: 540.)
constexpr int kShortTiles = 2;
constexpr int kD = 64;
constexpr int kWorkers = 4;          // per CTA
// Warps: four softmax warps per worker (their number modulo 4 is their lane quarter of tensor memory), then one driver per worker.
constexpr int kSoftmaxWarps = 4 * kWorkers;
constexpr int kWarps = kSoftmaxWarps + kWorkers;
constexpr int kThreads = kWarps * 32;          // 640
constexpr int kInfoBufs = 4;         // units of a worker whose information is resident at once
// setmaxnreg moves registers inside the CTA's own launch allocation (registers per thread at launch x threads): a request
// that does not fit blocks forever.  640 threads start with 96 registers each (the host checks this).
constexpr int kLaunchRegs = 96;
constexpr int kSoftmaxRegs = 104, kDriverRegs = 64;
static_assert(kSoftmaxWarps * kSoftmaxRegs + kWorkers * kDriverRegs <= kWarps * kLaunchRegs,
              "setmaxnreg targets exceed the CTA's register allocation: the kernel would hang");
static_assert(kSoftmaxRegs >= kLaunchRegs && kDriverRegs <= kLaunchRegs, "the softmax warps gain registers, the drivers give");

constexpr int kTileBytes = kTile * kD;
constexpr int kWorkerBytes = 3 * kTileBytes;                   // K, V, Q
// A worker's tensor memory: 128 columns.  S of a step; then P over its first 32 columns and P.V over its last 64.
constexpr uint32_t kOCol = 64;

// What the workers need to know about a unit.
struct UnitInfo {
  int n_live;                         // key tiles with at least one unmasked key, never none; -1: there are no more units
  int last;                           // 1: no unit follows, of which the softmax warps then need not hear separately
  int rows;                           // query rows of the unit: 128, fewer in a head's last tile
  int64_t first_row;                  // of the slice's query rows, the unit's first
  uint8_t live[kMaxTiles];            // indices of the live key tiles, ascending
  uint8_t kind[kMaxTiles];            // their kinds (kTile...)
};
struct WorkerCtl {
  uint64_t q_full, k_full, v_full;    // the tiles have landed
  uint64_t early_full;                // the first unit's Q and K have, which are asked for before its mask is known
  uint64_t s_full, s_free;            // S has completed / its P.V has been drained
  uint64_t p_ready, o_full;           // P is written (and S consumed) / P.V has completed
  uint64_t info_full[kInfoBufs], info_empty[kInfoBufs];
  UnitInfo info[kInfoBufs];
};
struct Ctl {
  uint32_t tmem_base;
  int abort;
  int next;                           // how many of the CTA's units are taken
  WorkerCtl w[kWorkers];
};

// Operands of the preset MMA (see fill_bias_operands): A, B, and one B per worker for tiles with masked keys.  Only the first
// two of the K = 16 columns are not zero, so the second core matrix of every row group is one and the same stretch of zeros.
constexpr int kPresetBytes = kTile * 16;
constexpr int kPresets = 2 + kWorkers, kPresetBytesTotal = (kPresets + 1) * kPresetBytes;
__device__ __forceinline__ void fill_presets(uint8_t* preset) {
  for (int i = threadIdx.x; i < (kPresets + 1) * kTile; i += blockDim.x)
    reinterpret_cast<uint4*>(preset)[i] = make_uint4(i < kTile ? kBiasA : i < kPresets * kTile ? kBiasB : 0u, 0u, 0u, 0u);
  fence_proxy_async_smem();
}
__device__ __forceinline__ uint64_t preset_desc(uint32_t preset_smem, uint32_t operand) {
  return make_smem_desc_noswizzle(preset_smem + operand * kPresetBytes, (kPresets - operand) * kPresetBytes, 128);
}

constexpr size_t kSmemBytes = 1024 + kWorkers * kWorkerBytes + kPresetBytesTotal + sizeof(Ctl);

// Unit number `taken` of this CTA (unsigned: the first that does not exist may lie beyond the range of int).
__device__ __forceinline__ uint32_t cta_unit(int taken) { return blockIdx.x + gridDim.x * static_cast<uint32_t>(taken); }

// Largest of kChunks times 16 columns (biased integers), two loads in flight.
template <int kChunks>
__device__ __forceinline__ int columns_max(const uint32_t taddr) {
  int max_a = INT_MIN, max_b = INT_MIN;
  uint32_t ra[16], rb[16];
  tmem_ld16_issue(taddr, ra);
  tmem_ld16_issue(taddr + 16, rb);
#pragma unroll
  for (int c = 0; c < kChunks; c += 2) {
    tmem_ld_fence(ra); tmem_ld_fence(rb);
    chunk_max<16>(ra, max_a, max_b);
    if (c + 2 < kChunks) tmem_ld16_issue(taddr + (c + 2) * 16, ra);
    chunk_max<16>(rb, max_a, max_b);
    if (c + 2 < kChunks) tmem_ld16_issue(taddr + (c + 3) * 16, rb);
  }
  return max(max_a, max_b);
}

// ---------------------------------------------------------------------------------------------- softmax role
// One thread = one query row: its scores, probabilities, fp32 running output row, maximum and sum.
template <bool kShort, bool kCalib>
__device__ __forceinline__ void softmax_role(const FwdParams& p, Ctl* all, const int worker, const uint32_t tmem_base) {
  WorkerCtl* ctl = &all->w[worker];
  const int lane = threadIdx.x & 31, quad = warp_index() & 3;
  const int row = quad * 32 + lane;
  const uint32_t t_lane = tmem_base + (static_cast<uint32_t>(quad * 32) << 16);
  const uint32_t tS = t_lane + static_cast<uint32_t>(worker * kTile), tP = tS;
  volatile int* abort_flag = &all->abort;
  uint32_t g = 0;                               // steps so far
  auto or_fail = [&](bool waited, unsigned code) -> bool {
    if (!waited) raise_status(abort_flag, p.status, code, g);
    return waited;
  };
  int announced = 1;
  // The running row is never cleared: the first tile of a unit multiplies what the unit before has left by zero.
  float2 o2[kD / 2];
#pragma unroll
  for (int i = 0; i < kD / 2; ++i) o2[i] = make_float2(0.f, 0.f);
#pragma unroll 1
  for (int it = 0; it < announced; ++it) {
    const int buf = it % kInfoBufs;
    // (this wait and P.V's are long while the driver goes through units without keys)
    if (!or_fail(warp_wait_long(smem_u32(&ctl->info_full[buf]), static_cast<uint32_t>((it / kInfoBufs) & 1), abort_flag), FMHA_I8_DEV_WAIT_INFO)) return;
    const int n_live = ctl->info[buf].n_live;
    if (n_live < 0) continue;
    announced += 1 - ctl->info[buf].last;
    float m_run = -INFINITY, l_run = 0.f;
    // this thread's output row, -1 past the last row of the head (looked up where it is needed: nothing of it stays in registers)
    auto output_row = [&]() -> int64_t { return row < ctl->info[buf].rows ? ctl->info[buf].first_row + row : -1; };

#pragma unroll 1
    for (int j = 0; j < n_live; ++j, ++g) {
      const bool whole = (ctl->info[buf].kind[j] & kTileHalf) == 0;      // 128 columns of scores, or 64
      if (!or_fail(warp_wait(smem_u32(&ctl->s_full), g & 1u, abort_flag), FMHA_I8_DEV_WAIT_S_READY)) return;
      tc_fence_after();
      FMHA_STAMP(quad == 0 ? worker * 4 + 0 : 47, g);
      // ---- pass 1: biased integer maximum of the row (inc/fmha_i8.cuh:183-206)
      int imax;
      if constexpr (kShort) {
        imax = whole ? columns_max<8>(tS) : columns_max<4>(tS);
      } else {
        uint32_t ra[16], rb[16];
        int max_a = INT_MIN, max_b = INT_MIN;
        auto two_chunks = [&]() {
          tmem_ld_fence(ra); tmem_ld_fence(rb);
          chunk_max<16>(ra, max_a, max_b);
          chunk_max<16>(rb, max_a, max_b);
        };
        auto two_chunks_and_next = [&](int next) {
          tmem_ld_fence(ra); tmem_ld_fence(rb);
          chunk_max<16>(ra, max_a, max_b);
          tmem_ld16_issue(tS + next * 16, ra);
          chunk_max<16>(rb, max_a, max_b);
          tmem_ld16_issue(tS + next * 16 + 16, rb);
        };
        tmem_ld16_issue(tS, ra);
        tmem_ld16_issue(tS + 16, rb);
        two_chunks_and_next(2);
        if (whole) {
          two_chunks_and_next(4);
          two_chunks_and_next(6);
          two_chunks();
        } else {
          two_chunks();
        }
        imax = max(max_a, max_b);
      }
      const RowConsts k = row_consts(imax, p.c2, p.row_scale, p.scale_qk, p.p_mul);
      FMHA_STAMP(quad == 0 ? worker * 4 + 1 : 47, g);

      // ---- pass 2: exp, row sum, requantise (inc/fmha_i8.cuh:208-253); the bytes go over columns already consumed
      float2 sum[2] = {make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
      uint32_t sa[8], sb[8], packed[2];
      auto sixteen = [&](uint32_t c, auto more) {           // columns 8 c to 8 c + 15; the first eight are in flight
        tmem_ld_fence(sa);
        tmem_ld8_issue(tS + (c + 1) * 8, sb);
        chunk_exp_pack<8>(sa, k.c2, k.neg_hi, k.p_mul_f, sum, packed);
        tmem_st2(tP + c * 2, packed);
        tmem_ld_fence(sb);
        if (decltype(more)::value) tmem_ld8_issue(tS + (c + 2) * 8, sa);
        chunk_exp_pack<8, false, 1>(sb, k.c2, k.neg_hi, k.p_mul_f, sum, packed);
        tmem_st2(tP + c * 2 + 2, packed);
      };
      constexpr Flight<1> more;
      constexpr Flight<0> last;
      tmem_ld8_issue(tS, sa);
      if (whole) {
#pragma unroll
        for (uint32_t c = 0; c < 14; c += 2) sixteen(c, more);
        sixteen(14, last);
      } else {
#pragma unroll
        for (uint32_t c = 0; c < 6; c += 2) sixteen(c, more);
        sixteen(6, last);
      }
      tmem_wait_st();
      tc_fence_before();
      mbar_arrive(smem_u32(&ctl->p_ready));
      FMHA_STAMP(quad == 0 ? worker * 4 + 2 : 47, g);

      // ---- merge of tile statistics (inc/fmha_i8.cuh:301-304), while P.V is under way
      const float l_tile = k.f * ((sum[0].x + sum[0].y) + (sum[1].x + sum[1].y));
      const float m_new = fmaxf(m_run, k.m_tile);
      const float e_old = __expf(m_run - m_new);                       // 0 on the first tile (m_run = -inf)
      const float e_cur = clear_low2(__expf(k.m_tile - m_new));        // 22 significant bits: kMagic*e_cur is exact
      l_run = fmaf(e_old, l_run, e_cur * l_tile);
      m_run = m_new;
      const float2 e_cur2 = make_float2(e_cur, e_cur), e_bias = make_float2(-e_cur * kMagic, -e_cur * kMagic);
      const float2 e_old2 = make_float2(e_old, e_old);

      // ---- P.V of this step into the running row (inc/fmha_i8.cuh:306-310)
      if (!or_fail(warp_wait_long(smem_u32(&ctl->o_full), g & 1u, abort_flag), FMHA_I8_DEV_WAIT_O_READY)) return;
      tc_fence_after();
      FMHA_STAMP(quad == 0 ? worker * 4 + 3 : 47, g);
      // (two loads in flight: a round trip to tensor memory costs more than folding a chunk in)
      uint32_t ra[16], rb[16];
      tmem_ld16_issue(tS + kOCol, ra);
      tmem_ld16_issue(tS + kOCol + 16, rb);
      tmem_ld_fence(ra); tmem_ld_fence(rb);
      drain_chunk<16>(ra, o2, e_cur2, e_bias, e_old2);
      tmem_ld16_issue(tS + kOCol + 32, ra);
      drain_chunk<16>(rb, o2 + 8, e_cur2, e_bias, e_old2);
      tmem_ld16_issue(tS + kOCol + 48, rb);
      tmem_ld_fence(ra); tmem_ld_fence(rb);
      // the last columns are in registers: the driver may go on with the next S
      tc_fence_before();
      mbar_arrive(smem_u32(&ctl->s_free));
      drain_chunk<16>(ra, o2 + 16, e_cur2, e_bias, e_old2);
      drain_chunk<16>(rb, o2 + 24, e_cur2, e_bias, e_old2);
    }

    // ---- the unit is finished
    const int64_t out_row = output_row();
    __syncwarp();
    if (lane == 0) mbar_arrive(smem_u32(&ctl->info_empty[buf]));
    const float inv = l_run > 0.f ? __frcp_rn(l_run) : 0.f;
    if (kCalib) {
      // calibration: only the largest magnitude of the unquantised output is wanted (the reference takes o_amax from its
      // fp32 CPU result, test_fmha_i8.cpp:161); non-negative floats order like their bit patterns
      float mx = 0.f;
#pragma unroll
      for (int i = 0; i < kD / 2; ++i) mx = fmaxf(mx, fmaxf(fabsf(o2[i].x * inv), fabsf(o2[i].y * inv)));
      const unsigned bits = __reduce_max_sync(0xFFFFFFFFu, __float_as_uint(out_row >= 0 ? mx * p.amax_scale : 0.f));
      if (lane == 0 && bits != 0u) atomicMax(reinterpret_cast<unsigned*>(p.amax_out), bits);
      continue;
    }
    // normalise, requantise, store (inc/fmha_i8.cuh:318-332)
    const float scale = p.scale_v_out * inv;
    // (the clamp only where a warp has an output beyond 127: B256 H16 S256 with lengths 64..256 -1.7 %, B200 H12 S128 -3.5 %)
    const bool clamp = __any_sync(0xFFFFFFFFu, needs_clamp<kD / 2>(o2, scale));
    if (out_row >= 0) {
      int8_t* dst = p.o + out_row * kD;
#pragma unroll
      for (int c = 0; c < kD / 32; ++c) {
        uint32_t wide[8];
        requantise16(o2 + c * 16, make_float2(scale, scale), clamp, wide);
        requantise16(o2 + c * 16 + 8, make_float2(scale, scale), clamp, wide + 4);
        // 32-byte stores: a warp's rows are 64 bytes apart, so every store touches 32 lines whatever its width
        if (p.o_wide) {
          st_global_v8(dst + c * 32, wide);
        } else {
          *reinterpret_cast<uint4*>(dst + c * 32) = make_uint4(wide[0], wide[1], wide[2], wide[3]);
          *reinterpret_cast<uint4*>(dst + c * 32 + 16) = make_uint4(wide[4], wide[5], wide[6], wide[7]);
        }
      }
    }
  }
}

// ---------------------------------------------------------------------------------------------- driver
// One warp per worker, run warp-wide (every lane waits and counts, one elected lane issues).  Per step: S, then -- while the
// softmax warps work -- V of the step, the mask scan and, S having completed, K (and Q) of the step after it, then P.V.  A
// worker has one tile of each: a step is long enough (3600 cycles at least) to hide a load behind it, and no barrier guards
// the reuse of a tile, which the driver itself has seen used.
struct DriverStep {
  int tile;                  // key tile, -1: no more steps
  int kind;                  // its kind (kTile...)
  bool first;                // of its unit
  int bh, batch;
};
template <bool kEarlyK, bool kCalib>
__device__ __forceinline__ void driver_role(const FwdParams& p, Ctl* all, const int worker, const CUtensorMap* map_q, const CUtensorMap* map_k,
                                            const CUtensorMap* map_v, const uint32_t tmem_base, const uint32_t worker_smem, uint8_t* presets) {
  WorkerCtl* ctl = &all->w[worker];
  volatile int* abort_flag = &all->abort;
  const int lane = threadIdx.x & 31;
  const uint32_t tS = tmem_base + static_cast<uint32_t>(worker * kTile), tO = tS + kOCol;
  const uint32_t k_smem = worker_smem, v_smem = worker_smem + kTileBytes, q_smem = worker_smem + 2 * kTileBytes;
  constexpr uint32_t idesc_s = make_idesc_i8(kTile, false);       // S = Q.K^T : N = 128 keys, both K-major
  constexpr uint32_t idesc_half = make_idesc_i8(kTile / 2, false), idesc_preset_half = make_idesc_bf16(kTile / 2);
  constexpr uint32_t idesc_preset_s = make_idesc_bf16(kTile), idesc_preset_o = make_idesc_bf16(kD);
  constexpr uint32_t idesc_o = make_idesc_i8(kD, true, true);     // P.V : P unsigned, V an MN-major operand
  const uint32_t preset_smem = smem_u32(presets);
  const uint64_t d_a = preset_desc(preset_smem, 0), d_b = preset_desc(preset_smem, 1);
  const uint64_t dq = make_smem_desc(q_smem, kD), dk = make_smem_desc(k_smem, kD), dv = make_smem_desc(v_smem, kD);
  const int n_tiles = (p.S + kTile - 1) / kTile;
  const bool lead = elect_one();
  uint32_t fail = 0u, g = 0, units = 0;
  auto wait = [&](uint32_t bar, uint32_t parity, uint32_t code) -> bool {
    if (warp_wait(bar, parity, abort_flag)) return true;
    fail = code;
    return false;
  };

  int taken = worker;                         // number of the unit to begin with; -1: ask for one
  bool last = false;                          // the unit handed out last is known to be the last
  int it = -1, j = 0, n_live = 0;
  uint32_t u = 0u;                            // the unit of the step handed out last
  int bh = 0, batch = 0, q_row0 = 0;          // its head, sequence and first query row
  // The results of rows without an unmasked key.  (Not unrolled: 1 KB of code.)
  auto empty_unit = [&](int rows, int64_t first_row) {
    if (!kCalib) {
      uint4* dst = reinterpret_cast<uint4*>(p.o + first_row * kD);
#pragma unroll 1
      for (int i = lane; i < rows * (kD / 16); i += 32) dst[i] = make_uint4(0u, 0u, 0u, 0u);
    }
  };
  auto next_step = [&]() -> DriverStep {
    constexpr DriverStep none{-1, 0, false, 0, 0};
    while (j >= n_live) {
      if (n_live < 0 || last) return none;
      // The workers of a CTA take its units as they finish: with a fixed stride all wait for the one with the most tiles (B32 H12 S1024,
      // lengths 300..1024, -6 %; B256 H16 S256, 64..256, -3 %).
      if (taken < 0) {
        if (lane == 0) taken = atomicAdd(&all->next, 1);
        taken = uniform(taken);
      }
      u = cta_unit(taken);
      taken = -1;
      const int buf = ++it % kInfoBufs;
      if (it >= kInfoBufs && !wait(smem_u32(&ctl->info_empty[buf]), static_cast<uint32_t>(((it / kInfoBufs) - 1) & 1), FMHA_I8_DEV_WAIT_INFO)) return none;
      UnitInfo* info = &ctl->info[buf];
      if (u >= static_cast<uint32_t>(p.n_units)) {
        n_live = -1;
        if (elect_one()) {
          info->n_live = -1;
          mbar_arrive(smem_u32(&ctl->info_full[buf]));
        }
        return none;
      }
      bh = fast_div(static_cast<int>(u), p.by_q_tiles);
      batch = fast_div(p.bh_begin + bh, p.by_heads);
      q_row0 = (static_cast<int>(u) - bh * p.q_tiles) * kTile;
      const int8_t* mask_row = p.mask + static_cast<int64_t>(batch) * p.S;
      if (kEarlyK) scan_few_tiles<2, true>(info, mask_row, p.S);
      else if (n_tiles <= 4) scan_few_tiles<4, true>(info, mask_row, p.S);
      else scan_mask_warp<true, 2>(info, mask_row, p.S, n_tiles);
      if (info->n_live == 0) {
        // Nobody else hears of a unit without keys: this warp is the one that P.V of the step before is waiting for, and may not wait
        // until the softmax warps have got through a row of such units.
        empty_unit(min(kTile, p.Sq - q_row0), static_cast<int64_t>(bh) * p.Sq + q_row0);
        --it;
        continue;
      }
      // All units are taken when the counter says so.  A call of one round of workers knows it from the beginning, and need not ask for
      // another unit nor announce that there is none while P.V of its last step waits: -0.3 to -1 % for calls of one round, B256 H16 S256
      // (64..256) -1 %.
      last = uniform(cta_unit(*reinterpret_cast<volatile int*>(&all->next)) >= static_cast<uint32_t>(p.n_units));
      if (elect_one()) {
        info->last = last ? 1 : 0;
        info->rows = min(kTile, p.Sq - q_row0);
        info->first_row = static_cast<int64_t>(bh) * p.Sq + q_row0;
      }
      __syncwarp();
      if (elect_one()) mbar_arrive(smem_u32(&ctl->info_full[buf]));
      n_live = info->n_live;
      j = 0;
    }
    const UnitInfo* info = &ctl->info[it % kInfoBufs];
    const DriverStep s{info->live[j], info->kind[j], j == 0, bh, batch};
    ++j;
    return s;
  };
  auto load_k = [&](const DriverStep& s) {
    if (s.tile >= 0 && elect_one()) {
      mbar_arrive_expect_tx(smem_u32(&ctl->k_full), kTileBytes);
      tma_load_3d(k_smem, map_k, smem_u32(&ctl->k_full), 0, s.tile * kTile, bh);
      if (s.first) {
        mbar_arrive_expect_tx(smem_u32(&ctl->q_full), kTileBytes);
        tma_load_3d(q_smem, map_q, smem_u32(&ctl->q_full), 0, q_row0, bh);
      }
    }
    __syncwarp();
  };

  // The first unit's Q rows, and with few key tiles to a unit its first K tile, are asked for while its mask is still on the way.  Both
  // with many key tiles: B8 H16 S512 18.1 -> 18.3 us.  Neither: B32 H12 S512 (256..512) 36.7 -> 37.4.
  // Only Q with few: B200 H12 S128 22.6 -> 22.8.
  const uint32_t first = cta_unit(worker);
  const bool early = first < static_cast<uint32_t>(p.n_units);
  if (early && elect_one()) {
    const int head = fast_div(static_cast<int>(first), p.by_q_tiles);
    mbar_arrive_expect_tx(smem_u32(&ctl->early_full), kEarlyK ? 2 * kTileBytes : kTileBytes);
    tma_load_3d(q_smem, map_q, smem_u32(&ctl->early_full), 0, (static_cast<int>(first) - head * p.q_tiles) * kTile, head);
    if (kEarlyK) tma_load_3d(k_smem, map_k, smem_u32(&ctl->early_full), 0, 0, head);
  }
  __syncwarp();
  DriverStep cur = next_step();
  if (early) wait(smem_u32(&ctl->early_full), 0u, FMHA_I8_DEV_WAIT_Q_LOAD);
  if (cur.tile >= 0 && u == first && (!kEarlyK || cur.tile == 0)) {
    if (elect_one()) {
      if (kEarlyK) {
        mbar_arrive(smem_u32(&ctl->k_full));
      } else {
        mbar_arrive_expect_tx(smem_u32(&ctl->k_full), kTileBytes);
        tma_load_3d(k_smem, map_k, smem_u32(&ctl->k_full), 0, cur.tile * kTile, bh);
      }
      mbar_arrive(smem_u32(&ctl->q_full));
    }
    __syncwarp();
  } else {
    load_k(cur);
  }
  while (cur.tile >= 0 && fail == 0u) {
    const bool mixed = (cur.kind & kTileMixed) != 0, whole = (cur.kind & kTileHalf) == 0;
    const uint32_t row0 = (cur.kind & kTileUpper) != 0 ? kTile / 2 : 0u;          // first row in use of the K and V tiles
    bool masked[4] = {};
    if (mixed) {
      const int8_t* mask_row = p.mask + static_cast<int64_t>(cur.batch) * p.S;
      const int key0 = cur.tile * kTile + static_cast<int>(row0) + lane;
#pragma unroll
      for (int i = 0; i < 4; ++i) masked[i] = key0 + 32 * i >= p.S || mask_row[key0 + 32 * i] != 0;
    }
    // What the MMAs need is formed and kept in registers before the waits that they follow (the compiler would form it where it is used): 120 of the
    // 290 cycles from S's buffer being free to its last instruction.  B8 H32 S2048 334.7 -> 332.6 us, B256 H16 S256 (64..256) 86.7 -> 85.7, B32 H12 S512
    // (256..512) 36.3 -> 36.0.  (The instructions under a predicate instead of a branch: +2 %.)
    // The tile's preset operand: the common one, or this worker's own, which nothing has read since the last S.
    const uint32_t operand = mixed ? 2u + static_cast<uint32_t>(worker) : 1u;
    if (mixed) fill_mask_operand(presets + operand * kPresetBytes, masked, 128);
    uint64_t d_preset = preset_desc(preset_smem, operand), d_k = desc_advance(dk, row0 * kD), d_v = desc_advance(dv, row0 * kD);
    uint32_t idesc_preset = whole ? idesc_preset_s : idesc_preset_half, idesc = whole ? idesc_s : idesc_half;
    asm volatile("" : "+l"(d_preset), "+l"(d_k), "+l"(d_v), "+r"(idesc_preset), "+r"(idesc));
    if (cur.first && !wait(smem_u32(&ctl->q_full), units++ & 1u, FMHA_I8_DEV_WAIT_Q_LOAD)) break;
    if (!wait(smem_u32(&ctl->k_full), g & 1u, FMHA_I8_DEV_WAIT_K_LOAD)) break;
    if (g > 0u && !wait(smem_u32(&ctl->s_free), (g - 1u) & 1u, FMHA_I8_DEV_WAIT_O_FREE)) break;
    tc_fence_after();
    FMHA_STAMP(16 + worker * 4 + 0, g);
    if (lead) {
      mma_f16_ss(tS, d_a, d_preset, idesc_preset, 0u);        // accumulator := 0x4B400000, masked keys -2^127
#pragma unroll
      for (int kk = 0; kk < kD / 32; ++kk) mma_i8_ss(tS, desc_advance(dq, kk * 32), desc_advance(d_k, kk * 32), idesc, 1u);
      mma_commit(smem_u32(&ctl->s_full));
      mbar_arrive_expect_tx(smem_u32(&ctl->v_full), kTileBytes);
      tma_load_3d(v_smem, map_v, smem_u32(&ctl->v_full), 0, cur.tile * kTile, cur.bh);
    }
    FMHA_STAMP(16 + worker * 4 + 1, g);
    const DriverStep next = next_step();
    if (fail != 0u || !wait(smem_u32(&ctl->s_full), g & 1u, FMHA_I8_DEV_WAIT_S_READY)) break;
    load_k(next);
    if (!wait(smem_u32(&ctl->v_full), g & 1u, FMHA_I8_DEV_WAIT_V_LOAD)) break;
    if (!wait(smem_u32(&ctl->p_ready), g & 1u, FMHA_I8_DEV_WAIT_P_READY)) break;
    tc_fence_after();
    FMHA_STAMP(16 + worker * 4 + 2, g);
    if (lead) {
      mma_f16_ss(tO, d_a, d_b, idesc_preset_o, 0u);
#pragma unroll
      for (int kk = 0; kk < kTile / 64; ++kk) mma_i8_ts(tO, tS + kk * 8, desc_advance(d_v, kk * 32 * kD), idesc_o, 1u);
      if (whole) {
#pragma unroll
        for (int kk = kTile / 64; kk < kTile / 32; ++kk) mma_i8_ts(tO, tS + kk * 8, desc_advance(dv, kk * 32 * kD), idesc_o, 1u);
      }
      mma_commit(smem_u32(&ctl->o_full));
    }
    FMHA_STAMP(16 + worker * 4 + 3, g);
    cur = next;
    ++g;
  }
  if (fail != 0u) {
    if (elect_one()) raise_status(abort_flag, p.status, fail, g);
    // unwinding: let copies that are still in flight land before the CTA may exit
    const long long t0 = clock64();
    while (clock64() - t0 < 2000000LL) { /* about a millisecond */ }
  }
}

template <bool kShort, bool kCalib>
__global__ void __launch_bounds__(kThreads, 1)
fwd_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k, const __grid_constant__ CUtensorMap map_v,
           const FwdParams p) {
  extern __shared__ uint8_t smem_raw[];
  // The next launch of the stream may set itself up on SMs this one leaves free, and waits below for this one to finish
  // before it reads anything.
  grid_launch_dependents();
  // tiles need 1024-byte alignment (swizzle atoms); the launch reserves the slack (pointer arithmetic on the shared array:
  // the compiler then knows that everything derived from it is shared memory)
  uint8_t* tiles = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
  uint8_t* presets = tiles + kWorkers * kWorkerBytes;
  Ctl* ctl = reinterpret_cast<Ctl*>(presets + kPresetBytesTotal);
  const int warp = warp_index();
  if (threadIdx.x == 0) {
    ctl->abort = 0;
    ctl->next = kWorkers;
    for (WorkerCtl& w : ctl->w) {
      mbar_init(smem_u32(&w.q_full), 1);
      mbar_init(smem_u32(&w.k_full), 1);
      mbar_init(smem_u32(&w.v_full), 1);
      mbar_init(smem_u32(&w.early_full), 1);
      mbar_init(smem_u32(&w.s_full), 1);
      mbar_init(smem_u32(&w.s_free), kTile);
      mbar_init(smem_u32(&w.p_ready), kTile);
      mbar_init(smem_u32(&w.o_full), 1);
      for (int b = 0; b < kInfoBufs; ++b) {
        mbar_init(smem_u32(&w.info_full[b]), 1);
        mbar_init(smem_u32(&w.info_empty[b]), 4);
      }
    }
    mbar_init_fence();
    tma_prefetch_desc(&map_q);
    tma_prefetch_desc(&map_k);
    tma_prefetch_desc(&map_v);
  }
  if (warp == kWarps - 1) {
    __syncwarp();
    tmem_alloc(smem_u32(&ctl->tmem_base), kTmemCols);
    tmem_relinquish();
  }
  fill_presets(presets);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *reinterpret_cast<volatile uint32_t*>(&ctl->tmem_base);
  grid_dependency_wait();      // nothing above touches global memory

  const int worker = warp < kSoftmaxWarps ? warp >> 2 : warp - kSoftmaxWarps;
  uint8_t* worker_smem = tiles + worker * kWorkerBytes;
  if (warp < kSoftmaxWarps) {
    setmaxnreg_inc<kSoftmaxRegs>();
    w64::softmax_role<kShort, kCalib>(p, ctl, worker, tmem_base);
  } else {
    setmaxnreg_dec<kDriverRegs>();
    driver_role<kShort, kCalib>(p, ctl, worker, &map_q, &map_k, &map_v, tmem_base, smem_u32(worker_smem), presets);
  }
  tc_fence_before();
  __syncthreads();
  if (warp == kWarps - 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, kTmemCols);
  }
}

}  // namespace w64
}  // namespace fmha
