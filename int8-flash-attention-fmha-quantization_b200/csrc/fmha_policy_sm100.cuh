// The whole-row P scaling policies (fmha_i8_sm100_infer_policy; the reference's accuracy study, fmha_i8_quant_deviation.py:57-121) in one
// launch.  A row's scale is known only when all its keys have been seen, so every unit (128 query rows of one head) goes over its keys
// twice: phase 1 forms the scores and keeps their maximum (static policy: and the exp-sum), phase 2 forms them again, with the
// probabilities in bytes and P.V.  What one scale per row changes against the plain forward pass:
//
//   - the sums of P.V over all keys are whole numbers below 127 * 128 * 32768 = 2^29: they stay in tensor memory, in the integer
//     accumulator, until the row is done.  No step drains a partial output, no thread holds one.
//   - a step needs no maximum of its own, so it can be any number of keys: 64, whose scores leave room for the sums beside them.
//
//   worker  = the warps of one unit, two to a CTA: two threads per query row, each with every other group of 64 keys (its chain), a
//             loader warp (mask scan, TMA copies) and an issuer warp (S = Q.K^T, P.V).
//   tensor memory of a worker, 256 columns: buffers of 64 columns of scores, three at head_dim 64 and two at 128, each with its group's P
//             bytes over the first 16 of them; then the sums of P.V.  In phase 1 a step is a group for each chain, in columns [0, 128) and
//             [128, 256) in turn.
//
// What bounds it: the exponential unit in phase 2 (with two units to an SM 1130 cycles for 128 x 128 scores, 1024 of exponentials; an eighth of them go to
// the multiply-add pipe, 4 to 8 % of the time at both head_dims), the chain of one issuer per worker in phase 1.  An issuer's instructions
// follow one another, so what it takes together shares a barrier (a wait for K and one for V: 25.6 us instead of 19.5 with one unit to an SM, B1 H4
// S2048).
// us, as two launches of the forward kernels -> here: per-row B4 H16 S1024 D64 (512..1024 keys) 35.1 -> 24.6, B64 H16 S256 46.0 -> 33.1, B1 H32
// S2048 70.8 -> 53.2, B1 H2 S64 7.2 -> 4.5, D128 B8 H16 S512 31.6 -> 20.8, B2 H32 S2048 155 -> 117; static the first 45.1 -> 35.6, D128 B8 H16 S512
// 35.9 -> 28.2; one unit to an SM, static, B1 H2 S8192 D64 107.0 -> 98.7, D128 108.9 -> 108.1, eight units of 16,384 keys at head_dim 128 207.8 -> 206.5.
// (The static policy's sum with constants of its own for each group, and a quarter of its exponentials on the multiply-add pipe in two of four
// chunks instead of in all: 37.3 for the first, B1 H2 Sq1 Sk32768 D64 399.9 instead of 375.8, D128 424.5 instead of 401.3; its clip by minima instead
// of by multiplications that saturate: 35.8, 375.5 instead of 364.9, 401.3 instead of 394.9; two launches 384 and 404.)
// (Four workers of one thread per row with one buffer of 64 columns each: 28.6 for the first, 2650 cycles of which 900 go by between the last
// exponential of a group and the first of the next.)
#pragma once
#include "fmha_fwd_sm100.cuh"

namespace fmha {
namespace wholerow {
constexpr float kLevels = 127.f;               // quantisation levels of P in the reference's study
constexpr int kKeys = 64;                      // keys of a step
constexpr int kMaxGroups = kMaxSeq / kKeys;
constexpr int kSoftmaxWarps = 16;
constexpr int kInfoBufs = 2, kQBufs = 2, kMaxStages = 8;
constexpr uint16_t kMixed = 0x8000;            // the group has masked keys

constexpr int kChains = 2, kWorkers = 2;
constexpr int kThreads = 32 * (kSoftmaxWarps + 2 * kWorkers);
// setmaxnreg moves registers inside the CTA's own launch allocation (a request beyond it blocks forever; the host checks the launch's)
constexpr int kLaunchRegs = 96, kSoftmaxRegs = 104, kOtherRegs = 64;
static_assert(kSoftmaxWarps * kSoftmaxRegs + 2 * kWorkers * kOtherRegs <= kThreads / 32 * kLaunchRegs, "setmaxnreg targets exceed the CTA's registers");
constexpr int kCols = 512 / kWorkers;          // of tensor memory per worker
constexpr int kStep1 = kKeys * kChains;        // keys, and columns, of a step of phase 1
// Position in a ring of N places, and the parity of the round.
template <uint32_t N> struct Ring {
  uint32_t at = 0u, parity = 0u;
  template <uint32_t kBy = 1> __device__ __forceinline__ void advance() {
    at += kBy;
    if (at >= N) { at -= N; parity ^= 1u; }
  }
  __device__ __forceinline__ void skip(uint32_t by) {
    at += by;
    parity ^= (at / N) & 1u;
    at %= N;
  }
};

template <int D> struct Cfg {
  static constexpr uint32_t kBufs = (kCols - D) / kKeys;
  static constexpr int kOutCol = kCols - D;              // first column of the sums
  static constexpr int kOutCols = D / kChains;           // output columns of a thread
  static constexpr int kGroupBytes = kKeys * D, kQBytes = kTile * D;
  // One ring for K and V, whose places hold what the issuer takes together: two groups of K (phase 1), or V of a group and K of the group
  // that is kBufs later (phase 2).
  static constexpr uint32_t kStages = D == 64 ? 8 : 4;
  static constexpr int kStageBytes = 2 * kGroupBytes;
  static constexpr int kWorkerBytes = kQBufs * kQBytes + static_cast<int>(kStages) * kStageBytes;
};

struct UnitInfo {
  int n;                              // groups with at least one unmasked key, never none; -1: there are no more units
  int first_mixed;                    // the first of them with masked keys too, n if none has
  int rows;                           // query rows: 128, fewer in a head's last unit
  int64_t first_row;                  // of the slice's query rows, the unit's first
  const int8_t* mask_row;
  uint16_t group[kMaxGroups];         // indices of those groups, ascending, with kMixed
};
struct WorkerCtl {
  uint64_t q_full[kQBufs], q_empty[kQBufs];                              // Q rows have landed / the unit's last S has completed
  uint64_t full[kMaxStages], empty[kMaxStages];                          // a place of the ring has landed / has been multiplied
  uint64_t max_full[2], max_free[2];                                     // phase 1: scores are there / have been read
  uint64_t s_full[3], p_ready[3];                                        // phase 2, per buffer: scores are there / P is, and the scores have been read
  uint64_t p_brief[kChains];                                             // kBrief, per group: P is there
  uint64_t o_full, o_free;                                               // the sums are complete / have been read
  uint64_t xch[4];                                                       // per lane quarter: both threads of a row have left their values
  uint64_t info_full[kInfoBufs], info_empty[kInfoBufs];
  float2 stat[2][kChains][kTile];                                        // what the threads of a row tell each other, by parity of the unit
  float sum[2][kChains][kTile];
  UnitInfo info[kInfoBufs];
};
struct Ctl {
  uint32_t tmem_base;
  int abort;
  int next;                           // how many of the CTA's units are taken
  WorkerCtl w[kWorkers];
};

// Operands of the preset MMA (see fill_bias_operands): A, the common B, and four B per worker for groups with masked keys.  Only the
// first two of the K = 16 columns are not zero, so the second core matrix of every row group is one and the same stretch of zeros.
constexpr int kOwnOperands = 4, kOperands = kOwnOperands * kWorkers, kOperandBytes = kKeys * 16, kABytes = kTile * 16;
constexpr int kPresetBytes = kABytes + (1 + kOperands) * kOperandBytes + kABytes;
__device__ __forceinline__ void fill_presets(uint8_t* preset) {
  constexpr int kB = kABytes / 16, kZero = kB + (1 + kOperands) * kOperandBytes / 16;
  for (int i = threadIdx.x; i < kPresetBytes / 16; i += blockDim.x)
    reinterpret_cast<uint4*>(preset)[i] = make_uint4(i < kB ? kBiasA : i < kZero ? kBiasB : 0u, 0u, 0u, 0u);
  fence_proxy_async_smem();
}
__device__ __forceinline__ uint64_t preset_desc(uint32_t preset_smem, uint32_t offset) {
  return make_smem_desc_noswizzle(preset_smem + offset, kPresetBytes - kABytes - offset, 128);
}
constexpr uint32_t kCommonB = kABytes, kOwnB = kABytes + kOperandBytes;

template <int D> constexpr size_t smem_bytes() { return 1024 + kWorkers * Cfg<D>::kWorkerBytes + kPresetBytes + sizeof(Ctl); }

// kBrief: the static policy's calls of no more groups than chains.  A thread has one group at the most, forms its exponentials once, in terms of
// the group's own maximum, keeps them, and makes them bytes when the exchange has told it what they are worth: no second S, no second pass
// over the keys.  In two phases such units are bound by their chain of dependent steps, and an SM has two units only: with many of them two
// launches of the forward kernels were faster.  us, those -> two phases -> this, B512 H16 S128 D64 110.5 -> 113.7 -> 84.0, with 64..128 keys 110.6
// -> 116.8 -> 87.4, 16 query rows 102.9 -> 111.6 -> 82.1, 16384 units of S64 with one row 137.8 -> 147.0 -> 113.1, B512 H16 S128 D128 190 -> 139 -> 109.
// (The exponentials left in tensor memory meanwhile, which spills nothing instead of some 30 bytes: 92.4 for the first.  Both forms in one
// instance: the longer units lose 4 to 8 %.)
// Sixteen scores to their exponentials, in place, and into the sums; a quarter of them on the multiply-add pipe.
__device__ __forceinline__ void exps_in_place(uint32_t (&r)[16], const RowConsts& k, float2 (&sum)[2]) {
#pragma unroll
  for (int g = 0; g < 16; g += 4) {
    const float2 a01 = __ffma2_rn(make_float2(__uint_as_float(r[g]), __uint_as_float(r[g + 1])), k.c2, k.neg_hi);
    const float2 a23 = __ffma2_rn(make_float2(__uint_as_float(r[g + 2]), __uint_as_float(r[g + 3])), k.c2, k.neg_hi);
    const float2 p01 = make_float2(ex2_approx(a01.x), ex2_approx(a01.y));
    const float2 p23 = (g & 4) == 0 ? exp2_poly(a23) : make_float2(ex2_approx(a23.x), ex2_approx(a23.y));
    sum[0] = __fadd2_rn(sum[0], make_float2(p01.x, p23.x));
    sum[1] = __fadd2_rn(sum[1], make_float2(p01.y, p23.y));
    r[g] = __float_as_uint(p01.x);
    r[g + 1] = __float_as_uint(p01.y);
    r[g + 2] = __float_as_uint(p23.x);
    r[g + 3] = __float_as_uint(p23.y);
  }
}
// Those to bytes, as in chunk_exp_pack.
__device__ __forceinline__ void pack_shares(const uint32_t (&r)[16], const float share, uint32_t (&packed)[4]) {
  const float2 levels = make_float2(kLevels, kLevels);
#pragma unroll
  for (int g = 0; g < 4; ++g) {
    auto p = [&](int i) { return __saturatef(__uint_as_float(r[4 * g + i]) * share); };
    const float2 high = __ffma2_rn(__ffma2_rn(make_float2(p(1), p(3)), levels, make_float2(kMagic, kMagic)), make_float2(256.f, 256.f),
                                   make_float2(-255.f * kMagic, -255.f * kMagic));
    const float2 y = __ffma2_rn(make_float2(p(0), p(2)), levels, high);
    packed[g] = __byte_perm(__float_as_uint(y.x), __float_as_uint(y.y), 0x5410);
  }
}

// ---------------------------------------------------------------------------------------------- softmax role
// One thread = every kChains-th group of 64 keys of one query row, and D / kChains columns of its output.
template <int D, bool kStatic, bool kBrief>
__device__ __forceinline__ void softmax_role(const FwdParams& p, Ctl* all, const int worker, const int chain, const uint32_t tmem_base) {
  using C = Cfg<D>;
  WorkerCtl* ctl = &all->w[worker];
  const int lane = threadIdx.x & 31, quad = warp_index() & 3, row = quad * 32 + lane;
  const uint32_t t_worker = tmem_base + (static_cast<uint32_t>(quad * 32) << 16) + static_cast<uint32_t>(worker * kCols);
  const uint32_t tO = t_worker + static_cast<uint32_t>(C::kOutCol + chain * C::kOutCols);
  volatile int* abort_flag = &all->abort;
  uint32_t uses0 = 0, uses1 = 0;                // phase 1: uses of each buffer
  // static, phase 1: scores that much above the sum's reference are exponentials of up to two
  const int slack = kStatic ? static_cast<int>(fminf(1.f / p.c2, 4194304.f)) : 0;
  Ring<C::kBufs> unit_begin;                    // buffer of the unit's first group in phase 2
  auto or_fail = [&](bool waited, unsigned code) -> bool {
    if (!waited) raise_status(abort_flag, p.status, code, uses0);
    return waited;
  };
  auto wait_or_fail = [&](uint32_t bar, uint32_t parity, unsigned code) -> bool { return or_fail(warp_wait(bar, parity, abort_flag), code); };
  // What a sum in terms of `from` is worth in terms of the larger `to`.  (Of whole numbers: a difference of two scaled maxima would have to be
  // of two rounded products, and the compiler may form one of one product and a fused multiply-add.)
  auto rescale = [&](int from, int to) { return ex2_approx(__int2float_rn(from - to) * p.c2); };
#pragma unroll 1
  for (int it = 0;; ++it) {
    const int buf = it % kInfoBufs;
    const uint32_t parity = static_cast<uint32_t>(it & 1);
    // (long, as the issuer's, while the loader goes through units without keys)
    if (!or_fail(warp_wait_long(smem_u32(&ctl->info_full[buf]), static_cast<uint32_t>((it / kInfoBufs) & 1), abort_flag), FMHA_I8_DEV_WAIT_INFO)) return;
    const UnitInfo* info = &ctl->info[buf];
    const int n = info->n;
    if (n < 0) return;

    float l = 1.f;                            // static: the integer sum becomes the output through one factor, else through that / l
    if constexpr (kBrief) {
      int imax = INT_MIN, ref = 0;
      float l_run = 0.f;
      RowConsts base = {};
      const uint32_t tS = t_worker + static_cast<uint32_t>(chain * kKeys);
      uint32_t r0[16], r1[16], r2[16], r3[16];
      if (!wait_or_fail(smem_u32(&ctl->max_full[0]), uses0++ & 1u, FMHA_I8_DEV_WAIT_S_READY)) return;
      if (chain < n) {
        tc_fence_after();
        tmem_ld16_issue(tS, r0);
        tmem_ld16_issue(tS + 16, r1);
        tmem_ld16_issue(tS + 32, r2);
        tmem_ld16_issue(tS + 48, r3);
        tmem_ld_fence(r0); tmem_ld_fence(r1); tmem_ld_fence(r2); tmem_ld_fence(r3);
        int max_a = INT_MIN, max_b = INT_MIN;
        chunk_max<16>(r0, max_a, max_b);
        chunk_max<16>(r1, max_a, max_b);
        chunk_max<16>(r2, max_a, max_b);
        chunk_max<16>(r3, max_a, max_b);
        imax = ref = max(max_a, max_b);
        base = row_consts(imax, p.c2, p.row_scale, p.scale_qk, 1.f);
        float2 sum[2] = {make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
        exps_in_place(r0, base, sum);
        exps_in_place(r1, base, sum);
        exps_in_place(r2, base, sum);
        exps_in_place(r3, base, sum);
        l_run = base.f * ((sum[0].x + sum[0].y) + (sum[1].x + sum[1].y));
      }
      ctl->stat[parity][chain][row] = make_float2(__int_as_float(imax), l_run);
      ctl->sum[parity][chain][row] = __int_as_float(ref);
      mbar_arrive(smem_u32(&ctl->xch[quad]));
      if (!wait_or_fail(smem_u32(&ctl->xch[quad]), parity, FMHA_I8_DEV_WAIT_S_READY)) return;
      const float2 other = ctl->stat[parity][chain ^ 1][row];
      imax = max(imax, __float_as_int(other.x));
      const float mine = rescale(ref, imax);
      // (a thread without a group has a sum of zero; the other one has one)
      l_run = fmaf(mine, l_run, rescale(__float_as_int(ctl->sum[parity][chain ^ 1][row]), imax) * other.y);
      // P8 = rn(levels * min(e / (l s_max), 1))
      if (chain < n) {
        const float share = p.p_mul / (l_run > 0.f ? l_run : 1.f) * (base.f * mine);
        uint32_t packed[4];
        pack_shares(r0, share, packed); tmem_st4(tS, packed);
        pack_shares(r1, share, packed); tmem_st4(tS + 4, packed);
        pack_shares(r2, share, packed); tmem_st4(tS + 8, packed);
        pack_shares(r3, share, packed); tmem_st4(tS + 12, packed);
        tmem_wait_st();
        tc_fence_before();
        mbar_arrive(smem_u32(&ctl->p_brief[chain]));
      }
    } else {
      // ---- phase 1: the row's maximum over all keys, as a biased integer (static: and the exp-sum, in terms of that of `ref`)
      int imax = INT_MIN;
      float l_run = 0.f;
      RowConsts base = {};
      int ref = 0, limit = INT_MIN;               // (biased integers of unmasked keys are positive)
#pragma unroll 1
      for (int a = 0; a * kChains < n; ++a) {
        const int b = a & 1, i = a * kChains + chain;
        if (!wait_or_fail(smem_u32(&ctl->max_full[b]), (b ? uses1++ : uses0++) & 1u, FMHA_I8_DEV_WAIT_S_READY)) return;
        if (i < n) {
          tc_fence_after();
          const uint32_t from = t_worker + static_cast<uint32_t>(b * kStep1 + chain * kKeys);
          uint32_t r0[16], r1[16], r2[16], r3[16];
          tmem_ld16_issue(from, r0);
          tmem_ld16_issue(from + 16, r1);
          tmem_ld16_issue(from + 32, r2);
          tmem_ld16_issue(from + 48, r3);
          tmem_ld_fence(r0); tmem_ld_fence(r1); tmem_ld_fence(r2); tmem_ld_fence(r3);
          tc_fence_before();
          mbar_arrive(smem_u32(&ctl->max_free[b]));
          int max_a = INT_MIN, max_b = INT_MIN;
          chunk_max<16>(r0, max_a, max_b);
          chunk_max<16>(r1, max_a, max_b);
          chunk_max<16>(r2, max_a, max_b);
          chunk_max<16>(r3, max_a, max_b);
          const int mine = max(max_a, max_b);
          if (!kStatic) {
            // (only groups with masked keys are preset)
            imax = max(imax, (info->group[i] & kMixed) != 0 ? mine : mine + static_cast<int>(kMagicBits));
          } else {
            // The sum is kept in terms of a maximum that is renewed when a row of the warp has gone beyond it by more than a factor of two, which few groups do
            // after the first: a group adds to the sum and forms no constants.
            imax = max(imax, mine);
            if (__any_sync(0xFFFFFFFFu, mine > limit)) {
              base = row_consts(imax, p.c2, p.row_scale, p.scale_qk, 1.f);
              l_run *= rescale(ref, imax);
              ref = imax;
              limit = imax + slack;
            }
            float2 sum[2] = {make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
            uint32_t none[4];
            chunk_exp_pack<16, false, 1, false>(r0, base.c2, base.neg_hi, base.p_mul_f, sum, none);
            chunk_exp_pack<16, false, 1, false>(r1, base.c2, base.neg_hi, base.p_mul_f, sum, none);
            chunk_exp_pack<16, false, 1, false>(r2, base.c2, base.neg_hi, base.p_mul_f, sum, none);
            chunk_exp_pack<16, false, 1, false>(r3, base.c2, base.neg_hi, base.p_mul_f, sum, none);
            l_run = fmaf(base.f, (sum[0].x + sum[0].y) + (sum[1].x + sum[1].y), l_run);
          }
        } else {
          mbar_arrive(smem_u32(&ctl->max_free[b]));
        }
      }
      ctl->stat[parity][chain][row] = make_float2(__int_as_float(imax), l_run);
      if (kStatic) ctl->sum[parity][chain][row] = __int_as_float(ref);
      mbar_arrive(smem_u32(&ctl->xch[quad]));
      // (with the row policy a unit has two exchanges, with the static one)
      if (!wait_or_fail(smem_u32(&ctl->xch[quad]), kStatic ? parity : 0u, FMHA_I8_DEV_WAIT_S_READY)) return;
      const float2 other = ctl->stat[parity][chain ^ 1][row];
      imax = max(imax, __float_as_int(other.x));
      if (kStatic) {
        // (a thread without a group has a sum of zero; the other one has some)
        l_run = fmaf(rescale(ref, imax), l_run, rescale(__float_as_int(ctl->sum[parity][chain ^ 1][row]), imax) * other.y);
      }
      // dynamic: P8 = rn(levels * e), e <= 1; static: P8 = rn(levels * min(e / (l s_max), 1))
      const RowConsts k = row_consts(imax, p.c2, p.row_scale, p.scale_qk, kStatic ? p.p_mul / (l_run > 0.f ? l_run : 1.f) : p.p_mul);
      const float2 p_mul = kStatic ? make_float2(kLevels, kLevels) : k.p_mul_f;

      // ---- phase 2: exp, row sum, requantise; the bytes go over columns already read
      float l_sum = 0.f;
      Ring<C::kBufs> set = unit_begin;
      if (chain == 1) set.advance();
      unit_begin.skip(static_cast<uint32_t>(n));
#pragma unroll 1
      for (int i = chain; i < n; i += kChains, set.template advance<kChains>()) {
        const uint32_t tS = t_worker + set.at * kKeys;
        if (!wait_or_fail(smem_u32(&ctl->s_full[set.at]), set.parity, FMHA_I8_DEV_WAIT_S_READY)) return;
        tc_fence_after();
        uint32_t ra[16], rb[16], packed[4];
        float2 sum[2] = {make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
        auto sixteen = [&](const uint32_t (&r)[16], uint32_t c, auto poly) {
          chunk_exp_pack<16, kStatic, decltype(poly)::value>(r, k.c2, k.neg_hi, p_mul, sum, packed, k.p_mul_f.x);
          tmem_st4(tS + c * 4, packed);
        };
        constexpr Flight<0> mufu;
        constexpr Flight<1> some_poly;          // a quarter of them on the multiply-add pipe
        tmem_ld16_issue(tS, ra);
        tmem_ld16_issue(tS + 16, rb);
        tmem_ld_fence(ra); tmem_ld_fence(rb);
        sixteen(ra, 0, mufu);
        tmem_ld16_issue(tS + 32, ra);
        sixteen(rb, 1, some_poly);
        tmem_ld16_issue(tS + 48, rb);
        tmem_ld_fence(ra); tmem_ld_fence(rb);
        sixteen(ra, 2, mufu);
        sixteen(rb, 3, some_poly);
        tmem_wait_st();
        tc_fence_before();
        mbar_arrive(smem_u32(&ctl->p_ready[set.at]));
        // (a sum for each group: over all groups of 32,768 keys in one, equal probabilities lost 5e-5 of it instead of 4e-6)
        l_sum += (sum[0].x + sum[0].y) + (sum[1].x + sum[1].y);
      }
      if (!kStatic) {
        l = k.f * l_sum;
        ctl->sum[parity][chain][row] = l;
        mbar_arrive(smem_u32(&ctl->xch[quad]));
        if (!wait_or_fail(smem_u32(&ctl->xch[quad]), 1u, FMHA_I8_DEV_WAIT_S_READY)) return;
        l += ctl->sum[parity][chain ^ 1][row];
      }
    }
    const float scale = p.scale_v_out * (kStatic ? 1.f : l > 0.f ? __frcp_rn(l) : 0.f);

    // ---- the sums of P.V are complete: normalise, requantise, store, 32 columns at a time
    const bool stored = row < info->rows;
    int8_t* dst = p.o + (info->first_row + row) * D + chain * C::kOutCols;
    if (!wait_or_fail(smem_u32(&ctl->o_full), parity, FMHA_I8_DEV_WAIT_O_READY)) return;
    __syncwarp();
    if (lane == 0) mbar_arrive(smem_u32(&ctl->info_empty[buf]));
    tc_fence_after();
#pragma unroll
    for (int c = 0; c < C::kOutCols; c += 32) {
      uint32_t ra[16], rb[16];
      tmem_ld16_issue(tO + c, ra);
      tmem_ld16_issue(tO + c + 16, rb);
      tmem_ld_fence(ra); tmem_ld_fence(rb);
      if (c + 32 == C::kOutCols) {
        tc_fence_before();
        mbar_arrive(smem_u32(&ctl->o_free));
      }
      float2 o2[16];
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        o2[i] = make_float2(__int2float_rn(static_cast<int>(ra[2 * i])), __int2float_rn(static_cast<int>(ra[2 * i + 1])));
        o2[8 + i] = make_float2(__int2float_rn(static_cast<int>(rb[2 * i])), __int2float_rn(static_cast<int>(rb[2 * i + 1])));
      }
      const bool clamp = __any_sync(0xFFFFFFFFu, needs_clamp<16>(o2, scale));
      uint32_t wide[8];
      requantise16(o2, make_float2(scale, scale), clamp, wide);
      requantise16(o2 + 8, make_float2(scale, scale), clamp, wide + 4);
      if (stored) {
        if (p.o_wide) {
          st_global_v8(dst + c, wide);
        } else {
          *reinterpret_cast<uint4*>(dst + c) = make_uint4(wide[0], wide[1], wide[2], wide[3]);
          *reinterpret_cast<uint4*>(dst + c + 16) = make_uint4(wide[4], wide[5], wide[6], wide[7]);
        }
      }
      __syncwarp();
    }
  }
}

// ---------------------------------------------------------------------------------------------- loader
// One warp per worker, run warp-wide: takes the CTA's units as its worker gets on, scans their masks and copies their tiles, a unit
// ahead of the other warps at the most.
__device__ __forceinline__ int scan_groups(uint16_t* list, const int8_t* mask_row, int S, int& first_mixed) {
  const uint32_t* words = reinterpret_cast<const uint32_t*>(mask_row);
  const int lane = threadIdx.x & 31;
  int n = 0;
#pragma unroll 1
  for (int base = 0; base < S; base += 32 * 32) {         // a lane looks at 32 keys, two lanes make a group
    const int key0 = base + lane * 32;
    uint32_t open = 0u, masked = 0u;
    if (key0 < S) {                                       // (S is a multiple of 64)
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const uint32_t w = words[(key0 >> 2) + i];
        masked |= w;
        open |= __vcmpeq4(w, 0u);
      }
    }
    const uint32_t any_open = __ballot_sync(0xFFFFFFFFu, open != 0u), any_masked = __ballot_sync(0xFFFFFFFFu, masked != 0u);
    const bool live = lane < 16 && ((any_open >> (2 * lane)) & 3u) != 0u;
    const uint32_t ballot = __ballot_sync(0xFFFFFFFFu, live);
    const uint32_t mixed = __ballot_sync(0xFFFFFFFFu, live && ((any_masked >> (2 * lane)) & 3u) != 0u);
    if (mixed != 0u && first_mixed < 0) first_mixed = n + __popc(ballot & ((mixed & (0u - mixed)) - 1u));
    if (live) {
      list[n + __popc(ballot & ((1u << lane) - 1u))] =
          static_cast<uint16_t>((base / kKeys + lane) | (((any_masked >> (2 * lane)) & 3u) != 0u ? kMixed : 0));
    }
    n += __popc(ballot);
  }
  return n;
}

template <int D, bool kBrief>
__device__ __forceinline__ void loader_role(const FwdParams& p, Ctl* all, const int worker, const CUtensorMap* map_q, const CUtensorMap* map_k,
                                            const CUtensorMap* map_v, const uint32_t worker_smem) {
  using C = Cfg<D>;
  WorkerCtl* ctl = &all->w[worker];
  volatile int* abort_flag = &all->abort;
  const int lane = threadIdx.x & 31;
  const uint32_t q_smem = worker_smem, ring_smem = q_smem + kQBufs * C::kQBytes;
  uint32_t fail = 0u, loaded = 0;
  int taken = worker, it = 0;
  auto wait = [&](uint32_t bar, uint32_t parity, uint32_t code) -> bool {
    if (fail == 0u && warp_wait(bar, parity, abort_flag)) return true;
    if (fail == 0u) fail = code;
    return false;
  };
  while (fail == 0u) {
    if (taken < 0) {
      if (lane == 0) taken = atomicAdd(&all->next, 1);
      taken = uniform(taken);
    }
    const uint32_t u = blockIdx.x + gridDim.x * static_cast<uint32_t>(taken);       // (unsigned: the first that does not exist may lie beyond int)
    taken = -1;
    const int buf = it % kInfoBufs;
    if (it >= kInfoBufs && !wait(smem_u32(&ctl->info_empty[buf]), static_cast<uint32_t>((it / kInfoBufs - 1) & 1), FMHA_I8_DEV_WAIT_INFO)) break;
    UnitInfo* info = &ctl->info[buf];
    if (u >= static_cast<uint32_t>(p.n_units)) {
      if (elect_one()) {
        info->n = -1;
        mbar_arrive(smem_u32(&ctl->info_full[buf]));
      }
      break;
    }
    const UnitGeom geo = unit_geom(p, static_cast<int>(u));
    const int8_t* mask_row = p.mask + static_cast<int64_t>(geo.batch) * p.S;
    int first_mixed = -1;
    const int n = scan_groups(info->group, mask_row, p.S, first_mixed), rows = min(kTile, p.Sq - geo.q_row0);
    const int64_t first_row = static_cast<int64_t>(geo.bh_local) * p.Sq + geo.q_row0;
    if (n == 0) {
      // rows without an unmasked key are zeros; nobody else hears of such a unit
      uint4* dst = reinterpret_cast<uint4*>(p.o + first_row * D);
      for (int i = lane; i < rows * (D / 16); i += 32) dst[i] = make_uint4(0u, 0u, 0u, 0u);
      continue;
    }
    if (lane == 0) {
      info->n = n;
      info->first_mixed = first_mixed < 0 ? n : first_mixed;
      info->rows = rows;
      info->first_row = first_row;
      info->mask_row = mask_row;
    }
    __syncwarp();
    if (elect_one()) mbar_arrive(smem_u32(&ctl->info_full[buf]));
    const uint32_t qb = static_cast<uint32_t>(it % kQBufs), bar_q = smem_u32(&ctl->q_full[qb]);
    if (it >= kQBufs && !wait(smem_u32(&ctl->q_empty[qb]), static_cast<uint32_t>((it / kQBufs - 1) & 1), FMHA_I8_DEV_WAIT_K_FREE)) break;
    if (elect_one()) {
      mbar_arrive_expect_tx(bar_q, C::kQBytes);
      tma_load_3d(q_smem + qb * C::kQBytes, map_q, bar_q, 0, geo.q_row0, geo.bh_local);
    }
    __syncwarp();
    // A place: group i0 of one tensor and, if it is one of the unit's, group i1 of K.
    auto load = [&](const CUtensorMap* map, int i0, int i1) {
      const uint32_t at = loaded % C::kStages, bar = smem_u32(&ctl->full[at]), to = ring_smem + at * C::kStageBytes;
      if (loaded >= C::kStages && !wait(smem_u32(&ctl->empty[at]), (loaded / C::kStages - 1) & 1u, FMHA_I8_DEV_WAIT_K_FREE)) return;
      ++loaded;
      const bool two = i1 < n;
      const int key0 = (info->group[i0] & ~kMixed) * kKeys, key1 = two ? (info->group[i1] & ~kMixed) * kKeys : 0;
      if (elect_one()) {
        mbar_arrive_expect_tx(bar, two ? C::kStageBytes : C::kGroupBytes);
        tma_load_3d(to, map, bar, 0, key0, geo.bh_local);
        if (two) tma_load_3d(to + C::kGroupBytes, map_k, bar, 0, key1, geo.bh_local);
      }
      __syncwarp();
    };
    constexpr int kAhead = static_cast<int>(C::kBufs);
    // phase 1, then what phase 2 begins with
    const int pairs = (n + 1) / 2, first = kBrief ? 0 : (min(n, kAhead) + 1) / 2;
#pragma unroll 1
    for (int a = 0; a < pairs + first; ++a) {
      const int i = 2 * (a < pairs ? a : a - pairs);
      load(map_k, i, a < pairs || i + 1 < kAhead ? i + 1 : n);
    }
#pragma unroll 1
    for (int i = 0; i < n; ++i) load(map_v, i, i + kAhead);
    ++it;
  }
  if (fail != 0u) {
    if (elect_one()) raise_status(abort_flag, p.status, fail, loaded);
    // unwinding: let copies that are still in flight land before the CTA may exit
    const long long t0 = clock64();
    while (clock64() - t0 < 2000000LL) { /* about a millisecond */ }
  }
}

// ---------------------------------------------------------------------------------------------- issuer
// One warp per worker, run warp-wide (every lane waits and counts, one elected lane issues): the MMAs of both phases.
//
// The order it relies on: MMAs of one thread run in the order of their issue, so S may go over the columns of P bytes right behind the P.V
// that reads them, in phase 2 and at the beginning of the next unit.  PTX promises the order of two tcgen05.mma with one accumulator and one
// shape, which these are not; that an earlier one has read its operand in tensor memory before a later one writes there is what published
// kernels for this chip rely on too (FlashAttention's forward pass for sm_100 and CUTLASS's example 77_blackwell_fmha: P over S, the next
// S issued behind P.V).  With a wait for P.V's completion in between, in both places, 80 forms of calls gave the same outputs to the last
// bit, 30 % later and more, since the wait joins the issuer's chain: B4 H16 S1024 D64 (512..1024 keys) per-row 24.6 -> 31.8 us, B1 H32 S2048 D128
// 57.2 -> 92.4, one unit to an SM B1 H2 S8192 D128 79.8 -> 168.  (The forward kernels need no such order: there the drain of P.V comes first.)
template <int D, bool kStatic, bool kBrief>
__device__ __forceinline__ void issuer_role(const FwdParams& p, Ctl* all, const int worker, const uint32_t tmem_base, const uint32_t worker_smem,
                                            uint8_t* presets) {
  using C = Cfg<D>;
  WorkerCtl* ctl = &all->w[worker];
  volatile int* abort_flag = &all->abort;
  const int lane = threadIdx.x & 31;
  const uint32_t q_smem = worker_smem, ring_smem = q_smem + kQBufs * C::kQBytes;
  const uint32_t t_worker = tmem_base + static_cast<uint32_t>(worker * kCols), tO = t_worker + C::kOutCol;
  constexpr uint32_t idesc_s = make_idesc_i8(kKeys, false), idesc_pair = make_idesc_i8(kStep1, false), idesc_preset = make_idesc_bf16(kKeys);
  constexpr uint32_t idesc_o = make_idesc_i8(D, true, true);
  const uint32_t preset_smem = smem_u32(presets);
  const uint64_t d_a = preset_desc(preset_smem, 0);
  const bool lead = elect_one();
  uint32_t fail = 0u, used = 0, groups = 0, uses0 = 0, uses1 = 0;      // places of the ring, and S, so far
  Ring<C::kBufs> s_set, p_set;
  uint32_t briefs[kChains] = {};                                        // kBrief: units that had a first, a second group
  auto wait = [&](uint32_t bar, uint32_t parity, uint32_t code) -> bool {
    if (warp_wait(bar, parity, abort_flag)) return true;
    fail = code;
    return false;
  };
  for (int it = 0; fail == 0u; ++it) {
    const int buf = it % kInfoBufs;
    if (!warp_wait_long(smem_u32(&ctl->info_full[buf]), static_cast<uint32_t>((it / kInfoBufs) & 1), abort_flag)) {
      fail = FMHA_I8_DEV_WAIT_INFO;
      break;
    }
    const UnitInfo* info = &ctl->info[buf];
    const int n = info->n;
    if (n < 0) break;
    const int8_t* mask_row = info->mask_row;
    const uint32_t qb = static_cast<uint32_t>(it % kQBufs);
    if (!wait(smem_u32(&ctl->q_full[qb]), static_cast<uint32_t>((it / kQBufs) & 1), FMHA_I8_DEV_WAIT_Q_LOAD)) break;
    const uint64_t dq = make_smem_desc(q_smem + qb * C::kQBytes, D);

    // The preset operand of group i, filled if it has masked keys.  The worker's four are used in turn: S of the group that used this one has
    // completed (in phase 2 S runs three groups ahead of P.V at the most, and P of the group before those has been seen; in phase 1
    // this group's columns have been read, and with them those of the four groups before this step and the one before it).
    auto preset_of = [&](int i, uint32_t number) -> uint64_t {
      uint32_t operand = kCommonB;
      if ((info->group[i] & kMixed) != 0) {
        operand = kOwnB + (static_cast<uint32_t>(worker) * kOwnOperands + number % kOwnOperands) * kOperandBytes;
        const int8_t* m = mask_row + (info->group[i] & ~kMixed) * kKeys;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int key = 32 * h + lane;
          *reinterpret_cast<uint32_t*>(presets + operand + key * 16) = m[key] != 0 ? kBiasBMasked : kBiasB;
        }
        fence_proxy_async_smem();
        __syncwarp();
      }
      return preset_desc(preset_smem, operand);
    };
    auto landed = [&]() { return wait(smem_u32(&ctl->full[used % C::kStages]), (used / C::kStages) & 1u, FMHA_I8_DEV_WAIT_K_LOAD); };
    auto place_desc = [&]() { return make_smem_desc(ring_smem + (used % C::kStages) * C::kStageBytes, D); };
    // (one lane)
    auto issue_s = [&](uint32_t tS, uint64_t d_preset, uint64_t dk, bool preset) {
      if (preset) mma_f16_ss(tS, d_a, d_preset, idesc_preset, 0u);      // accumulator := 0x4B400000, masked keys -2^127
#pragma unroll
      for (int kk = 0; kk < D / 32; ++kk) mma_i8_ss(tS, desc_advance(dq, kk * 32), desc_advance(dk, kk * 32), idesc_s, preset || kk > 0 ? 1u : 0u);
    };
    auto issue_pv = [&](uint32_t tP, uint64_t dv, bool first) {
#pragma unroll
      for (int kk = 0; kk < kKeys / 32; ++kk) mma_i8_ts(tO, tP + kk * 8, desc_advance(dv, kk * 32 * D), idesc_o, !first || kk > 0 ? 1u : 0u);
    };

    // ---- phase 1: two groups a step
    // (Which groups are preset is looked up only from the first of them on: the issuer's instructions are what a step here waits for, 750 cycles of which
    // 200 issue.  B1 H32 S2048 54.2 -> 53.1 us, B2 H32 S2048 D128 113 -> 110.5.)
    const int plain = kStatic ? 0 : info->first_mixed;
#pragma unroll 1
    for (int a = 0; a * kChains < n && fail == 0u; ++a) {
      const int b = a & 1, i = a * kChains;
      const bool two = i + 1 < n, whole = i + 1 < plain;
      uint32_t tS = t_worker + static_cast<uint32_t>(b * kStep1);
      uint64_t dk = place_desc();
      uint32_t bar_full = smem_u32(&ctl->max_full[b]), bar_empty = smem_u32(&ctl->empty[used % C::kStages]);
      asm volatile("" : "+r"(tS), "+l"(dk), "+r"(bar_full), "+r"(bar_empty));
      const uint32_t before = b ? uses1++ : uses0++;
      if (!landed()) break;
      // (kBrief: the P.V of the unit before has waited for everything that is read)
      if (!kBrief && before > 0u && !wait(smem_u32(&ctl->max_free[b]), (before - 1u) & 1u, FMHA_I8_DEV_WAIT_O_FREE)) break;
      // (The first half of the columns may still hold P bytes of the unit before, whose P.V was issued in front: see the order above.)  The second
      // half is where its sums were.
      if (a == 1 && it > 0 && !wait(smem_u32(&ctl->o_free), static_cast<uint32_t>((it - 1) & 1), FMHA_I8_DEV_WAIT_O_FREE)) break;
      tc_fence_after();
      if (whole) {
        if (lead) {
#pragma unroll
          for (int kk = 0; kk < D / 32; ++kk) mma_i8_ss(tS, desc_advance(dq, kk * 32), desc_advance(dk, kk * 32), idesc_pair, kk > 0 ? 1u : 0u);
          mma_commit(bar_full);
          mma_commit(bar_empty);
        }
      } else {
        const bool preset0 = kStatic || (info->group[i] & kMixed) != 0, preset1 = two && (kStatic || (info->group[i + 1] & kMixed) != 0);
        const uint64_t d_preset0 = preset0 ? preset_of(i, groups) : 0u, d_preset1 = preset1 ? preset_of(i + 1, groups + 1u) : 0u;
        if (lead) {
          issue_s(tS, d_preset0, dk, preset0);
          if (two) issue_s(tS + kKeys, d_preset1, desc_advance(dk, C::kGroupBytes), preset1);
          mma_commit(bar_full);
          mma_commit(bar_empty);
          if (kBrief) mma_commit(smem_u32(&ctl->q_empty[qb]));
        }
      }
      __syncwarp();
      ++used;
      groups += two ? 2u : 1u;
    }
    if constexpr (kBrief) {
      // the P bytes are over the columns of the scores
#pragma unroll
      for (int i = 0; i < kChains; ++i) {
        if (i >= n || !landed()) break;
        uint64_t dv = place_desc();
        uint32_t tP = t_worker + static_cast<uint32_t>(i * kKeys), bar_empty = smem_u32(&ctl->empty[used % C::kStages]);
        asm volatile("" : "+l"(dv), "+r"(tP), "+r"(bar_empty));
        if (!wait(smem_u32(&ctl->p_brief[i]), briefs[i]++ & 1u, FMHA_I8_DEV_WAIT_P_READY)) break;
        tc_fence_after();
        if (lead) {
          issue_pv(tP, dv, i == 0);
          if (i == n - 1) mma_commit(smem_u32(&ctl->o_full));
          mma_commit(bar_empty);
        }
        __syncwarp();
        ++used;
      }
    } else {
      // all scores of phase 1 have been read (and with them the sums of the unit before)
      if (fail != 0u || !wait(smem_u32(&ctl->max_free[0]), (uses0 - 1u) & 1u, FMHA_I8_DEV_WAIT_O_FREE)) break;
      if (uses1 > 0u && !wait(smem_u32(&ctl->max_free[1]), (uses1 - 1u) & 1u, FMHA_I8_DEV_WAIT_O_FREE)) break;
      tc_fence_after();

      // ---- phase 2: S runs kBufs groups ahead of P.V
      constexpr int kAhead = static_cast<int>(C::kBufs);
#pragma unroll 1
      for (int i = 0; i < kAhead && i < n; ++i) {
        if (!landed()) break;
        const uint64_t d_preset = preset_of(i, groups), dk = place_desc() + static_cast<uint64_t>((i & 1) * C::kGroupBytes >> 4);
        const bool last_of_place = (i & 1) != 0 || i + 1 == kAhead || i + 1 == n;
        if (lead) {
          issue_s(t_worker + s_set.at * kKeys, d_preset, dk, true);
          mma_commit(smem_u32(&ctl->s_full[s_set.at]));
          if (last_of_place) mma_commit(smem_u32(&ctl->empty[used % C::kStages]));
          if (i == n - 1) mma_commit(smem_u32(&ctl->q_empty[qb]));
        }
        __syncwarp();
        if (last_of_place) ++used;
        ++groups;
        s_set.advance();
      }
#pragma unroll 1
      for (int i = 0; i < n && fail == 0u; ++i) {
        const int ahead = i + kAhead;
        if (!landed()) break;
        uint64_t d_preset = ahead < n ? preset_of(ahead, groups) : 0u, dv = place_desc();
        uint32_t tP = t_worker + p_set.at * kKeys, tS = t_worker + s_set.at * kKeys;
        uint32_t bar_s = smem_u32(&ctl->s_full[s_set.at]), bar_empty = smem_u32(&ctl->empty[used % C::kStages]);
        asm volatile("" : "+l"(d_preset), "+l"(dv), "+r"(tP), "+r"(tS), "+r"(bar_s), "+r"(bar_empty));          // formed here, not behind the wait
        if (!wait(smem_u32(&ctl->p_ready[p_set.at]), p_set.parity, FMHA_I8_DEV_WAIT_P_READY)) break;
        tc_fence_after();
        if (lead) {
          issue_pv(tP, dv, i == 0);
          if (ahead < n) {
            // (over the P bytes, behind the P.V that reads them: see the issuer's order above)
            issue_s(tS, d_preset, desc_advance(dv, C::kGroupBytes), true);
            mma_commit(bar_s);
            if (ahead == n - 1) mma_commit(smem_u32(&ctl->q_empty[qb]));
          } else if (i == n - 1) {
            mma_commit(smem_u32(&ctl->o_full));
          }
          mma_commit(bar_empty);
        }
        __syncwarp();
        p_set.advance();
        ++used;
        if (ahead < n) {
          ++groups;
          s_set.advance();
        }
      }
    }
    if (fail == 0u && elect_one()) mbar_arrive(smem_u32(&ctl->info_empty[buf]));
    __syncwarp();
  }
  if (fail != 0u && elect_one()) raise_status(abort_flag, p.status, fail, used);
}

// Everything in front of the roles: barriers, tensor memory, constant operands, then the wait for the launch before this one.  Returns
// the address of tensor memory.
__device__ __forceinline__ uint32_t set_up(Ctl* ctl, uint8_t* presets, const CUtensorMap* map_q, const CUtensorMap* map_k, const CUtensorMap* map_v) {
  const int warp = warp_index();
  if (threadIdx.x == 0) {
    ctl->abort = 0;
    ctl->next = kWorkers;
    for (WorkerCtl& w : ctl->w) {
      for (int i = 0; i < kQBufs; ++i) { mbar_init(smem_u32(&w.q_full[i]), 1); mbar_init(smem_u32(&w.q_empty[i]), 1); }
      for (int i = 0; i < kMaxStages; ++i) { mbar_init(smem_u32(&w.full[i]), 1); mbar_init(smem_u32(&w.empty[i]), 1); }
      for (int i = 0; i < 2; ++i) { mbar_init(smem_u32(&w.max_full[i]), 1); mbar_init(smem_u32(&w.max_free[i]), kChains * kTile); }
      for (int i = 0; i < 3; ++i) { mbar_init(smem_u32(&w.s_full[i]), 1); mbar_init(smem_u32(&w.p_ready[i]), kTile); }
      for (int i = 0; i < kChains; ++i) mbar_init(smem_u32(&w.p_brief[i]), kTile);
      mbar_init(smem_u32(&w.o_full), 1);
      mbar_init(smem_u32(&w.o_free), kChains * kTile);
      for (int i = 0; i < 4; ++i) mbar_init(smem_u32(&w.xch[i]), 64);
      for (int i = 0; i < kInfoBufs; ++i) { mbar_init(smem_u32(&w.info_full[i]), 1); mbar_init(smem_u32(&w.info_empty[i]), 1 + 4 * kChains); }
    }
    mbar_init_fence();
    tma_prefetch_desc(map_q);
    tma_prefetch_desc(map_k);
    tma_prefetch_desc(map_v);
  }
  if (warp == kSoftmaxWarps) {
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
  return tmem_base;
}

template <int D, bool kStatic, bool kBrief>
__global__ void __launch_bounds__(kThreads, 1)
policy_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k, const __grid_constant__ CUtensorMap map_v,
              const FwdParams p) {
  using C = Cfg<D>;
  extern __shared__ uint8_t smem_raw[];
  grid_launch_dependents();
  uint8_t* tiles = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
  uint8_t* presets = tiles + kWorkers * C::kWorkerBytes;
  Ctl* ctl = reinterpret_cast<Ctl*>(presets + kPresetBytes);
  const int warp = warp_index();
  const uint32_t tmem_base = set_up(ctl, presets, &map_q, &map_k, &map_v);

  // warps: 4 kChains softmax warps per worker (their number modulo 4 is their lane quarter), the issuers, the loaders
  if (warp < kSoftmaxWarps) {
    setmaxnreg_inc<kSoftmaxRegs>();
    softmax_role<D, kStatic, kBrief>(p, ctl, warp / (4 * kChains), (warp >> 2) % kChains, tmem_base);
  } else {
    setmaxnreg_dec<kOtherRegs>();
    const int worker = (warp - kSoftmaxWarps) % kWorkers;
    const uint32_t worker_smem = smem_u32(tiles + worker * C::kWorkerBytes);
    if (warp < kSoftmaxWarps + kWorkers) issuer_role<D, kStatic, kBrief>(p, ctl, worker, tmem_base, worker_smem, presets);
    else loader_role<D, kBrief>(p, ctl, worker, &map_q, &map_k, &map_v, worker_smem);
  }
  tc_fence_before();
  __syncthreads();
  if (warp == kSoftmaxWarps) {
    tc_fence_after();
    tmem_dealloc(tmem_base, kTmemCols);
  }
}

}  // namespace wholerow
}  // namespace fmha
