// Inline-PTX building blocks for sm_100a: mbarrier, TMA (cp.async.bulk.tensor), tensor memory
// (tcgen05.alloc/ld/st) and the 5th-generation tensor-core MMA (tcgen05.mma kind::i8).
// Every wait is bounded: a wait that runs out returns false and the caller unwinds.
#pragma once
#include <cuda.h>
#include <cstdint>

namespace fmha {

// A value that is the same in all lanes, in a form from which the compiler can see it (all 32 lanes call this together).  What
// is derived from it -- addresses of tensor memory and of barriers, descriptors, ring positions -- then lives in uniform registers
// and on the uniform datapath; otherwise every tcgen05 instruction has its address brought over lane by lane, and the issue
// slots this takes are what the forward kernels are short of.
template <typename T> __device__ __forceinline__ T uniform(T v) { return __shfl_sync(0xFFFFFFFFu, v, 0); }
__device__ __forceinline__ int warp_index() { return uniform(static_cast<int>(threadIdx.x >> 5)); }
// max(a, |b|, |c|) for a >= 0
__device__ __forceinline__ float max3_abs(float a, float b, float c) {
  float r;
  asm("max.abs.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
  return r;
}
// The same, and NaN if one of the three is.
__device__ __forceinline__ float max3_abs_nan(float a, float b, float c) {
  float r;
  asm("max.NaN.abs.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
  return r;
}
__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

// ---------------------------------------------------------------- mbarrier
__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
// Makes freshly initialised barriers visible to the async proxy (TMA, tcgen05.commit).
__device__ __forceinline__ void mbar_init_fence() {
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void mbar_arrive_expect_tx(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(bar), "r"(parity)
      : "memory");
  return ok != 0;
}


// The limits of a wait.  Most are for one key tile of one CTA, microseconds, and are counted, kWaitProbes: a time slice of another context on a
// shared GPU, in which no probes are made, cannot end such a wait.  How long a probe blocks that finds the phase incomplete is the system's
// choice: 2911 cycles here, so that all of them take one and a half seconds (tests/test_gpu_h_status.py measures it); if they did not block at
// all their instructions would still take some 20 ms.
// That is not enough for waits which may be long for a good reason: those of a warp that does not hear of units without keys while another
// one goes through a row of them (warp_wait_long).  1.1 us a unit with 64 keys, 8.8 with 32,768, measured in the workers, shared by the CTA's
// four: as many as outputs fit into 180 GB (11 million of 8 KB with long masks, 43 million of one row with short ones) are 0.2 s or less.  Such
// a wait ends when kWaitLimitCycles, about one second at boost clock, have passed as well.
constexpr long long kWaitLimitCycles = 2000000000LL;
constexpr uint32_t kWaitProbes = 1u << 20;

// Waits for the phase with the given parity to complete.  Gives up when the cycle limit is reached (and at least min_probes probes were
// made) or when another thread of the CTA has already raised *abort_flag.
__device__ __forceinline__ bool mbar_wait_limited(uint32_t bar, uint32_t parity, const volatile int* abort_flag, long long limit_cycles, uint32_t min_probes = 0u) {
  if (mbar_try_wait(bar, parity)) return true;
  const long long t0 = clock64();
  for (uint32_t it = 1;; ++it) {
    if (mbar_try_wait(bar, parity)) return true;
    if ((it & 31u) == 0u) {
      if (*abort_flag) return false;
      if (it >= min_probes && clock64() - t0 > limit_cycles) return false;
    }
  }
}
// For the kernels that stream through memory and have few waits: the quantiser and decoding are 0.3 to 0.4 % faster with the first probe apart
// than with the loop below (67,108,864 elements 75.8 and 76.1 us).
__device__ __forceinline__ bool mbar_wait_timed(uint32_t bar, uint32_t parity, const volatile int* abort_flag) {
  return mbar_wait_limited(bar, parity, abort_flag, kWaitLimitCycles, 4096u);
}
// For the forward kernels, in as few instructions as can be: they have some twenty waits each, and how far their code is spread costs them
// time.  B64 H32 S256 D128: the form above 82.9 us, this loop left to the compiler 78.6, as it is 77.8.  (kProbes: for tests.)
template <uint32_t kProbes = kWaitProbes>
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, const volatile int* abort_flag) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p, q;\n\t.reg .u32 left, flag;\n\t"
      "mov.u32 left, %4;\n"
      "WAIT_%=:\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "@p bra DONE_%=;\n\t"
      "ld.volatile.shared.u32 flag, [%3];\n\t"
      "sub.u32 left, left, 1;\n\t"
      "setp.eq.u32 q, flag, 0;\n\t"
      "setp.ne.and.u32 q, left, 0, q;\n\t"
      "@q bra WAIT_%=;\n"
      "DONE_%=:\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(bar), "r"(parity), "r"(smem_u32(const_cast<const int*>(abort_flag))), "n"(kProbes)
      : "memory");
  return ok != 0u;
}
// For a warp whose lanes run together, with one answer for all of them: the vote in the loop makes its branches uniform, and none is needed
// behind it.  The workers: B256 H16 S256 D64 (64..256 keys) 87.8 us with the loop above and a vote behind it, 85.6 with this one; the general
// kernel is the same with either.
template <uint32_t kProbes = kWaitProbes>
__device__ __forceinline__ bool warp_wait(uint32_t bar, uint32_t parity, const volatile int* abort_flag) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p, q, r;\n\t.reg .u32 left, flag;\n\t"
      "mov.u32 left, %4;\n"
      "WAIT_%=:\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "vote.sync.all.pred q, p, 0xffffffff;\n\t"
      "@q bra.uni DONE_%=;\n\t"
      "ld.volatile.shared.u32 flag, [%3];\n\t"
      "sub.u32 left, left, 1;\n\t"
      "setp.eq.u32 r, flag, 0;\n\t"
      "setp.ne.and.u32 r, left, 0, r;\n\t"
      "vote.sync.all.pred r, r, 0xffffffff;\n\t"
      "@r bra.uni WAIT_%=;\n"
      "DONE_%=:\n\t"
      "selp.u32 %0, 1, 0, q;\n\t}"
      : "=r"(ok)
      : "r"(bar), "r"(parity), "r"(smem_u32(const_cast<const int*>(abort_flag))), "n"(kProbes)
      : "memory");
  return ok != 0u;
}

// The same where the wait may be long (see kWaitLimitCycles), four instructions more: it ends when the probes are used up and the cycles have
// passed.  (The low half of the cycle counter is enough: a probe takes microseconds, so the first that comes too late sees it.)  With all
// waits like this, B64 H32 S256 D128 74.0 -> 74.7 us, B128 H16 S128 D128 28.3 -> 28.6, B64 H16 S64 D64 8.50 -> 8.64, B32 H12 S512 D64 (256..512)
// 34.9 -> 35.1.
template <uint32_t kProbes = kWaitProbes>
__device__ __forceinline__ bool warp_wait_long(uint32_t bar, uint32_t parity, const volatile int* abort_flag, uint32_t limit_cycles = kWaitLimitCycles) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p, q, r;\n\t.reg .s32 left;\n\t.reg .u32 flag, start, t;\n\t"
      "mov.u32 start, %%clock;\n\t"
      "mov.s32 left, %4;\n"
      "WAIT_%=:\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "vote.sync.all.pred q, p, 0xffffffff;\n\t"
      "@q bra.uni DONE_%=;\n\t"
      "ld.volatile.shared.u32 flag, [%3];\n\t"
      "sub.s32 left, left, 1;\n\t"
      "mov.u32 t, %%clock;\n\t"
      "sub.u32 t, t, start;\n\t"
      "setp.gt.s32 r, left, 0;\n\t"
      "setp.lt.or.u32 r, t, %5, r;\n\t"
      "setp.eq.and.u32 r, flag, 0, r;\n\t"
      "vote.sync.all.pred r, r, 0xffffffff;\n\t"
      "@r bra.uni WAIT_%=;\n"
      "DONE_%=:\n\t"
      "selp.u32 %0, 1, 0, q;\n\t}"
      : "=r"(ok)
      : "r"(bar), "r"(parity), "r"(smem_u32(const_cast<const int*>(abort_flag))), "n"(kProbes), "r"(limit_cycles)
      : "memory");
  return ok != 0u;
}

// One lane of a converged warp (the same one every time).  The single-thread roles of the forward kernel run
// warp-wide with only their side-effecting instructions behind this predicate: addresses, descriptors and loop
// counters are then warp-uniform values.
__device__ __forceinline__ bool elect_one() {
  uint32_t pred;
  asm volatile(
      "{\n\t.reg .pred P;\n\t"
      "elect.sync _|P, 0xFFFFFFFF;\n\t"
      "selp.u32 %0, 1, 0, P;\n\t}"
      : "=r"(pred));
  return pred != 0;
}

// One 32-byte store (address 32-byte aligned) that does not allocate a line in L1: the output is written once and
// never read by this kernel (measured 1.6 % of the C3 launch against the plain store).
__device__ __forceinline__ void st_global_v8(void* ptr, const uint32_t (&r)[8]) {
  asm volatile("st.global.L1::no_allocate.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};"
               ::"l"(ptr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7])
               : "memory");
}

// ---------------------------------------------------------------- programmatic dependent launch
// Blocks until every kernel before this one in the stream has finished and its writes are visible.  With the launch
// attribute that allows it, a kernel starts before that: what precedes this instruction must not touch global memory
// that an earlier kernel may write or still read.
// What comes after it reads global memory with ordinary loads: __ldg and loads through const __restrict__ parameters are for memory
// that nobody writes while the kernel runs, and the kernel before may still be writing when this one has begun.  (The compiler may
// move such a load in front of the wait, and the L1 may answer it with what another kernel on that SM has left there.)
__device__ __forceinline__ void grid_dependency_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
// Lets the next kernel of the stream start (up to its own grid_dependency_wait) once all CTAs have executed this.
__device__ __forceinline__ void grid_launch_dependents() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// ---------------------------------------------------------------- thread-block clusters
__device__ __forceinline__ uint32_t cluster_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ uint32_t cluster_ctas() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(r));
  return r;
}
// Barrier over all threads of the cluster, in two halves; orders the shared-memory accesses of all its CTAs.
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }
// Address, in the cluster's shared window, of CTA `rank`'s copy of the shared-memory object at `addr` in this CTA.
__device__ __forceinline__ uint32_t map_to_rank(uint32_t addr, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
  return r;
}
__device__ __forceinline__ void st_cluster_f32(uint32_t addr, uint32_t rank, float v) {
  asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(map_to_rank(addr, rank)), "f"(v) : "memory");
}
// Two floats to a cluster address (8-byte aligned).
__device__ __forceinline__ void st_cluster_v2(uint32_t cluster_addr, float a, float b) {
  asm volatile("st.shared::cluster.v2.f32 [%0], {%1, %2};" ::"r"(cluster_addr), "f"(a), "f"(b) : "memory");
}
__device__ __forceinline__ float2 ld_cluster_v2(uint32_t cluster_addr) {
  float2 v;
  asm volatile("ld.shared::cluster.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "r"(cluster_addr) : "memory");
  return v;
}
__device__ __forceinline__ float4 ld_cluster_v4(uint32_t cluster_addr) {
  float4 v;
  asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(cluster_addr) : "memory");
  return v;
}

// ---------------------------------------------------------------- TMA
// L2 replacement policies for such copies.
__device__ __forceinline__ uint64_t l2_evict_first() {
  uint64_t p;
  asm("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(p));
  return p;
}
__device__ __forceinline__ uint64_t l2_evict_last() {
  uint64_t p;
  asm("createpolicy.fractional.L2::evict_last.b64 %0, 1.0;" : "=l"(p));
  return p;
}
// Untiled copy global -> shared: both addresses and the size are multiples of 16 bytes.
__device__ __forceinline__ void bulk_load(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar, uint64_t policy) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes.L2::cache_hint [%0], [%1], %2, [%3], %4;"
               ::"r"(dst), "l"(src), "r"(bytes), "r"(bar), "l"(policy)
               : "memory");
}
__device__ __forceinline__ void tma_prefetch_desc(const CUtensorMap* map) {
  asm volatile("prefetch.tensormap [%0];" ::"l"(map) : "memory");
}
// 3-D tiled load global -> shared, completion counted in bytes on an mbarrier.  x must be a
// multiple of 16 bytes (it is always 0 here).
__device__ __forceinline__ void tma_load_3d(uint32_t dst, const CUtensorMap* map, uint32_t bar, int x, int y, int z) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];"
      ::"r"(dst), "l"(map), "r"(bar), "r"(x), "r"(y), "r"(z)
      : "memory");
}
// Generic-proxy writes to shared memory -> visible to the async proxy (tensor core / TMA reads).
__device__ __forceinline__ void fence_proxy_async_smem() {
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}

// ---------------------------------------------------------------- tensor memory
__device__ __forceinline__ void tmem_alloc(uint32_t smem_result, uint32_t ncols) {
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_result), "r"(ncols) : "memory");
}
__device__ __forceinline__ void tmem_relinquish() {
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t ncols) {
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tmem_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

// Warp-collective: lane t of warp w reads TMEM lane 32*(w%4)+t, 32 consecutive 32-bit columns.
// The load and its completion wait sit in ONE asm statement: the destination registers are only
// defined once tcgen05.wait::ld has retired, and nothing may be scheduled between the two.
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
      "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];\n\t"
      "tcgen05.wait::ld.sync.aligned;"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
        "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
        "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr)
      : "memory");
}
// Split form for software pipelining: issue the load now, consume later.  The registers are only
// defined after tmem_ld_fence(r); its "+r" operands make every consumer depend on the wait, so the
// compiler cannot hoist a use above it.  (tcgen05.wait::ld waits for ALL loads in flight.)
// 16-column variants of the split load.
__device__ __forceinline__ void tmem_ld16_issue(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr)
      : "memory");
}
__device__ __forceinline__ void tmem_ld_fence(uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.wait::ld.sync.aligned;"
      : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]), "+r"(r[7]),
        "+r"(r[8]), "+r"(r[9]), "+r"(r[10]), "+r"(r[11]), "+r"(r[12]), "+r"(r[13]), "+r"(r[14]), "+r"(r[15])
      :
      : "memory");
}
// 8-column variants of the split load.
__device__ __forceinline__ void tmem_ld8_issue(uint32_t taddr, uint32_t (&r)[8]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
               : "r"(taddr)
               : "memory");
}
__device__ __forceinline__ void tmem_ld_fence(uint32_t (&r)[8]) {
  asm volatile("tcgen05.wait::ld.sync.aligned;"
               : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]), "+r"(r[7])
               :
               : "memory");
}
// Warp-collective store of 2 consecutive 32-bit columns per lane.
__device__ __forceinline__ void tmem_st2(uint32_t taddr, const uint32_t (&r)[2]) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x2.b32 [%0], {%1, %2};" ::"r"(taddr), "r"(r[0]), "r"(r[1]) : "memory");
}
// Warp-collective store of 4 consecutive 32-bit columns per lane.
__device__ __forceinline__ void tmem_st4(uint32_t taddr, const uint32_t (&r)[4]) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x4.b32 [%0], {%1, %2, %3, %4};"
               ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3])
               : "memory");
}
// Warp-collective load (complete on return) and store of 32 consecutive 32-bit columns per lane, as eight float4.  The instructions ask for
// lanes that run together, and the lanes of those who call these may have parted: in copies that one of them asks for, in values that
// only some of them have to look at again.
__device__ __forceinline__ void tmem_ld_tile(uint32_t taddr, float4 (&v)[8]) {
  __syncwarp();
  uint32_t r[32];
  tmem_ld32(taddr, r);
#pragma unroll
  for (int i = 0; i < 8; ++i)
    v[i] = make_float4(__uint_as_float(r[4 * i]), __uint_as_float(r[4 * i + 1]), __uint_as_float(r[4 * i + 2]), __uint_as_float(r[4 * i + 3]));
}
__device__ __forceinline__ void tmem_st_tile(uint32_t taddr, const float4 (&v)[8]) {
  __syncwarp();
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
      "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, "
      "%17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31, %32};"
      ::"r"(taddr), "f"(v[0].x), "f"(v[0].y), "f"(v[0].z), "f"(v[0].w), "f"(v[1].x), "f"(v[1].y), "f"(v[1].z), "f"(v[1].w),
      "f"(v[2].x), "f"(v[2].y), "f"(v[2].z), "f"(v[2].w), "f"(v[3].x), "f"(v[3].y), "f"(v[3].z), "f"(v[3].w),
      "f"(v[4].x), "f"(v[4].y), "f"(v[4].z), "f"(v[4].w), "f"(v[5].x), "f"(v[5].y), "f"(v[5].z), "f"(v[5].w),
      "f"(v[6].x), "f"(v[6].y), "f"(v[6].z), "f"(v[6].w), "f"(v[7].x), "f"(v[7].y), "f"(v[7].z), "f"(v[7].w)
      : "memory");
}
// Warp-collective store of 8 consecutive 32-bit columns per lane.
__device__ __forceinline__ void tmem_st8(uint32_t taddr, const uint32_t (&r)[8]) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};"
               ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7])
               : "memory");
}

// ---------------------------------------------------------------- tensor-core MMA, 8-bit integer
// D[tmem] (+)= A[smem] * B[smem]; issued by ONE thread.  accumulate == 0 overwrites D.
__device__ __forceinline__ void mma_i8_ss(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, p;\n\t}"
      ::"r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate)
      : "memory");
}
// D[tmem] (+)= A[tmem] * B[smem].  A is M x K, one row per TMEM lane, four int8 per 32-bit column.
__device__ __forceinline__ void mma_i8_ts(uint32_t d_tmem, uint32_t a_tmem, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::i8 [%0], [%1], %2, %3, p;\n\t}"
      ::"r"(d_tmem), "r"(a_tmem), "l"(b_desc), "r"(idesc), "r"(accumulate)
      : "memory");
}
// D[tmem] (+)= A[smem] * B[smem] with fp16 (or bf16: the instruction descriptor says) operands and an fp32 accumulator
// (K = 16 per instruction).
__device__ __forceinline__ void mma_f16_ss(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
      ::"r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate)
      : "memory");
}
// The mbarrier receives one arrival when every MMA issued so far by this thread has completed.
__device__ __forceinline__ void mma_commit(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}

// ---------------------------------------------------------------- descriptors
// Instruction descriptor for kind::i8: int32 accumulator, 8-bit A (signed unless a_unsigned) and signed
// 8-bit B, M = 128.
//   bits 4-5 D format (2 = s32) | 7-9 A format (0 = u8, 1 = s8) | 10-12 B format (1 = s8)
//   bit 15 A major (0 = K) | bit 16 B major (0 = K, 1 = MN) | 17-22 N>>3 | 24-28 M>>4
__host__ __device__ constexpr uint32_t make_idesc_i8(int n, bool b_mn_major, bool a_unsigned = false) {
  return (2u << 4) | ((a_unsigned ? 0u : 1u) << 7) | (1u << 10) | ((b_mn_major ? 1u : 0u) << 16) |
         (static_cast<uint32_t>(n >> 3) << 17) | (static_cast<uint32_t>(128 >> 4) << 24);
}

// Shared-memory matrix descriptor for a swizzled tile whose rows are `row_bytes` (64 or 128) long
// and whose 8-row groups follow each other every 8*row_bytes bytes -- exactly what a TMA box
// {row_bytes, rows} with the matching swizzle mode writes.  The same bit pattern serves a K-major
// operand (rows = M or N index, contraction along the row) and an MN-major operand (rows =
// contraction index, M/N along the row); which one is meant is said by the instruction descriptor.
//   bits 0-13 address>>4 | 16-29 leading byte offset>>4 (unused here: one swizzle atom wide)
//   32-45 stride byte offset>>4 | 46-47 version = 1 | 61-63 layout (2 = 128B swizzle, 4 = 64B)
__device__ __forceinline__ uint64_t make_smem_desc(uint32_t smem_addr, int row_bytes) {
  const uint32_t sbo = static_cast<uint32_t>(8 * row_bytes) >> 4;
  const uint32_t layout = (row_bytes == 128) ? 2u : 4u;
  const uint32_t lo = ((smem_addr & 0x3FFFFu) >> 4) | (1u << 16);
  const uint32_t hi = sbo | (1u << 14) | (layout << 29);
  return (static_cast<uint64_t>(hi) << 32) | lo;
}
// kind::f16 instruction descriptor: fp32 accumulator (D format 1), fp16 A and B (format 0), both K-major, M = 128.
__host__ __device__ constexpr uint32_t make_idesc_f16(int n) {
  return (1u << 4) | (static_cast<uint32_t>(n >> 3) << 17) | (static_cast<uint32_t>(128 >> 4) << 24);
}
// The same with bf16 A and B (format 1).
__host__ __device__ constexpr uint32_t make_idesc_bf16(int n) { return make_idesc_f16(n) | (1u << 7) | (1u << 10); }
// Descriptor of an unswizzled K-major operand made of 8-row x 16-byte core matrices (128 contiguous
// bytes each): `lbo` = byte distance between core matrices that follow each other along K,
// `sbo` = along M/N.
__device__ __forceinline__ uint64_t make_smem_desc_noswizzle(uint32_t smem_addr, uint32_t lbo, uint32_t sbo) {
  const uint32_t lo = ((smem_addr & 0x3FFFFu) >> 4) | ((lbo >> 4) << 16);
  const uint32_t hi = (sbo >> 4) | (1u << 14);
  return (static_cast<uint64_t>(hi) << 32) | lo;
}
// Moves the start address of a descriptor by `bytes` (a multiple of 16).
__device__ __forceinline__ uint64_t desc_advance(uint64_t desc, uint32_t bytes) {
  return desc + (bytes >> 4);
}

// Register reallocation between warpgroups (all four warps of a warpgroup must execute it).
template <int N> __device__ __forceinline__ void setmaxnreg_inc() { asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(N)); }
template <int N> __device__ __forceinline__ void setmaxnreg_dec() { asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(N)); }

}  // namespace fmha
