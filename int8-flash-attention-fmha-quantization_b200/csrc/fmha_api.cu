// Host side of libfmha_i8_sm100.so: argument checks, tensor-map encoding, launches and the C ABI
// declared in include/fmha_i8_c.h.  Replaces the reference project's launcher
// (src/fmha_i8.cu:31-173): one runtime-shaped kernel instead of a table of compile-time shapes.
#include <cuda.h>
#include <cuda_runtime.h>
#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <mutex>
#include <type_traits>
#include <utility>

#include "../../include/fmha_i8_c.h"
#include "fmha_debug_sm100.cuh"
#include "fmha_decode_sm100.cuh"
#include "fmha_fwd64_sm100.cuh"
#include "fmha_fwd_sm100.cuh"
#include "fmha_host_sm100.cuh"
#include "fmha_policy_sm100.cuh"
#include "fmha_quant_sm100.cuh"

namespace {

using namespace fmha;

__device__ unsigned g_status_words[8];

thread_local int t_last_status = FMHA_I8_OK;
std::atomic<unsigned long long> g_launch_count{0};

int finish(int status) {
  t_last_status = status;
  return status;
}

constexpr int kMaxDevices = 64;

constexpr int kClusterSizes = 3;
struct DeviceInfo {
  int checked = 0;      // 0 = not yet, 1 = sm_100, -1 = something else
  unsigned* status = nullptr;
  // One word of mapped, pinned host memory per device.  A kernel whose bounded wait runs out writes 1 to
  // it (besides the device status words), so the next host call can see the failure without synchronising.
  volatile unsigned* host_flag = nullptr;
  int sm_count = 0;
  int max_clusters[kClusterSizes] = {};      // clusters of 2, 4, 8 CTAs of the forward kernel that are resident at once
  bool quant_clusters_of_16 = false;         // one cluster of 16 CTAs of the quantiser can be resident
  std::atomic<bool> attr_set{false};         // the kernel attributes are set and what the device was asked about them is filled in
};
DeviceInfo g_dev[kMaxDevices];
std::mutex g_dev_mutex;

// Returns the per-device record of the current device (compute capability check, address of the
// status words, one-time kernel attributes), or nullptr with *err set.
DeviceInfo* current_device(int* err) {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) { *err = FMHA_I8_ERR_LAUNCH; return nullptr; }
  std::lock_guard<std::mutex> lock(g_dev_mutex);
  DeviceInfo& d = g_dev[dev];
  if (d.checked == 0) {
    int major = 0, minor = 0;
    if (cudaDeviceGetAttribute(&major, cudaDevAttrComputeCapabilityMajor, dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&minor, cudaDevAttrComputeCapabilityMinor, dev) != cudaSuccess) {
      *err = FMHA_I8_ERR_LAUNCH;
      return nullptr;
    }
    d.checked = (major == 10 && minor == 0) ? 1 : -1;
    if (cudaDeviceGetAttribute(&d.sm_count, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || d.sm_count < 1) d.sm_count = 1;
  }
  if (d.checked < 0) { *err = FMHA_I8_ERR_WRONG_ARCH; return nullptr; }
  if (!d.status) {
    void* ptr = nullptr;
    if (cudaGetSymbolAddress(&ptr, g_status_words) != cudaSuccess) { *err = FMHA_I8_ERR_LAUNCH; return nullptr; }
    // the host-visible failure word (set-up only: a few bytes of pinned host memory, nothing on the device)
    void* host_word = nullptr;
    void* dev_view = nullptr;
    if (cudaHostAlloc(&host_word, sizeof(unsigned), cudaHostAllocMapped) != cudaSuccess ||
        cudaHostGetDevicePointer(&dev_view, host_word, 0) != cudaSuccess) {
      cudaGetLastError();
      *err = FMHA_I8_ERR_LAUNCH;
      return nullptr;
    }
    *static_cast<volatile unsigned*>(host_word) = 0u;
    if (cudaMemcpyToSymbol(g_host_flag_ptr, &dev_view, sizeof(dev_view)) != cudaSuccess) {
      cudaGetLastError();
      *err = FMHA_I8_ERR_LAUNCH;
      return nullptr;
    }
    d.host_flag = static_cast<volatile unsigned*>(host_word);
    d.status = static_cast<unsigned*>(ptr);
  }
  return &d;
}

template <int D> size_t fwd_smem_bytes() {
  return 1024 + FwdCfg<D>::kTilesBytesTotal + bias_bytes<D>() + sizeof(FwdCtl<FwdCfg<D>::kStagesK, FwdCfg<D>::kStagesV>);
}
template <int D> size_t qk_smem_bytes() { return 1024 + 2 * kTile * D + sizeof(DebugCtl); }
template <int D> size_t pv_smem_bytes() { return 1024 + kTile * D + kTile * kTile + sizeof(DebugCtl); }

template <typename Set> void set_decode_attributes(Set set) {
  auto one = [&](auto d, auto r) {
    constexpr int D = decltype(d)::value, R = decltype(r)::value;
    set(reinterpret_cast<const void*>(&fmha_decode_kernel<D, R>), sizeof(DecodeSmem<D, R>));
  };
  auto rows = [&](auto d) {
    one(d, std::integral_constant<int, 1>());
    one(d, std::integral_constant<int, 2>());
    one(d, std::integral_constant<int, 4>());
  };
  rows(std::integral_constant<int, 64>());
  rows(std::integral_constant<int, 128>());
  one(std::integral_constant<int, 64>(), std::integral_constant<int, 8>());
}

// Calls use(kernel, bytes of shared memory, registers per thread at launch) for every instance of the whole-row policies' kernel.
template <typename Use> void for_policy_kernels(Use use) {
  auto one = [&](auto d) {
    constexpr int D = decltype(d)::value;
    use(reinterpret_cast<const void*>(&wholerow::policy_kernel<D, false, false>), wholerow::smem_bytes<D>(), wholerow::kLaunchRegs);
    use(reinterpret_cast<const void*>(&wholerow::policy_kernel<D, true, false>), wholerow::smem_bytes<D>(), wholerow::kLaunchRegs);
    use(reinterpret_cast<const void*>(&wholerow::policy_kernel<D, true, true>), wholerow::smem_bytes<D>(), wholerow::kLaunchRegs);
  };
  one(std::integral_constant<int, 64>());
  one(std::integral_constant<int, 128>());
}

int set_kernel_attributes(DeviceInfo* d) {
  if (d->attr_set.load(std::memory_order_acquire)) return FMHA_I8_OK;
  std::lock_guard<std::mutex> lock(g_dev_mutex);
  if (d->attr_set.load(std::memory_order_relaxed)) return FMHA_I8_OK;
  cudaError_t e = cudaSuccess;
  auto set = [&](const void* fn, size_t bytes) {
    if (e == cudaSuccess) e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(bytes));
  };
  const void* const general64[] = {reinterpret_cast<const void*>(&fmha_fwd_kernel<64, true>), reinterpret_cast<const void*>(&fmha_fwd_kernel<64, false>)};
  const void* const general128[] = {reinterpret_cast<const void*>(&fmha_fwd_kernel<128, true>), reinterpret_cast<const void*>(&fmha_fwd_kernel<128, false>)};
  for (const void* fn : general64) set(fn, fwd_smem_bytes<64>());
  for (const void* fn : general128) set(fn, fwd_smem_bytes<128>());
  set_decode_attributes(set);
  const void* const workers[] = {reinterpret_cast<const void*>(&w64::fwd_kernel<true, false>), reinterpret_cast<const void*>(&w64::fwd_kernel<false, false>), reinterpret_cast<const void*>(&w64::fwd_kernel<true, true>), reinterpret_cast<const void*>(&w64::fwd_kernel<false, true>)};
  for (const void* fn : workers) set(fn, w64::kSmemBytes);
  for_policy_kernels([&](const void* fn, size_t bytes, int) { set(fn, bytes); });
  set(reinterpret_cast<const void*>(&quant_grid_kernel<false>), kQuantGridSmem);
  set(reinterpret_cast<const void*>(&quant_grid_kernel<true>), kQuantGridSmem);
  if (e == cudaSuccess) e = cudaFuncSetAttribute(reinterpret_cast<const void*>(&quant_cluster_kernel), cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
  set(reinterpret_cast<const void*>(&debug_qk_kernel<64>), qk_smem_bytes<64>());
  set(reinterpret_cast<const void*>(&debug_qk_kernel<128>), qk_smem_bytes<128>());
  set(reinterpret_cast<const void*>(&debug_pv_kernel<64, true>), pv_smem_bytes<64>());
  set(reinterpret_cast<const void*>(&debug_pv_kernel<64, false>), pv_smem_bytes<64>());
  set(reinterpret_cast<const void*>(&debug_pv_kernel<128, true>), pv_smem_bytes<128>());
  set(reinterpret_cast<const void*>(&debug_pv_kernel<128, false>), pv_smem_bytes<128>());
  if (e != cudaSuccess) { cudaGetLastError(); return FMHA_I8_ERR_LAUNCH; }
  // The forward kernel redistributes registers with setmaxnreg; that only terminates if the launch
  // allocation is the one the targets were sized for.
  auto check = [](const void* fn, int regs) {
    cudaFuncAttributes fa{};
    if (cudaFuncGetAttributes(&fa, fn) == cudaSuccess && fa.numRegs == regs) return true;
    cudaGetLastError();
    std::fprintf(stderr, "fmha_i8_sm100: forward kernel built with %d registers per thread, expected %d; refusing to launch\n", fa.numRegs, regs);
    return false;
  };
  bool as_built = true;
  for (const void* fn : general64) as_built = as_built && check(fn, kLaunchRegs);
  for (const void* fn : general128) as_built = as_built && check(fn, kLaunchRegs);
  for (const void* fn : workers) as_built = as_built && check(fn, w64::kLaunchRegs);
  for_policy_kernels([&](const void* fn, size_t, int regs) { as_built = as_built && check(fn, regs); });
  if (!as_built) return FMHA_I8_ERR_LAUNCH;
  for (int i = 0; i < kClusterSizes; ++i) {
    cudaLaunchConfig_t cfg{};
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 2u << i;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    cfg.gridDim = dim3(static_cast<unsigned>(d->sm_count / (2 << i) * (2 << i)));
    cfg.blockDim = dim3(kFwdThreads);
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    int n64 = 0, n128 = 0;
    cfg.dynamicSmemBytes = fwd_smem_bytes<64>();
    if (cudaOccupancyMaxActiveClusters(&n64, fmha_fwd_kernel<64, true>, &cfg) != cudaSuccess) n64 = 0;
    cfg.dynamicSmemBytes = fwd_smem_bytes<128>();
    if (cudaOccupancyMaxActiveClusters(&n128, fmha_fwd_kernel<128, true>, &cfg) != cudaSuccess) n128 = 0;
    cudaGetLastError();
    d->max_clusters[i] = n64 < n128 ? n64 : n128;
  }
  {
    cudaLaunchConfig_t cfg{};
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = kQuantClusterMax;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    cfg.gridDim = dim3(kQuantClusterMax);
    cfg.blockDim = dim3(kQuantClusterThreads);
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    int n = 0;
    d->quant_clusters_of_16 = cudaOccupancyMaxActiveClusters(&n, quant_cluster_kernel, &cfg) == cudaSuccess && n >= 1;
    cudaGetLastError();
  }
  d->attr_set.store(true, std::memory_order_release);
  return FMHA_I8_OK;
}

// Driver entry points, fetched through the runtime so the library has no link-time libcuda dependency.
using EncodeTiledFn = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                   const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                   CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
using ReplaceAddressFn = CUresult (*)(CUtensorMap*, void*);
using PointerAttributeFn = CUresult (*)(void*, CUpointer_attribute, CUdeviceptr);
template <typename Fn> Fn driver_fn(const char* name) {
  void* f = nullptr;
  cudaDriverEntryPointQueryResult q;
  if (cudaGetDriverEntryPoint(name, &f, cudaEnableDefault, &q) != cudaSuccess || q != cudaDriverEntryPointSuccess) return nullptr;
  return reinterpret_cast<Fn>(f);
}
EncodeTiledFn encode_fn() {
  static EncodeTiledFn fn = driver_fn<EncodeTiledFn>("cuTensorMapEncodeTiled");
  return fn;
}
ReplaceAddressFn replace_address_fn() {
  static ReplaceAddressFn fn = driver_fn<ReplaceAddressFn>("cuTensorMapReplaceAddress");
  return fn;
}
PointerAttributeFn pointer_attribute_fn() {
  static PointerAttributeFn fn = driver_fn<PointerAttributeFn>("cuPointerGetAttribute");
  return fn;
}

// int8 tensor [n_heads, S, D] seen as a 3-D map (D innermost) with boxes of 128 rows of one head.
// Rows past S are zero-filled by the copy engine instead of running into the next head.
int make_map(CUtensorMap* map, const void* base, int n_heads, int S, int D, int rows = kTile) {
  EncodeTiledFn fn = encode_fn();
  if (!fn) return FMHA_I8_ERR_DRIVER;
  const cuuint64_t dims[3] = {static_cast<cuuint64_t>(D), static_cast<cuuint64_t>(S), static_cast<cuuint64_t>(n_heads)};
  const cuuint64_t strides[2] = {static_cast<cuuint64_t>(D), static_cast<cuuint64_t>(S) * D};
  const cuuint32_t box[3] = {static_cast<cuuint32_t>(D), static_cast<cuuint32_t>(rows), 1u};
  const cuuint32_t estr[3] = {1u, 1u, 1u};
  const CUtensorMapSwizzle sw = (D == 128) ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_64B;
  const CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_UINT8, 3, const_cast<void*>(base), dims, strides, box, estr,
                        CU_TENSOR_MAP_INTERLEAVE_NONE, sw, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                        CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? FMHA_I8_OK : FMHA_I8_ERR_DRIVER;
}

// The map of another tensor of the same form, in 9 ns instead of the 46 of a new one: two of a call's three where queries and keys are as many, one
// otherwise.  B1 H2 S64 D64, whose time is the host's: 3.66 -> 3.59 us.
int same_map(CUtensorMap* map, const CUtensorMap& of, const void* base) {
  ReplaceAddressFn fn = replace_address_fn();
  if (!fn) return FMHA_I8_ERR_DRIVER;
  *map = of;
  return fn(map, const_cast<void*>(base)) == CUDA_SUCCESS ? FMHA_I8_OK : FMHA_I8_ERR_DRIVER;
}

bool aligned(const void* p, uintptr_t a) { return (reinterpret_cast<uintptr_t>(p) & (a - 1)) == 0; }

// Shape as the kernel sees it: Sq query rows and Sk keys per head (equal for the reference's self-attention).
struct Shape {
  int B, Sq, Sk, H, D;
};

int check_shape_x(const Shape& sh) {
  if (sh.B < 1 || sh.H < 1 || sh.Sk < 64 || sh.Sk > kMaxSeq || (sh.Sk % 64) != 0) return FMHA_I8_ERR_BAD_SHAPE;
  if (sh.Sq < 1 || sh.Sq > kMaxSeq) return FMHA_I8_ERR_BAD_SHAPE;
  if (sh.D != 64 && sh.D != 128) return FMHA_I8_ERR_BAD_SHAPE;
  if (static_cast<long long>(sh.B) * sh.H > 0x7FFFFFFFLL / 2) return FMHA_I8_ERR_BAD_SHAPE;
  return FMHA_I8_OK;
}

int check_shape(const int desc[4]) {
  const Shape sh{desc[0], desc[1], desc[1], desc[2], desc[3]};
  return check_shape_x(sh);
}

// The reference evaluates 1/sqrt(head_dim) with a Newton iteration carried in float
// (inc/fmha_i8.cuh:13-34,71); the same recurrence gives the same constant.
float reference_row_scale(int D) {
  const float x = static_cast<float>(D);
  float curr = x, prev = 0.f;
  while (curr != prev) {
    const float next = static_cast<float>(0.5 * (static_cast<double>(curr) + static_cast<double>(x / curr)));
    prev = curr;
    curr = next;
  }
  return 1.0f / curr;
}

int fill_params(FwdParams* p, const float amax[5], int D, unsigned flags = 0u) {
  for (int i = 0; i < 4; ++i)
    if (!(amax[i] > 0.f) || !std::isfinite(amax[i])) return FMHA_I8_ERR_BAD_AMAX;
  const bool up = (flags & FMHA_I8_FLAG_UINT8_P) != 0u;
  p->row_scale = reference_row_scale(D);
  p->scale_qk = amax[0] * amax[1] / (127.f * 127.f);
  p->scale_v_out = amax[2] * (1.0f / (amax[3] * (up ? 255.f : 128.f)));
  p->p_mul = up ? 255.f : 128.f;
  p->amax_out = nullptr;
  p->amax_scale = amax[2] / ((up ? 255.f : 128.f) * 127.f);   // O~/l counts P in 1/128 (1/255) and V in v_amax/127
  p->c2 = static_cast<float>(static_cast<double>(p->row_scale) * static_cast<double>(p->scale_qk) * 1.4426950408889634);
  if (!(p->c2 > 0.f) || !std::isfinite(p->c2 * kMagic)) return FMHA_I8_ERR_BAD_AMAX;
  p->c2 = std::fmin(std::fmax(p->c2, kMinC2), kMaxC2);
  return FMHA_I8_OK;
}

// How a kernel is launched.  `overlap`: it may start while the kernel before it in the stream drains (the kernel waits for
// that one itself, grid_dependency_wait): the set-up of a call and most of its launch latency leave the critical path.
// Measured: the smallest call 8.4 -> 6.2 us a pass, a one-request encoder call 10.4 -> 8.2 us.
struct LaunchHow {
  bool overlap = false;
  bool cooperative = false;    // the CTAs wait for one another: all of them have to be resident
  unsigned cluster = 0;        // CTAs per cluster, 0 = no clusters
};
template <typename... Params, typename... Args>
int launch_kernel(void (*fn)(Params...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream, const LaunchHow& how, Args&&... args) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[3];
  cfg.attrs = attr;
  if (how.overlap) {
    attr[cfg.numAttrs].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[cfg.numAttrs++].val.programmaticStreamSerializationAllowed = 1;
  }
  if (how.cooperative) {
    attr[cfg.numAttrs].id = cudaLaunchAttributeCooperative;
    attr[cfg.numAttrs++].val.cooperative = 1;
  }
  if (how.cluster != 0) {
    attr[cfg.numAttrs].id = cudaLaunchAttributeClusterDimension;
    attr[cfg.numAttrs].val.clusterDim.x = how.cluster;
    attr[cfg.numAttrs].val.clusterDim.y = 1;
    attr[cfg.numAttrs++].val.clusterDim.z = 1;
  }
  g_launch_count.fetch_add(1, std::memory_order_relaxed);
  if (cudaLaunchKernelEx(&cfg, fn, std::forward<Args>(args)...) == cudaSuccess) return FMHA_I8_OK;
  cudaGetLastError();
  return FMHA_I8_ERR_LAUNCH;
}

// CTAs that share one unit (query tile), each with a part of its key tiles: for calls whose units leave most SMs idle, as long as
// all clusters are resident at once (a second wave of them starts from nothing and costs 10 us).  In nanoseconds, measured: 860
// per key tile of a CTA, and for cluster launch, two cluster barriers and the merge of the partial results through distributed
// shared memory, with 2, 4 and 8 CTAs, kShareNs for up to 64 rows at head_dim 128 or 128 at 64, kShareMoreNs more for twice as many:
constexpr int kTileNs = 860;
constexpr int kShareNs[kClusterSizes] = {3300, 2900, 4300}, kShareMoreNs[kClusterSizes] = {700, 1900, 1700};
// us without -> with: head_dim 64 B1 H8 S1024 Sq256 10.9 -> 8.7, B1 H8 S8192 Sq64 57.9 -> 16.9; head_dim 128 B2 H16 S1984 Sq200 19.1 -> 15.6, B1 H2
// S16384 Sq128 114 -> 27.  Where the line lies, 12 units of 128 rows with 1 / 2 / 4 CTAs each: head_dim 64, 5 tiles 8.3 / 8.9 / 8.5, 6 tiles 9.1 / 8.9 /
// 8.6; head_dim 128, 7 tiles 10.7 / 11.0 / 11.2, 8 tiles 11.6 / 11.2 / 11.2, 12 tiles 15.1 / 13.1 / 12.1.
// Pairs are for so many units that larger clusters do not fit, and more CTAs make the merge longer: 72 units of 6 tiles at head_dim 64, one CTA
// each / pairs, 8.2 / 9.15, 70 units of 8 tiles 9.8 / 9.85 and at head_dim 128 11.9 / 12.9 (with 12 units pairs would cost 2700).
//
// With more units than SMs the same is done for those of the last round: where they are half as many as the SMs or fewer, a pair
// of CTAs shares each.  Head_dim 128: B1 H16 S1280 23.1 -> 21.8 us, B1 H5 S4096 60.9 -> 50.2, B1 H32 S2048 61.7 -> 58.0; where the line lies, 208
// units of 6 tiles 16.3 -> 16.5, of 8 tiles 19.8 -> 19.4; head_dim 64, of 5 tiles 13.1 -> 13.8, of 6 tiles 14.9 -> 14.7.  (kTileNs, kPairNs and the figures of
// this paragraph are of kernels 4 % slower than the present ones.)
constexpr int kPairNs = 2400;
bool pairs_share_last_round(const FwdParams& p, const DeviceInfo* dev) {
  const int last = p.n_units % dev->sm_count, tiles = (p.S + kTile - 1) / kTile;
  return p.n_units > dev->sm_count && last > 0 && last <= dev->max_clusters[0] && 2 * dev->max_clusters[0] == dev->sm_count &&
         kTileNs * (tiles / 2) > kPairNs;
}
// ceil(2^(31 + bits) / d) with 2^bits >= d > 2^(bits - 1): the quotient is exact for every dividend below 2^31.
FastDiv fast_div_by(int d) {
  int bits = 0;
  while ((1ll << bits) < d) ++bits;
  const uint64_t one = 1ull << (31 + bits);
  return FastDiv{static_cast<uint32_t>((one + static_cast<uint64_t>(d) - 1) / static_cast<uint64_t>(d)), 31 + bits};
}

void plan_parts(FwdParams* p, int D, const DeviceInfo* dev) {
  const int tiles = (p->S + kTile - 1) / kTile;
  p->own_rounds = p->n_units / dev->sm_count;
  if (p->own_rounds > 0) {
    if (pairs_share_last_round(*p, dev)) p->parts = 2;
    return;
  }
  const int outputs = (p->Sq < kTile ? p->Sq : kTile) * D, more = outputs > 8192 ? outputs - 8192 : 0;
  int best_ns = kTileNs * tiles;
  for (int i = 0; i < kClusterSizes; ++i) {
    const int c = 2 << i, ns = kTileNs * ((tiles + c - 1) / c) + kShareNs[i] + kShareMoreNs[i] * more / 8192;
    if (p->n_units <= dev->max_clusters[i] && ns < best_ns) { p->parts = c; best_ns = ns; }
  }
}

// Which of the two kernels a call at head_dim 64 runs: the one whose estimate is smaller, in cycles.  A CTA of fmha_fwd_sm100.cuh works on one
// unit at a time: 1530 per key tile and 650 per unit, 2900 at least (2400 in a last round of single tiles that leaves SMs idle); pairs that share the
// last round 980 and 3700.  One of fmha_fwd64_sm100.cuh works on four: 5350 per tile and 2500 for a round of four; 3100 / 3700 / 4700 / 5850 per tile
// and 2000 (one tile: 1200) for a last round of one to four; 600 for the call.  The half tile of an odd multiple of 64 keys is six tenths there.
// Fitted to 221 shapes of 100 to 3500 query tiles of 64 to 2048 keys, when the kernels were 4 to 9 % slower; since, over 61 of them (160 to 2368 units
// of 64 to 512 keys), the kernel chosen is 0.6 % slower than the better one on average and 4.4 % at the most (888 units of 320 keys).
// us, fmha_fwd_sm100.cuh / fmha_fwd64_sm100.cuh: 160 units of 64 keys 5.0 / 4.7; 160, 222, 444 of 128 5.1 / 5.5, 5.4 / 5.9, 7.3 / 6.95; 296, 592, 740, 1184
// of 256 7.4 / 8.4, 11.3 / 11.6, 13.1 / 14.8, 18.7 / 18.4; 444 of 512 14.0 / 14.8; of the slower kernels 592 and 888 of 1024 31.2 / 30.2, 44.8 / 46.25.
//
// Calibrations have a line of their own (1600 and 1200; 5850, 4900 / 4350 / 3400 per tile), of the slower kernels too.
bool use_workers(const FwdParams& p, bool plain, const DeviceInfo* dev) {
  const long long sms = dev->sm_count, tiles = (p.S + kTile - 1) / kTile, round = sms * w64::kWorkers;
  const long long own = p.n_units / sms, more = p.n_units % sms != 0, full = p.n_units / round, last = (p.n_units % round + sms - 1) / sms;
  if (plain) {
    const long long per_tile[w64::kWorkers + 1] = {0, 3100, 3700, 4700, 5850};
    const long long tenths = 10 * tiles - (p.S % kTile != 0 ? 4 : 0), unit = std::max(1530 * tiles + 650, 2900LL);
    const long long workers = 600 + full * (535 * tenths + 2500) + (last > 0 ? per_tile[last] * tenths / 10 + (tiles > 1 ? 2000 : 1200) : 0);
    return workers < own * unit + more * (pairs_share_last_round(p, dev) ? 980 * tiles + 3700 : tiles > 1 ? unit : unit - 500);
  }
  const long long per_tile[w64::kWorkers + 1] = {0, 3400, 4350, 4900, 5850}, unit = 1600 * tiles + 1200;
  return (full * 5850 + per_tile[last]) * tiles < own * unit + more * (pairs_share_last_round(p, dev) ? unit / 2 + 4500 : unit);
}

// Few query rows run the few-rows kernel.  Up to four rows it is bound by reading K and V; from five on (computed as eight) its integer dot
// products take as long or longer.  us, few-rows / general kernel:
//   D128, 1 row   B16 H32 S4096 (1025..4096 keys) 55.3 / 82.9
//   D128, 8 rows  B128 H32 S64 90.9 / 62.0, B64 H32 S256 50.1 / 40.2, B32 H32 S1024 71.8 / 61.5, B8 H32 S4096 83.3 / 63.2, B1 H8 S16384
//                 77.3 / 25.3, and so on: the general one at every length and number of heads measured
//   D64, 8 rows   B128 H32 S128 61.0 / 32.9, B1 H4 S128 5.9 / 4.7: the general one for a single key tile; beyond, with many heads, the
//                 few-rows one (B32 H32 S512 23.9 / 29.9, B8 H32 S4096 47.5 / 60.2), with few heads either (B1 H32 S2048 13.3 / 9.9)
//   D64, 4 rows   B128 H32 S128 42.6 / 32.9, S256 and beyond the few-rows one or within a few per cent
bool few_rows(int Sq, int S, int D) { return Sq <= 4 || (D == 64 && Sq <= kDecodeMaxRows && S > kTile); }

// Chooses the kernel of a call and how its units are divided: fills p->parts and p->own_rounds.  `plain`: no calibration; `busy_sms`: SMs that
// something else is using.
int plan_call(FwdParams* p, int D, int policy, bool plain, int busy_sms, const DeviceInfo* dev) {
  p->parts = 1;
  if (policy != FMHA_I8_POLICY_TILE) return FMHA_I8_KERNEL_POLICY;
  if (plain && few_rows(p->Sq, p->S, D)) return FMHA_I8_KERNEL_FEW_ROWS;
  if (D == 64 && use_workers(*p, plain, dev)) return FMHA_I8_KERNEL_WORKERS;
  if (plain && busy_sms == 0) plan_parts(p, D, dev);
  return FMHA_I8_KERNEL_GENERAL;
}

template <int D>
int launch_policy(cudaStream_t stream, DeviceInfo* dev, const FwdParams& p, const void* q, const void* k, const void* v, bool is_static) {
  CUtensorMap mq, mk, mv;
  int st;
  if ((st = make_map(&mq, q, p.bh_count, p.Sq, D)) != FMHA_I8_OK) return st;
  if ((st = make_map(&mk, k, p.bh_count, p.S, D, wholerow::kKeys)) != FMHA_I8_OK) return st;
  if ((st = same_map(&mv, mk, v)) != FMHA_I8_OK) return st;
  LaunchHow how;
  how.overlap = true;
  const unsigned grid = static_cast<unsigned>(p.n_units < dev->sm_count ? p.n_units : dev->sm_count);
  auto* fn = !is_static ? wholerow::policy_kernel<D, false, false> : p.S <= wholerow::kStep1 ? wholerow::policy_kernel<D, true, true> : wholerow::policy_kernel<D, true, false>;
  return launch_kernel(fn, dim3(grid), dim3(wholerow::kThreads), wholerow::smem_bytes<D>(), stream, how, mq, mk, mv, p);
}

template <int D>
int launch_fwd(cudaStream_t stream, DeviceInfo* dev, const FwdParams& p, const void* q, const void* k, const void* v, int kernel, int busy_sms) {
  CUtensorMap mq, mk, mv;
  int st;
  if ((st = make_map(&mq, q, p.bh_count, p.Sq, D)) != FMHA_I8_OK) return st;
  if ((st = p.S == p.Sq ? same_map(&mk, mq, k) : make_map(&mk, k, p.bh_count, p.S, D)) != FMHA_I8_OK) return st;
  if ((st = same_map(&mv, mk, v)) != FMHA_I8_OK) return st;
  // Overlap takes the launch latency and the set-up of a launch out of the time of calls in a row; a call that nothing precedes gains
  // nothing.  (Per cent of the time with more than four rounds of units: B32 H12 S512 D64 with lengths 256..512 -6, B200 H12 S128 -9, B4 H32
  // S1024 D128 -4, B64 H32 S256 -4, B8 H32 S2048 and B256 H16 S256 D64 with lengths 64..256 -1 to 0.)  Its price: the CTAs of the next launch
  // take an SM as soon as this one leaves it, and wait there for the last of this one; a kernel of another stream that would have run
  // on such SMs meanwhile comes after them.
  LaunchHow how;
  how.overlap = true;
  // persistent CTAs: one per SM (tensor memory is allocated whole), each walking its share of the units
  const int sms = dev->sm_count - busy_sms;
  unsigned grid = static_cast<unsigned>(p.n_units < sms ? p.n_units : sms);
  if constexpr (D == 64) {
    if (kernel == FMHA_I8_KERNEL_WORKERS) {
      const bool few = p.S <= w64::kShortTiles * kTile;
      auto* fn = p.amax_out != nullptr ? (few ? w64::fwd_kernel<true, true> : w64::fwd_kernel<false, true>) : few ? w64::fwd_kernel<true, false> : w64::fwd_kernel<false, false>;
      return launch_kernel(fn, dim3(grid), dim3(w64::kThreads), w64::kSmemBytes, stream, how, mq, mk, mv, p);
    }
  }
  if (p.parts > 1) {
    how.cluster = static_cast<unsigned>(p.parts);
    grid = static_cast<unsigned>(p.own_rounds > 0 ? dev->sm_count : p.n_units * p.parts);
  }
  auto* fn = p.parts > 1 || p.amax_out != nullptr ? fmha_fwd_kernel<D, true> : fmha_fwd_kernel<D, false>;
  return launch_kernel(fn, dim3(grid), dim3(kFwdThreads), fwd_smem_bytes<D>(), stream, how, mq, mk, mv, p);
}

// The few-rows kernel.  CTAs per head: enough for two rounds of the 3 CTAs that an SM holds, so that heads of different
// length even out, as long as a warp keeps two tiles (B16 H32, 1025..4096 keys, one row, clusters of 1 / 2 / 4 / 8: 60.9 / 55.3 / 59.0 /
// 80.2 us, the last where the set-up of a CTA outweighs its tiles); where even that leaves SMs idle, down
// to one tile per warp.
template <int D, int R>
int launch_decode_rows(cudaStream_t stream, DeviceInfo* dev, FwdParams p, const void* q, const void* k, const void* v) {
  constexpr int W = DecodeCfg<D>::kWarps;
  p.q_tiles = (p.Sq + R - 1) / R;
  const long long units = static_cast<long long>(p.bh_count) * p.q_tiles;
  const int n_tiles = (p.S + kTile - 1) / kTile;
  const long long resident = 3LL * dev->sm_count;
  int c = 1;
  constexpr int kMaxCtas = R == 8 ? kDecodeMaxCluster / 2 : kDecodeMaxCluster;      // their partial results fit into the tiles of one CTA
  static_assert(kMaxCtas * W * R * DecodeCfg<D>::kPartFloats * 4 <= DecodeCfg<D>::kRingBytes, "partial results do not fit");
  while (c < kMaxCtas && ((units * c < 2 * resident && n_tiles >= 4 * c * W) || (units * c * 2 <= resident && n_tiles >= 2 * c * W))) c *= 2;
  if (units * c > 0x7FFFFFFFLL) return FMHA_I8_ERR_BAD_SHAPE;
  LaunchHow how;
  how.cluster = static_cast<unsigned>(c);
  how.overlap = true;
  return launch_kernel(fmha_decode_kernel<D, R>, dim3(static_cast<unsigned>(units * c)), dim3(DecodeCfg<D>::kThreads),
                       sizeof(DecodeSmem<D, R>), stream, how, static_cast<const int8_t*>(q), static_cast<const int8_t*>(k),
                       static_cast<const int8_t*>(v), p);
}
template <int D>
int launch_decode(cudaStream_t s, DeviceInfo* dev, const FwdParams& p, const void* q, const void* k, const void* v) {
  if (p.Sq == 1) return launch_decode_rows<D, 1>(s, dev, p, q, k, v);
  if (p.Sq == 2) return launch_decode_rows<D, 2>(s, dev, p, q, k, v);
  if constexpr (D == 64) {
    if (p.Sq > 4) return launch_decode_rows<D, 8>(s, dev, p, q, k, v);
  }
  return launch_decode_rows<D, 4>(s, dev, p, q, k, v);
}

int fill_units(FwdParams* p, const Shape& sh, int bh_count) {
  p->S = sh.Sk;
  p->Sq = sh.Sq;
  p->H = sh.H;
  p->bh_count = bh_count;
  p->q_tiles = (p->Sq + kTile - 1) / kTile;
  p->by_q_tiles = fast_div_by(p->q_tiles);
  p->by_heads = fast_div_by(p->H);
  const long long units = static_cast<long long>(bh_count) * p->q_tiles;
  if (units > 0x7FFFFFFFLL) return FMHA_I8_ERR_BAD_SHAPE;
  p->n_units = static_cast<int>(units);
  return FMHA_I8_OK;
}

int infer_x_impl(void* stream, const float amax[5], const Shape& sh, const void* q, const void* k,
                 const void* v, const void* mask, void* o, int bh_begin, int bh_count, unsigned flags,
                 float* calib = nullptr, int policy = FMHA_I8_POLICY_TILE, int busy_sms = 0) {
  if (!amax || !q || !k || !v || !mask || (!o && !calib)) return FMHA_I8_ERR_NULL_POINTER;
  if (!(flags & FMHA_I8_FLAG_USE_TCU)) return FMHA_I8_ERR_NO_CUDA_CORE_PATH;
  if (flags & ~(FMHA_I8_FLAG_USE_TCU | FMHA_I8_FLAG_UINT8_P)) return FMHA_I8_ERR_BAD_FLAGS;
  int st = check_shape_x(sh);
  if (st != FMHA_I8_OK) return st;
  const long long BH = static_cast<long long>(sh.B) * sh.H;
  if (bh_begin < 0 || bh_count < 1 || static_cast<long long>(bh_begin) + bh_count > BH) return FMHA_I8_ERR_BAD_SLICE;
  if (!aligned(q, 16) || !aligned(k, 16) || !aligned(v, 16) || !aligned(o, 16) || !aligned(mask, 4) || !aligned(calib, 4))
    return FMHA_I8_ERR_MISALIGNED;
  FwdParams p{};
  if ((st = fill_params(&p, amax, sh.D, flags)) != FMHA_I8_OK) return st;
  p.amax_out = calib;
  const bool is_static = policy == FMHA_I8_POLICY_STATIC;
  if (policy != FMHA_I8_POLICY_TILE) {
    // fmha_i8_quant_deviation.py:7,38-43: 127 levels, unsigned, P8 = clip(rn(p * 127 / p_amax), 0, 127).
    // Per-row ("dynamic", :104-118): p_amax = the row's largest probability = 1/l, so P8 = rn(127 e) and the output
    // is (sum P8 v8) / (127 l) * v_amax/127.  Static (:82-98): p_amax = s_max for every row, so
    // P8 = min(rn(127 e / (l s_max)), 127) and the output is (sum P8 v8) * s_max/127 * v_amax/127.
    const float levels = wholerow::kLevels;
    if (is_static && (!(amax[4] > 0.f) || !std::isfinite(amax[4]))) return FMHA_I8_ERR_BAD_AMAX;
    p.p_mul = is_static ? 1.f / amax[4] : levels;
    p.scale_v_out = is_static ? amax[4] * amax[2] / (levels * amax[3]) : amax[2] / (levels * amax[3]);
  }
  int err = FMHA_I8_OK;
  DeviceInfo* dev = current_device(&err);
  if (!dev) return err;
  if ((st = set_kernel_attributes(dev)) != FMHA_I8_OK) return st;
  // A kernel launched earlier gave up on a bounded wait (its output is invalid): say so ONCE, on the first call
  // that can see it, without launching; the details stay in the status words until fmha_i8_sm100_device_status().
  if (*dev->host_flag != 0u) {
    *dev->host_flag = 0u;
    return FMHA_I8_ERR_DEVICE;
  }
  p.mask = static_cast<const int8_t*>(mask);
  p.o = static_cast<int8_t*>(o);
  p.o_wide = aligned(o, 32) ? 1 : 0;
  p.bh_begin = bh_begin;
  if ((st = fill_units(&p, sh, bh_count)) != FMHA_I8_OK) return st;
  p.status = dev->status;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const int kernel = plan_call(&p, sh.D, policy, !calib, busy_sms, dev);
  auto launch = [&](auto d) {
    constexpr int D = decltype(d)::value;
    if (kernel == FMHA_I8_KERNEL_POLICY) return launch_policy<D>(s, dev, p, q, k, v, is_static);
    if (kernel == FMHA_I8_KERNEL_FEW_ROWS) return launch_decode<D>(s, dev, p, q, k, v);
    return launch_fwd<D>(s, dev, p, q, k, v, kernel, busy_sms);
  };
  return sh.D == 128 ? launch(std::integral_constant<int, 128>()) : launch(std::integral_constant<int, 64>());
}

int infer_slice_impl(void* stream, const float amax[5], const int desc[4], const void* q, const void* k,
                     const void* v, const void* mask, void* o, int bh_begin, int bh_count, unsigned flags, int busy_sms = 0) {
  if (!desc) return FMHA_I8_ERR_NULL_POINTER;
  const Shape sh{desc[0], desc[1], desc[1], desc[2], desc[3]};
  return infer_x_impl(stream, amax, sh, q, k, v, mask, o, bh_begin, bh_count, flags, nullptr, FMHA_I8_POLICY_TILE, busy_sms);
}

// Device staging buffers of fmha_i8_sm100_infer_host, one set per device, grown on demand, plus the
// three streams and the events of its copy/compute pipeline.
constexpr int kHostChunks = 8;
struct HostStaging {
  void* q = nullptr; void* k = nullptr; void* v = nullptr; void* o = nullptr; void* mask = nullptr;
  size_t tensor_cap = 0, mask_cap = 0;
  cudaStream_t s_in = nullptr, s_run = nullptr, s_out = nullptr;
  cudaEvent_t landed[kHostChunks] = {}, computed[kHostChunks] = {};
  bool ready = false;
};
HostStaging g_staging[kMaxDevices];
std::mutex g_staging_mutex[kMaxDevices];     // one lock per device: host threads that drive different GPUs do not wait for each other

// How the inputs of a host-buffer call come in.  A kernel can leave rows of masked keys out and costs 5 us per chunk; the copy
// engine is 7 % faster per byte, 50.7 and 54.7 GB/s, but needs three copies of 4 us each.  (Both ways of the link together carry
// no more than 70 GB/s, so either pays for the output as well.)  The kernel needs pinned, device-readable, 16-byte aligned buffers,
// and takes its SMs from the forward kernels, so it is left where those, not the link, take the time: long sequences.
constexpr int kHostLongSeq = 4096;
struct FetchPlan {
  bool by_kernel = false;
  const void *q = nullptr, *k = nullptr, *v = nullptr;     // device addresses of the host buffers
};
// Device address of a host buffer, if all of it lies in one pinned, device-readable block (allocated or registered) and is 16-byte
// aligned; nullptr otherwise.  A kernel that reads past the registered part of a buffer faults, a copy is refused by the runtime.
const void* device_view(const void* host, size_t bytes) {
  cudaPointerAttributes attr{};
  if (cudaPointerGetAttributes(&attr, host) != cudaSuccess) { cudaGetLastError(); return nullptr; }
  if (attr.type != cudaMemoryTypeHost || attr.devicePointer == nullptr || !aligned(attr.devicePointer, 16)) return nullptr;
  const PointerAttributeFn query = pointer_attribute_fn();
  const CUdeviceptr at = reinterpret_cast<CUdeviceptr>(attr.devicePointer);
  CUdeviceptr block = 0;
  size_t block_bytes = 0;
  if (!query || query(&block, CU_POINTER_ATTRIBUTE_RANGE_START_ADDR, at) != CUDA_SUCCESS ||
      query(&block_bytes, CU_POINTER_ATTRIBUTE_RANGE_SIZE, at) != CUDA_SUCCESS || at < block || at - block > block_bytes ||
      bytes > block_bytes - (at - block))
    return nullptr;
  return attr.devicePointer;
}
FetchPlan plan_fetch(const int desc[4], const void* host_q, const void* host_k, const void* host_v, const int8_t* host_mask, int bh_begin, int bh_count, int n_chunks) {
  FetchPlan plan;
  const int S = desc[1], H = desc[2], D = desc[3];
  if (S > kHostLongSeq) return plan;
  // (the mask is read here by the host; one that lives on the device is left to the copies and what the runtime says to them)
  cudaPointerAttributes of_mask{};
  if (cudaPointerGetAttributes(&of_mask, host_mask) != cudaSuccess) { cudaGetLastError(); return plan; }
  if (of_mask.type == cudaMemoryTypeDevice) return plan;
  // rows that come in: all of Q, the groups of keys with an unmasked one (of the batches that the slice touches)
  double rows = static_cast<double>(bh_count) * S;
  for (int b = bh_begin / H; b <= (bh_begin + bh_count - 1) / H; ++b) {
    const int first = b * H > bh_begin ? b * H : bh_begin, last = (b + 1) * H < bh_begin + bh_count ? (b + 1) * H : bh_begin + bh_count;
    const int8_t* m = host_mask + static_cast<size_t>(b) * S;
    int groups = 0;
    for (int g = 0; g < S; g += kFetchRows) groups += std::memchr(m + g, 0, kFetchRows) != nullptr;
    rows += 2.0 * (last - first) * groups * kFetchRows;
  }
  const double us_kernel = rows * D / 50.7e3 + 5.0 * n_chunks, us_copies = 3.0 * bh_count * S * D / 54.7e3 + 12.0 * n_chunks;
  if (us_kernel > us_copies) return plan;
  const size_t bytes = static_cast<size_t>(bh_count) * S * D;
  plan.q = device_view(host_q, bytes);
  plan.k = plan.q ? device_view(host_k, bytes) : nullptr;
  plan.v = plan.k ? device_view(host_v, bytes) : nullptr;
  plan.by_kernel = plan.v != nullptr;
  return plan;
}

// Cuts the heads of a host-buffer call into the chunks of its pipeline; returns their number.
// Each piece of the inbound transfer costs some microseconds, so there are few; what follows the last of them -- its kernel
// and its outbound copy -- is exposed, so the pieces shrink by halves: a chunk's outbound copy, a third of its inbound
// bytes, is hidden behind the next chunk's inbound transfer.  Long sequences, where the kernels take the time, are cut evenly.
// (us, eight even chunks of three copies -> this: B32 H12 S512 D64 with lengths 256..512 976 -> 846, without padding 979 -> 890,
// B8 H12 S512 with lengths 300..512 340 -> 244, B1 H4 S256 82 -> 36, B4 H32 S2048 D128 2350 -> 2168.)
int cut_heads(const int desc[4], int bh_count, int (&bounds)[kHostChunks + 1]) {
  const int BH = bh_count;
  const size_t bytes_in = 3 * static_cast<size_t>(bh_count) * desc[1] * desc[3];
  const bool even = desc[1] > kHostLongSeq;
  const int wanted = even ? kHostChunks : bytes_in < (3u << 19) ? 1 : bytes_in < (6u << 20) ? 2 : bytes_in < (64u << 20) ? 4 : 6;
  const int n_chunks = BH < wanted ? BH : wanted;
  bounds[0] = 0;
  for (int i = 1; i <= n_chunks; ++i) {
    const double done = even ? static_cast<double>(i) / n_chunks : (1.0 - std::ldexp(1.0, -i)) / (1.0 - std::ldexp(1.0, -n_chunks));
    const int rounded = static_cast<int>(std::lround(done * BH)), least = bounds[i - 1] + 1, most = BH - (n_chunks - i);     // every chunk has a head
    bounds[i] = rounded < least ? least : rounded > most ? most : rounded;
  }
  return n_chunks;
}

int check_quant_args(const float* x, long long n, const int8_t* out) {
  if (!x || !out) return FMHA_I8_ERR_NULL_POINTER;
  if (n < 1) return FMHA_I8_ERR_BAD_SHAPE;
  if (!aligned(x, 16) || !aligned(out, 16)) return FMHA_I8_ERR_MISALIGNED;
  return FMHA_I8_OK;
}

// The largest tensor of fmha_i8_sm100_quantize_f32_noalloc (1 GiB of fp32), part of its contract.
constexpr long long kNoAllocMaxElements = 268435456LL;

// Up to what the registers of one cluster hold: one cluster -- of 16 CTAs where the device has room for one together (more than 8 is
// not a size that every device or partition of one offers), of 8 otherwise.  Beyond: the whole chip, every CTA with work for all its warps.
int launch_quantize(cudaStream_t stream, DeviceInfo* dev, const float* x, long long n, int8_t* out, float* amax_out, bool whole_chip) {
  LaunchHow how;
  if (!whole_chip && n <= (dev->quant_clusters_of_16 ? kQuantClusterMax : kQuantClusterPortable) * kQuantPerCta) {
    how.cluster = static_cast<unsigned>(quant_cluster_size(n));
    how.overlap = true;
    return launch_kernel(quant_cluster_kernel, dim3(how.cluster), dim3(kQuantClusterThreads), 0, stream, how, x, static_cast<int>(n), out, amax_out);
  }
  if (n / kQuantTile > 0x7FFFFFFFLL) return FMHA_I8_ERR_TOO_LARGE;
  how.cooperative = true;
  const long long wanted = (n / kQuantTile + kQuantWarps - 1) / kQuantWarps;
  const int most = dev->sm_count < kQuantMaxCtas ? dev->sm_count : kQuantMaxCtas;
  const int ctas = static_cast<int>(wanted < most ? wanted : most);
  auto* kernel = quant_needs_tmem(n, ctas) ? quant_grid_kernel<true> : quant_grid_kernel<false>;
  return launch_kernel(kernel, dim3(static_cast<unsigned>(ctas)), dim3(kQuantThreads), kQuantGridSmem, stream, how, x, n, out, amax_out, dev->status);
}

int quantize_impl(void* stream, const float* x, long long n, int8_t* out, float* amax_out, bool whole_chip = false) {
  int err = FMHA_I8_OK;
  DeviceInfo* dev = current_device(&err);
  if (!dev) return err;
  const int st = set_kernel_attributes(dev);
  return st != FMHA_I8_OK ? st : launch_quantize(static_cast<cudaStream_t>(stream), dev, x, n, out, amax_out, whole_chip);
}

}  // namespace

extern "C" {

int fmha_i8_sm100_infer(void* stream, const float amax[5], const int desc[4], const void* q, const void* k,
                        const void* v, const void* mask, void* o, unsigned flags) {
  if (!desc) return finish(FMHA_I8_ERR_NULL_POINTER);
  const long long BH = static_cast<long long>(desc[0]) * desc[2];
  if (BH < 1 || BH > 0x7FFFFFFFLL) return finish(FMHA_I8_ERR_BAD_SHAPE);
  return finish(infer_slice_impl(stream, amax, desc, q, k, v, mask, o, 0, static_cast<int>(BH), flags));
}

int fmha_i8_sm100_infer_slice(void* stream, const float amax[5], const int desc[4], const void* q, const void* k,
                              const void* v, const void* mask, void* o, int bh_begin, int bh_count, unsigned flags) {
  return finish(infer_slice_impl(stream, amax, desc, q, k, v, mask, o, bh_begin, bh_count, flags));
}

int fmha_i8_sm100_infer_cross(void* stream, const float amax[5], const int desc5[5], const void* q, const void* k,
                              const void* v, const void* mask, void* o, int bh_begin, int bh_count, unsigned flags) {
  if (!desc5) return finish(FMHA_I8_ERR_NULL_POINTER);
  const Shape sh{desc5[0], desc5[1], desc5[2], desc5[3], desc5[4]};
  return finish(infer_x_impl(stream, amax, sh, q, k, v, mask, o, bh_begin, bh_count, flags));
}

int fmha_i8_sm100_infer_policy(void* stream, const float amax[5], const int desc5[5], const void* q, const void* k,
                               const void* v, const void* mask, void* o, int bh_begin, int bh_count, unsigned flags,
                               int policy, float* row_scratch) {
  if (!desc5) return finish(FMHA_I8_ERR_NULL_POINTER);
  const Shape sh{desc5[0], desc5[1], desc5[2], desc5[3], desc5[4]};
  if (policy == FMHA_I8_POLICY_TILE) return finish(infer_x_impl(stream, amax, sh, q, k, v, mask, o, bh_begin, bh_count, flags));
  if (policy != FMHA_I8_POLICY_ROW && policy != FMHA_I8_POLICY_STATIC) return finish(FMHA_I8_ERR_BAD_FLAGS);
  if (flags & FMHA_I8_FLAG_UINT8_P) return finish(FMHA_I8_ERR_BAD_FLAGS);       // the policies bring their own P format
  if (!row_scratch || !o) return finish(FMHA_I8_ERR_NULL_POINTER);
  if (!aligned(row_scratch, 8)) return finish(FMHA_I8_ERR_MISALIGNED);
  return finish(infer_x_impl(stream, amax, sh, q, k, v, mask, o, bh_begin, bh_count, flags, nullptr, policy));
}

int fmha_i8_sm100_calibrate_o_amax(void* stream, const float amax[5], const int desc5[5], const void* q, const void* k,
                                   const void* v, const void* mask, float* o_amax_out, unsigned flags) {
  if (!desc5 || !amax || !o_amax_out) return finish(FMHA_I8_ERR_NULL_POINTER);
  const Shape sh{desc5[0], desc5[1], desc5[2], desc5[3], desc5[4]};
  const long long BH = static_cast<long long>(sh.B) * sh.H;
  if (BH < 1 || BH > 0x7FFFFFFFLL) return finish(FMHA_I8_ERR_BAD_SHAPE);
  // o_amax is what is being determined: any positive placeholder passes the argument check
  const float a[5] = {amax[0], amax[1], amax[2], 1.0f, 1.0f};
  if (cudaMemsetAsync(o_amax_out, 0, sizeof(float), static_cast<cudaStream_t>(stream)) != cudaSuccess) {
    cudaGetLastError();
    return finish(FMHA_I8_ERR_LAUNCH);
  }
  return finish(infer_x_impl(stream, a, sh, q, k, v, mask, nullptr, 0, static_cast<int>(BH), flags, o_amax_out));
}

// Host buffers in, host buffer out, for heads [bh_begin, bh_begin + bh_count): host_q/k/v/o point at the first head
// of the slice, host_mask is the whole [B,S] mask.
static int infer_host_slice_impl(const float amax[5], const int desc[4], const void* host_q, const void* host_k,
                                 const void* host_v, const void* host_mask, void* host_o, int bh_begin, int bh_count, unsigned flags) {
  if (!amax || !desc || !host_q || !host_k || !host_v || !host_mask || !host_o) return FMHA_I8_ERR_NULL_POINTER;
  int st = check_shape(desc);
  if (st != FMHA_I8_OK) return st;
  const long long BH_all = static_cast<long long>(desc[0]) * desc[2];
  if (bh_begin < 0 || bh_count < 1 || static_cast<long long>(bh_begin) + bh_count > BH_all) return FMHA_I8_ERR_BAD_SLICE;
  int dev_id = 0;
  if (cudaGetDevice(&dev_id) != cudaSuccess || dev_id < 0 || dev_id >= kMaxDevices) return FMHA_I8_ERR_LAUNCH;
  const size_t head_bytes = static_cast<size_t>(desc[1]) * desc[3];
  const size_t tensor_bytes = static_cast<size_t>(bh_count) * head_bytes;
  const size_t mask_bytes = static_cast<size_t>(desc[0]) * desc[1];
  std::lock_guard<std::mutex> lock(g_staging_mutex[dev_id]);
  HostStaging& s = g_staging[dev_id];
  if (!s.ready) {
    bool good = cudaStreamCreateWithFlags(&s.s_in, cudaStreamNonBlocking) == cudaSuccess &&
                cudaStreamCreateWithFlags(&s.s_run, cudaStreamNonBlocking) == cudaSuccess &&
                cudaStreamCreateWithFlags(&s.s_out, cudaStreamNonBlocking) == cudaSuccess;
    for (int i = 0; i < kHostChunks && good; ++i)
      good = cudaEventCreateWithFlags(&s.landed[i], cudaEventDisableTiming) == cudaSuccess &&
             cudaEventCreateWithFlags(&s.computed[i], cudaEventDisableTiming) == cudaSuccess;
    if (!good) { cudaGetLastError(); return FMHA_I8_ERR_LAUNCH; }
    s.ready = true;
  }
  if (s.tensor_cap < tensor_bytes) {
    cudaFree(s.q); cudaFree(s.k); cudaFree(s.v); cudaFree(s.o);
    s.q = s.k = s.v = s.o = nullptr;
    s.tensor_cap = 0;
    if (cudaMalloc(&s.q, tensor_bytes) != cudaSuccess || cudaMalloc(&s.k, tensor_bytes) != cudaSuccess ||
        cudaMalloc(&s.v, tensor_bytes) != cudaSuccess || cudaMalloc(&s.o, tensor_bytes) != cudaSuccess) {
      cudaGetLastError();
      return FMHA_I8_ERR_LAUNCH;
    }
    s.tensor_cap = tensor_bytes;
  }
  if (s.mask_cap < mask_bytes) {
    cudaFree(s.mask);
    s.mask = nullptr;
    s.mask_cap = 0;
    if (cudaMalloc(&s.mask, mask_bytes) != cudaSuccess) { cudaGetLastError(); return FMHA_I8_ERR_LAUNCH; }
    s.mask_cap = mask_bytes;
  }
  // Pipeline over contiguous ranges of heads: while chunk i is computed, chunk i+1 is on its way in and
  // chunk i-1 on its way out (the bus is full duplex).  Each chunk is one forward launch on a sub-slice.
  int bounds[kHostChunks + 1];
  const int n_chunks = cut_heads(desc, bh_count, bounds);
  const FetchPlan plan = plan_fetch(desc, host_q, host_k, host_v, static_cast<const int8_t*>(host_mask), bh_begin, bh_count, n_chunks);
  const int busy_sms = plan.by_kernel ? kFetchCtas : 0;
  cudaError_t e = cudaMemcpyAsync(s.mask, host_mask, mask_bytes, cudaMemcpyHostToDevice, s.s_in);
  for (int i = 0; i < n_chunks && e == cudaSuccess; ++i) {
    const int begin = bounds[i];
    const int end = bounds[i + 1];
    const size_t off = begin * head_bytes, bytes = (end - begin) * head_bytes;
    char* dq = static_cast<char*>(s.q) + off;
    char* dk = static_cast<char*>(s.k) + off;
    char* dv = static_cast<char*>(s.v) + off;
    char* dout = static_cast<char*>(s.o) + off;
    if (plan.by_kernel) {
      auto* fetch = desc[3] == 128 ? fetch_heads_kernel<128> : fetch_heads_kernel<64>;
      fetch<<<kFetchCtas, kFetchThreads, 0, s.s_in>>>(static_cast<const uint4*>(plan.q), static_cast<const uint4*>(plan.k), static_cast<const uint4*>(plan.v),
                                                      static_cast<uint4*>(s.q), static_cast<uint4*>(s.k), static_cast<uint4*>(s.v),
                                                      static_cast<const int8_t*>(s.mask), desc[1], desc[2], bh_begin, begin, end);
      g_launch_count.fetch_add(1, std::memory_order_relaxed);
      e = cudaGetLastError();
    } else {
      e = cudaMemcpyAsync(dq, static_cast<const char*>(host_q) + off, bytes, cudaMemcpyHostToDevice, s.s_in);
      if (e == cudaSuccess) e = cudaMemcpyAsync(dk, static_cast<const char*>(host_k) + off, bytes, cudaMemcpyHostToDevice, s.s_in);
      if (e == cudaSuccess) e = cudaMemcpyAsync(dv, static_cast<const char*>(host_v) + off, bytes, cudaMemcpyHostToDevice, s.s_in);
    }
    if (e == cudaSuccess) e = cudaEventRecord(s.landed[i], s.s_in);
    if (e == cudaSuccess) e = cudaStreamWaitEvent(s.s_run, s.landed[i], 0);
    if (e != cudaSuccess) break;
    st = infer_slice_impl(s.s_run, amax, desc, dq, dk, dv, s.mask, dout, bh_begin + begin, end - begin, flags, busy_sms);
    if (st != FMHA_I8_OK) break;
    e = cudaEventRecord(s.computed[i], s.s_run);
    if (e == cudaSuccess) e = cudaStreamWaitEvent(s.s_out, s.computed[i], 0);
    if (e == cudaSuccess) e = cudaMemcpyAsync(static_cast<char*>(host_o) + off, dout, bytes, cudaMemcpyDeviceToHost, s.s_out);
  }
  // drain all three streams whatever happened, so the staging buffers are idle when the lock is released
  const cudaError_t e1 = cudaStreamSynchronize(s.s_in), e2 = cudaStreamSynchronize(s.s_run), e3 = cudaStreamSynchronize(s.s_out);
  if (st != FMHA_I8_OK) return st;
  if (e != cudaSuccess || e1 != cudaSuccess || e2 != cudaSuccess || e3 != cudaSuccess) { cudaGetLastError(); return FMHA_I8_ERR_LAUNCH; }
  return FMHA_I8_OK;
}

int fmha_i8_sm100_infer_host(const float amax[5], const int desc[4], const void* host_q, const void* host_k,
                             const void* host_v, const void* host_mask, void* host_o, unsigned flags) {
  if (!desc) return finish(FMHA_I8_ERR_NULL_POINTER);
  const long long BH = static_cast<long long>(desc[0]) * desc[2];
  if (BH < 1 || BH > 0x7FFFFFFFLL) return finish(FMHA_I8_ERR_BAD_SHAPE);
  return finish(infer_host_slice_impl(amax, desc, host_q, host_k, host_v, host_mask, host_o, 0, static_cast<int>(BH), flags));
}

int fmha_i8_sm100_infer_host_slice(const float amax[5], const int desc[4], const void* host_q, const void* host_k,
                                   const void* host_v, const void* host_mask, void* host_o, int bh_begin, int bh_count,
                                   unsigned flags) {
  return finish(infer_host_slice_impl(amax, desc, host_q, host_k, host_v, host_mask, host_o, bh_begin, bh_count, flags));
}

int fmha_i8_sm100_debug_plan(const int desc5[5], int policy, int plan[3]) {
  if (!desc5 || !plan) return finish(FMHA_I8_ERR_NULL_POINTER);
  const Shape sh{desc5[0], desc5[1], desc5[2], desc5[3], desc5[4]};
  int st = check_shape_x(sh);
  if (st != FMHA_I8_OK) return finish(st);
  if (policy < FMHA_I8_POLICY_TILE || policy > FMHA_I8_PLAN_CALIBRATION) return finish(FMHA_I8_ERR_BAD_FLAGS);
  const bool calibration = policy == FMHA_I8_PLAN_CALIBRATION;
  int err = FMHA_I8_OK;
  DeviceInfo* dev = current_device(&err);
  if (!dev) return finish(err);
  if ((st = set_kernel_attributes(dev)) != FMHA_I8_OK) return finish(st);
  FwdParams p{};
  if ((st = fill_units(&p, sh, sh.B * sh.H)) != FMHA_I8_OK) return finish(st);
  plan[0] = plan_call(&p, sh.D, calibration ? FMHA_I8_POLICY_TILE : policy, !calibration, 0, dev);
  plan[1] = p.parts;
  plan[2] = p.parts > 1 ? p.own_rounds : 0;
  return finish(FMHA_I8_OK);
}

int fmha_i8_sm100_debug_host_fetch(const int desc[4], const void* host_q, const void* host_k, const void* host_v, const void* host_mask) {
  if (!desc || !host_q || !host_k || !host_v || !host_mask) return finish(FMHA_I8_ERR_NULL_POINTER);
  const int st = check_shape(desc);
  if (st != FMHA_I8_OK) return finish(st);
  const long long BH = static_cast<long long>(desc[0]) * desc[2];
  if (BH > 0x7FFFFFFFLL) return finish(FMHA_I8_ERR_BAD_SHAPE);
  int bounds[kHostChunks + 1];
  const int n_chunks = cut_heads(desc, static_cast<int>(BH), bounds);
  finish(FMHA_I8_OK);
  return plan_fetch(desc, host_q, host_k, host_v, static_cast<const int8_t*>(host_mask), 0, static_cast<int>(BH), n_chunks).by_kernel ? 1 : 0;
}

int fmha_i8_sm100_debug_qk(void* stream, const int desc[4], const void* q, const void* k, int32_t* s_out) {
  if (!desc || !q || !k || !s_out) return finish(FMHA_I8_ERR_NULL_POINTER);
  int st = check_shape(desc);
  if (st != FMHA_I8_OK) return finish(st);
  if (!aligned(q, 16) || !aligned(k, 16) || !aligned(s_out, 4)) return finish(FMHA_I8_ERR_MISALIGNED);
  int err = FMHA_I8_OK;
  DeviceInfo* dev = current_device(&err);
  if (!dev) return finish(err);
  if ((st = set_kernel_attributes(dev)) != FMHA_I8_OK) return finish(st);
  const int BH = desc[0] * desc[2], S = desc[1], D = desc[3];
  if (BH > 65535) return finish(FMHA_I8_ERR_TOO_LARGE);
  CUtensorMap mq, mk;
  if ((st = make_map(&mq, q, BH, S, D)) != FMHA_I8_OK) return finish(st);
  if ((st = make_map(&mk, k, BH, S, D)) != FMHA_I8_OK) return finish(st);
  const int nt = (S + kTile - 1) / kTile;
  const dim3 grid(nt, nt, BH);
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  if (D == 128) debug_qk_kernel<128><<<grid, 128, qk_smem_bytes<128>(), s>>>(mq, mk, s_out, S, dev->status);
  else debug_qk_kernel<64><<<grid, 128, qk_smem_bytes<64>(), s>>>(mq, mk, s_out, S, dev->status);
  g_launch_count.fetch_add(1, std::memory_order_relaxed);
  return finish(cudaGetLastError() == cudaSuccess ? FMHA_I8_OK : FMHA_I8_ERR_LAUNCH);
}

int fmha_i8_sm100_debug_pv(void* stream, const int desc[4], const void* p, const void* v, int32_t* o_out,
                           unsigned variant) {
  if (!desc || !p || !v || !o_out) return finish(FMHA_I8_ERR_NULL_POINTER);
  int st = check_shape(desc);
  if (st != FMHA_I8_OK) return finish(st);
  if (!aligned(p, 16) || !aligned(v, 16) || !aligned(o_out, 4)) return finish(FMHA_I8_ERR_MISALIGNED);
  if (variant > 1) return finish(FMHA_I8_ERR_BAD_SHAPE);
  int err = FMHA_I8_OK;
  DeviceInfo* dev = current_device(&err);
  if (!dev) return finish(err);
  if ((st = set_kernel_attributes(dev)) != FMHA_I8_OK) return finish(st);
  const int BH = desc[0] * desc[2], S = desc[1], D = desc[3];
  if (BH > 65535) return finish(FMHA_I8_ERR_TOO_LARGE);
  CUtensorMap mv;
  if ((st = make_map(&mv, v, BH, S, D)) != FMHA_I8_OK) return finish(st);
  const dim3 grid((S + kTile - 1) / kTile, BH);
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const int8_t* p8 = static_cast<const int8_t*>(p);
  if (D == 128) {
    if (variant == 0) debug_pv_kernel<128, true><<<grid, 128, pv_smem_bytes<128>(), s>>>(mv, p8, o_out, S, dev->status);
    else debug_pv_kernel<128, false><<<grid, 128, pv_smem_bytes<128>(), s>>>(mv, p8, o_out, S, dev->status);
  } else {
    if (variant == 0) debug_pv_kernel<64, true><<<grid, 128, pv_smem_bytes<64>(), s>>>(mv, p8, o_out, S, dev->status);
    else debug_pv_kernel<64, false><<<grid, 128, pv_smem_bytes<64>(), s>>>(mv, p8, o_out, S, dev->status);
  }
  g_launch_count.fetch_add(1, std::memory_order_relaxed);
  return finish(cudaGetLastError() == cudaSuccess ? FMHA_I8_OK : FMHA_I8_ERR_LAUNCH);
}

int fmha_i8_sm100_debug_simt_x(void* stream, const float amax[5], const int desc5[5], const void* q, const void* k,
                               const void* v, const void* mask, void* o, unsigned flags) {
  if (!amax || !desc5 || !q || !k || !v || !mask || !o) return finish(FMHA_I8_ERR_NULL_POINTER);
  const Shape sh{desc5[0], desc5[1], desc5[2], desc5[3], desc5[4]};
  int st = check_shape_x(sh);
  if (st != FMHA_I8_OK) return finish(st);
  if (!aligned(q, 16) || !aligned(k, 16) || !aligned(v, 16) || !aligned(o, 16)) return finish(FMHA_I8_ERR_MISALIGNED);
  FwdParams p{};
  if ((st = fill_params(&p, amax, sh.D, flags)) != FMHA_I8_OK) return finish(st);
  int err = FMHA_I8_OK;
  if (!current_device(&err)) return finish(err);
  const long long BH = static_cast<long long>(sh.B) * sh.H;
  if (BH > 65535) return finish(FMHA_I8_ERR_TOO_LARGE);
  const dim3 grid((sh.Sq + kTile - 1) / kTile, static_cast<unsigned>(BH));
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const int8_t* q8 = static_cast<const int8_t*>(q);
  const int8_t* k8 = static_cast<const int8_t*>(k);
  const int8_t* v8 = static_cast<const int8_t*>(v);
  const int8_t* m8 = static_cast<const int8_t*>(mask);
  int8_t* o8 = static_cast<int8_t*>(o);
  if (sh.D == 128)
    simt_check_kernel<128><<<grid, 128, 0, s>>>(q8, k8, v8, m8, o8, sh.Sq, sh.Sk, sh.H, 0, p.row_scale, p.scale_qk, p.scale_v_out, p.p_mul);
  else
    simt_check_kernel<64><<<grid, 128, 0, s>>>(q8, k8, v8, m8, o8, sh.Sq, sh.Sk, sh.H, 0, p.row_scale, p.scale_qk, p.scale_v_out, p.p_mul);
  g_launch_count.fetch_add(1, std::memory_order_relaxed);
  return finish(cudaGetLastError() == cudaSuccess ? FMHA_I8_OK : FMHA_I8_ERR_LAUNCH);
}

int fmha_i8_sm100_debug_simt(void* stream, const float amax[5], const int desc[4], const void* q, const void* k,
                             const void* v, const void* mask, void* o) {
  if (!desc) return finish(FMHA_I8_ERR_NULL_POINTER);
  const int desc5[5] = {desc[0], desc[1], desc[1], desc[2], desc[3]};
  return fmha_i8_sm100_debug_simt_x(stream, amax, desc5, q, k, v, mask, o, 0u);
}

int fmha_i8_sm100_debug_wait_probe(void* stream, long long limit_cycles) {
  if (limit_cycles < 1000 || limit_cycles > kWaitLimitCycles) return finish(FMHA_I8_ERR_TOO_LARGE);
  int err = FMHA_I8_OK;
  DeviceInfo* dev = current_device(&err);
  if (!dev) return finish(err);
  wait_probe_kernel<<<1, 32, 0, static_cast<cudaStream_t>(stream)>>>(dev->status, limit_cycles);
  g_launch_count.fetch_add(1, std::memory_order_relaxed);
  return finish(cudaGetLastError() == cudaSuccess ? FMHA_I8_OK : FMHA_I8_ERR_LAUNCH);
}

int fmha_i8_sm100_debug_wait_loops(void* stream, long long limit_cycles, unsigned* out20) {
  if (!out20) return finish(FMHA_I8_ERR_NULL_POINTER);
  if (limit_cycles < 1000 || limit_cycles > kWaitLimitCycles) return finish(FMHA_I8_ERR_TOO_LARGE);
  if (!aligned(out20, 4)) return finish(FMHA_I8_ERR_MISALIGNED);
  int err = FMHA_I8_OK;
  if (!current_device(&err)) return finish(err);
  wait_loops_kernel<<<1, 64, 0, static_cast<cudaStream_t>(stream)>>>(out20, limit_cycles);
  g_launch_count.fetch_add(1, std::memory_order_relaxed);
  return finish(cudaGetLastError() == cudaSuccess ? FMHA_I8_OK : FMHA_I8_ERR_LAUNCH);
}

int fmha_i8_sm100_quantize_f32(void* stream, const float* x, long long n, int8_t* out, float* amax_out) {
  const int st = check_quant_args(x, n, out);
  return finish(st != FMHA_I8_OK ? st : quantize_impl(stream, x, n, out, amax_out));
}

int fmha_i8_sm100_quantize_f32_noalloc(void* stream, const float* x, long long n, int8_t* out, float* amax_out) {
  const int st = check_quant_args(x, n, out);
  if (st != FMHA_I8_OK) return finish(st);
  if (n > kNoAllocMaxElements) {
    std::fprintf(stderr, "fmha_i8_sm100_quantize_f32_noalloc: %lld elements exceed the limit of this entry point (at most %lld)\n", n,
                 kNoAllocMaxElements);
    return finish(FMHA_I8_ERR_TOO_LARGE);
  }
  return finish(quantize_impl(stream, x, n, out, amax_out));
}

int fmha_i8_sm100_debug_quantize_whole_chip(void* stream, const float* x, long long n, int8_t* out, float* amax_out) {
  const int st = check_quant_args(x, n, out);
  if (st != FMHA_I8_OK) return finish(st);
  if (n <= kQuantClusterPortable * kQuantPerCta) return finish(FMHA_I8_ERR_BAD_SHAPE);
  return finish(quantize_impl(stream, x, n, out, amax_out, true));
}

int fmha_i8_sm100_device_status(unsigned words[8]) {
  if (!words) return finish(FMHA_I8_ERR_NULL_POINTER);
  if (cudaDeviceSynchronize() != cudaSuccess) { return finish(FMHA_I8_ERR_LAUNCH); }
  if (cudaMemcpyFromSymbol(words, g_status_words, sizeof(unsigned) * 8) != cudaSuccess) return finish(FMHA_I8_ERR_LAUNCH);
  const unsigned zeros[8] = {0, 0, 0, 0, 0, 0, 0, 0};
  if (cudaMemcpyToSymbol(g_status_words, zeros, sizeof zeros) != cudaSuccess) return finish(FMHA_I8_ERR_LAUNCH);
  {
    int dev_id = 0;
    if (cudaGetDevice(&dev_id) == cudaSuccess && dev_id >= 0 && dev_id < kMaxDevices) {
      std::lock_guard<std::mutex> lock(g_dev_mutex);
      if (g_dev[dev_id].host_flag) *g_dev[dev_id].host_flag = 0u;
    }
  }
  return finish(words[0] == 0u ? FMHA_I8_OK : FMHA_I8_ERR_DEVICE);
}

int fmha_i8_sm100_last_status(void) { return t_last_status; }

const char* fmha_i8_sm100_status_string(int status) {
  switch (status) {
    case FMHA_I8_OK: return "ok";
    case FMHA_I8_ERR_NULL_POINTER: return "a required pointer is NULL";
    case FMHA_I8_ERR_BAD_SHAPE: return "unsupported shape (head_dim must be 64 or 128, seq_len a multiple of 64 up to 32768)";
    case FMHA_I8_ERR_MISALIGNED: return "q/k/v/o must be 16-byte aligned and the mask 4-byte aligned";
    case FMHA_I8_ERR_NO_CUDA_CORE_PATH: return "use_tcu == false is not supported (the reference's CUDA-core kernel is an empty stub)";
    case FMHA_I8_ERR_WRONG_ARCH: return "the current device is not compute capability 10.0 (B200)";
    case FMHA_I8_ERR_LAUNCH: return "the CUDA runtime reported an error";
    case FMHA_I8_ERR_DRIVER: return "tensor-map encoding failed";
    case FMHA_I8_ERR_BAD_SLICE: return "bh_begin/bh_count outside the batch*head range";
    case FMHA_I8_ERR_BAD_AMAX: return "amax values must be finite and positive";
    case FMHA_I8_ERR_TOO_LARGE: return "size beyond the maximum of this entry point";
    case FMHA_I8_ERR_DEVICE: return "a device-side bounded wait ran out (see fmha_i8_sm100_device_status)";
    case FMHA_I8_ERR_BAD_FLAGS: return "an undefined flag bit is set";
    default: return "unknown status";
  }
}

unsigned long long fmha_i8_sm100_launch_count(void) { return g_launch_count.load(std::memory_order_relaxed); }

int fmha_i8_sm100_version(void) { return 100; }

#ifdef FMHA_TRACE
// Performance-work builds only: copies out the timeline stamps of the first CTA.
int fmha_i8_sm100_read_trace(long long* out) {
  if (cudaDeviceSynchronize() != cudaSuccess) return FMHA_I8_ERR_LAUNCH;
  return cudaMemcpyFromSymbol(out, fmha::g_trace, sizeof(long long) * 48 * 512) == cudaSuccess ? FMHA_I8_OK : FMHA_I8_ERR_LAUNCH;
}
#endif

}  // extern "C"

// The reference project's C++ entry point (inc/fmha_i8.h:5-17), kept symbol-for-symbol.
#include "../../include/fmha_i8.h"
namespace gpuImpl {
void FMHAInferI8(cudaStream_t stream, FMHAParamI8 fmha_param, AttnDataDescriptor attn_desc, const void* q,
                 const void* k, const void* v, const void* padding_mask, void* o, const bool use_tcu) {
  const float amax[5] = {fmha_param.q_amax, fmha_param.k_amax, fmha_param.v_amax, fmha_param.o_amax, fmha_param.s_max};
  const int desc[4] = {attn_desc.batch_num, attn_desc.seq_len, attn_desc.head_num, attn_desc.head_dim};
  const int st = fmha_i8_sm100_infer(stream, amax, desc, q, k, v, padding_mask, o, use_tcu ? FMHA_I8_FLAG_USE_TCU : 0u);
  if (st != FMHA_I8_OK) std::fprintf(stderr, "gpuImpl::FMHAInferI8: %s (status %d)\n", fmha_i8_sm100_status_string(st), st);
}
}  // namespace gpuImpl
