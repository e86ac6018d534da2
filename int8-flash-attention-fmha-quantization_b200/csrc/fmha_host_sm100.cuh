// Fetches the inputs of a range of heads from pinned host memory (fmha_i8_sm100_infer_host): rows of keys and values that the
// padding mask excludes stay where they are -- nothing reads their staging rows but the scores and products that the mask and a
// zero probability throw away.
//
// Bound by the PCIe link: eight CTAs of 16 warps, a warp with 32 rows (2 or 4 KB) in flight, reach the 50.7 GB/s that any number
// of SMs reaches, and keep more of it than larger grids while the output goes the other way (34 GB/s each way; 148 CTAs: 29),
// so the forward kernels keep the other SMs.
#pragma once
#include <cuda_runtime.h>
#include <cstdint>

namespace fmha {

constexpr int kFetchCtas = 8, kFetchThreads = 512, kFetchRows = 32;

template <int D>
__global__ void __launch_bounds__(kFetchThreads, 1)
fetch_heads_kernel(const uint4* __restrict__ host_q, const uint4* __restrict__ host_k, const uint4* __restrict__ host_v, uint4* __restrict__ q,
                   uint4* __restrict__ k, uint4* __restrict__ v, const int8_t* __restrict__ mask, int S, int H, int bh_begin, int head_begin, int head_end) {
  constexpr int kVec = kFetchRows * D / 16 / 32;        // 16-byte words per lane
  const int lane = threadIdx.x & 31;
  const int groups = S / kFetchRows;                     // S is a multiple of 64
  const long long items = static_cast<long long>(head_end - head_begin) * groups * 3;
  const int step = static_cast<int>(gridDim.x) * (kFetchThreads / 32);
  for (long long i = blockIdx.x * (kFetchThreads / 32) + (threadIdx.x >> 5); i < items; i += step) {
    const int head = head_begin + static_cast<int>(i / (3 * groups)), rest = static_cast<int>(i % (3 * groups));
    const int tensor = rest / groups, group = rest % groups;
    if (tensor != 0) {
      const int batch = (bh_begin + head) / H;
      if (!__any_sync(0xFFFFFFFFu, __ldg(mask + static_cast<int64_t>(batch) * S + group * kFetchRows + lane) == 0)) continue;
    }
    const uint4* src = tensor == 0 ? host_q : tensor == 1 ? host_k : host_v;
    uint4* dst = tensor == 0 ? q : tensor == 1 ? k : v;
    const int64_t at = (static_cast<int64_t>(head) * groups + group) * (kVec * 32) + lane;
    uint4 r[kVec];
#pragma unroll
    for (int w = 0; w < kVec; ++w) r[w] = src[at + w * 32];
#pragma unroll
    for (int w = 0; w < kVec; ++w) dst[at + w * 32] = r[w];
  }
}

}  // namespace fmha
