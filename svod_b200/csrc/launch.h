// Kernel launches with the two attributes this library uses: a cluster of CTAs and
// programmatic dependent launch.
//
// Every kernel launched here calls `pdl_wait` (common.cuh) before it first reads what an
// earlier launch wrote or writes what one may still read, and `pdl_trigger` as soon as
// all of its CTAs can be resident with what they need. The next kernel of the stream then
// comes up — barriers, tensor memory, descriptor fetches, constant weights — while this
// one still runs, which is worth 2-4 us of each of the ~170 launches of a small batch.
// A kernel launched without the attribute (or after one that never triggers) waits for
// the whole of its predecessor as ever, and `pdl_wait` then returns at once.
//
// Kernels over more than kEarlyRows rows are launched without it. What a launch saves is a
// few us whatever its size; what it costs grows with the kernel it comes up beside, whose
// issue slots and power its waiting warps share. Whole stacks, ms with and without it:
// XLM-R 1024 rows 2.02 | 2.06, 4096 rows 3.66 | 3.65, 8192 rows 6.35 | 6.29, 32768 rows
// 22.9 | 22.6; Qwen3 2048 rows 2.99 | 3.03, 8192 rows 9.29 | 9.16, 131072 rows 160.1 | 158.6;
// ModernBERT 2048 rows 1.54 | 1.58, 16384 rows 6.20 | 6.17, 65536 rows 27.5 | 27.2.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include <utility>

namespace svodb {

constexpr int64_t kEarlyRows = 4096;

// `rows`: the rows of activations the launch walks.
template <typename... K, typename... A>
cudaError_t launch_pdl(void (*kernel)(K...), dim3 grid, dim3 block, size_t smem, cudaStream_t s, unsigned cluster,
                       int64_t rows, A&&... args) {
  cudaLaunchConfig_t lc{};
  lc.gridDim = grid;
  lc.blockDim = block;
  lc.dynamicSmemBytes = smem;
  lc.stream = s;
  cudaLaunchAttribute attr[2];
  lc.numAttrs = 0;
  if (rows <= kEarlyRows) {
    cudaLaunchAttribute& early = attr[lc.numAttrs++];
    early.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    early.val.programmaticStreamSerializationAllowed = 1;
  }
  if (cluster > 1) {
    cudaLaunchAttribute& size = attr[lc.numAttrs++];
    size.id = cudaLaunchAttributeClusterDimension;
    size.val.clusterDim.x = cluster;
    size.val.clusterDim.y = 1;
    size.val.clusterDim.z = 1;
  }
  lc.attrs = attr;
  return cudaLaunchKernelEx(&lc, kernel, static_cast<K>(args)...);
}

}  // namespace svodb
