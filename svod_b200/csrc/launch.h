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
#pragma once

#include <cuda_runtime.h>

#include <utility>

namespace svodb {

template <typename... K, typename... A>
cudaError_t launch_pdl(void (*kernel)(K...), dim3 grid, dim3 block, size_t smem, cudaStream_t s, unsigned cluster,
                       A&&... args) {
  cudaLaunchConfig_t lc{};
  lc.gridDim = grid;
  lc.blockDim = block;
  lc.dynamicSmemBytes = smem;
  lc.stream = s;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  lc.numAttrs = 1;
  if (cluster > 1) {
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = cluster;
    attr[1].val.clusterDim.y = 1;
    attr[1].val.clusterDim.z = 1;
    lc.numAttrs = 2;
  }
  lc.attrs = attr;
  return cudaLaunchKernelEx(&lc, kernel, static_cast<K>(args)...);
}

}  // namespace svodb
