// Thread-block clusters on sm_100a: CTAs that run at the same time, reach each other's shared memory and meet at
// barriers of their own.  An input of a few tiles is one cluster's: the tiles' totals travel by stores into shared memory, so
// there are no descriptors, no ticket and nothing that has to be cleared beforehand, and no wait that could run out.
#pragma once
#include "common.cuh"

namespace tb200 {

// Launches `kernel` as one cluster of `ctas` CTAs if the device can hold it and takes the launch (launched = true).
// `largest`: the caller's note for this kernel, one per device, of the largest cluster that fits (0: not looked up yet).
template <class... Params, class... Args>
cudaError_t cluster_launch(void (*kernel)(Params...), unsigned ctas, int block, size_t smem, cudaStream_t stream, unsigned (&largest)[64], bool& launched, Args... args) {
  launched = false;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(ctas);
  cfg.blockDim = dim3(block);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = ctas; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64 || smem > (size_t)current_device_info().max_smem_optin) return cudaSuccess;
  if (largest[dev] == 0) {
    unsigned most = 1;
    if ((smem > 48 * 1024 && cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess) ||
        cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess) { cudaGetLastError(); return cudaSuccess; }
    for (unsigned c = CLUSTER_MAX_CTAS; c > 1; c >>= 1) {
      cudaLaunchConfig_t probe = cfg;
      cudaLaunchAttribute pa[1];
      pa[0].id = cudaLaunchAttributeClusterDimension;
      pa[0].val.clusterDim.x = c; pa[0].val.clusterDim.y = 1; pa[0].val.clusterDim.z = 1;
      probe.gridDim = dim3(c);
      probe.attrs = pa;
      int clusters = 0;
      if (cudaOccupancyMaxActiveClusters(&clusters, kernel, &probe) == cudaSuccess && clusters > 0) { most = c; break; }
      cudaGetLastError();
    }
    largest[dev] = most;
  }
  if (ctas > largest[dev]) return cudaSuccess;
  const cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, static_cast<Params>(args)...);
  if (launch_refused(e)) return cudaSuccess;
  launched = true;
  return e;
}

// CTAs for `tiles` tiles: a power of two, so that every GPC has room for it in one piece.  0: too many for a cluster.
inline unsigned cluster_ctas(size_t tiles) {
  unsigned ctas = 1;
  while (ctas < tiles && ctas <= (unsigned)CLUSTER_MAX_CTAS) ctas <<= 1;
  return ctas <= (unsigned)CLUSTER_MAX_CTAS ? ctas : 0;
}

}  // namespace tb200
