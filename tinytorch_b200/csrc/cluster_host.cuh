// How many CTAs of a cluster size a device holds.
#pragma once
#include <atomic>

#include "common.cuh"
#include "tma_host.cuh"

namespace ttattn {

// CTAs of clusters of this size that can be resident at once, one to an SM: a cluster lives inside one GPC, and GPCs differ in size, from
// one chip to the next too (on those measured 15 clusters of 8, not 16, and 33 of 4).  Asked once per device; 0 where it is not known.
static __global__ void room_kernel() {}
inline int cluster_room(int device, int cluster) {
  static std::atomic<int> known[64][8];
  if (device < 0 || device >= 64 || cluster < 1 || cluster > 8) return 0;
  if (cluster == 1) return sm_count(device);
  std::atomic<int>& k = known[device][cluster - 1];
  int n = k.load(std::memory_order_relaxed);
  if (n == 0) {
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = cluster, attr[0].val.clusterDim.y = 1, attr[0].val.clusterDim.z = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(sm_count(device) / cluster * cluster);
    cfg.blockDim = dim3(128);
    cfg.dynamicSmemBytes = 120 * 1024;  // (no second one beside it)
    cfg.attrs = attr, cfg.numAttrs = 1;
    int clusters = 0;
    if (cudaFuncSetAttribute(room_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024) != cudaSuccess ||
        cudaOccupancyMaxActiveClusters(&clusters, room_kernel, &cfg) != cudaSuccess) {
      cudaGetLastError();
      clusters = 0;
    }
    n = clusters > 0 ? clusters * cluster : -1;
    k.store(n, std::memory_order_relaxed);
  }
  return n;
}

}  // namespace ttattn
