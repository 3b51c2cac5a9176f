#include "umma_sk.cuh"
namespace rb200 {
namespace us {
int launch_i4(const Params& pp, const Launch& l, const CUtensorMap& tx, cudaStream_t stream) {
  return launch_bits<4>(pp, l, tx, stream);
}
// Asked of a kernel of the same block and shared memory but without tensor memory, and never launched: of kernels that allocate
// tensor memory the query sees one CTA per SM whatever they take.  (Registers allow two by the launch bounds; shared memory decides.)
__global__ void __launch_bounds__((4 + 4 * kGroups) * 32, 2) places_kernel() {}
int cluster_places(int ranges) {
  static thread_local int device = -1, places[9];
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return 0;
  if (dev != device) {
    device = dev;
    for (int& p : places) p = -1;
  }
  if (places[ranges] < 0) {
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = (unsigned)ranges;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)ranges, 1, 1);
    cfg.blockDim = dim3((4 + 4 * kGroups) * 32, 1, 1);
    cfg.dynamicSmemBytes = kCtaSmem;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    int n = 0;
    if (cudaFuncSetAttribute(places_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kCtaSmem) != cudaSuccess ||
        cudaOccupancyMaxActiveClusters(&n, places_kernel, &cfg) != cudaSuccess) {
      cudaGetLastError();  // no clusters then
      n = 0;
    }
    places[ranges] = n;
  }
  return places[ranges];
}
}  // namespace us
}  // namespace rb200
