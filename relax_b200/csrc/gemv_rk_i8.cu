#include "gemv_rk.cuh"
namespace rb200 {
namespace rk {
int launch_i8(const Params& pp, int zmode, int src, int warps, int grid, cudaStream_t stream) {
  return launch_bits<8>(pp, zmode, src, warps, grid, stream);
}
}  // namespace rk
}  // namespace rb200
