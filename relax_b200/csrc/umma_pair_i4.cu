#include "umma_pair.cuh"
namespace rb200 {
namespace up {
int launch_i4(const Params& pp, const Launch& l, const CUtensorMap& tx, cudaStream_t stream) {
  return launch_bits<4>(pp, l, tx, stream);
}
}  // namespace up
}  // namespace rb200
