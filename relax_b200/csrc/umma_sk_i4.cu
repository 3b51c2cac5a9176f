#include "umma_sk.cuh"
namespace rb200 {
namespace us {
int launch_i4(const Params& pp, const Launch& l, const CUtensorMap& tx, cudaStream_t stream) {
  return launch_bits<4>(pp, l, tx, stream);
}
}  // namespace us
}  // namespace rb200
