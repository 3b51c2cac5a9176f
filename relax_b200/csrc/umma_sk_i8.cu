#include "umma_sk.cuh"
namespace rb200 {
namespace us {
int launch_i8(const Params& pp, const Launch& l, const CUtensorMap& tx, cudaStream_t stream) {
  return launch_bits<8>(pp, l, tx, stream);
}
}  // namespace us
}  // namespace rb200
