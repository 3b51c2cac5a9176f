// Index arithmetic of the tensor-core kernels over packed weights that host code can run as well.
#pragma once

#ifdef __CUDACC__
#define RB200_HD __host__ __device__ __forceinline__
#else
#define RB200_HD inline
#endif

namespace rb200 {
namespace us {

// Whether the group-32 scales of two adjacent 64-k blocks may be one 8-byte load: every chunk (256 k of int4, 128
// of int8) is whole.  A decode group asks for its pair of every chunk, also of a last one that holds no such
// pair, where the load would take the next row's scales and, behind the last row, what lies past the tensor.
// (Clamped to the row instead, the load cost k 4096 x n 22016, 32 rows, 21.3 -> 21.6 us.)
RB200_HD bool pairs_fit_rows(int k, int bits) { return k % (bits == 4 ? 256 : 128) == 0; }

}  // namespace us
}  // namespace rb200
