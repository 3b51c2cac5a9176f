// Index arithmetic of the tensor-core kernels over packed weights that host code can run as well.
#pragma once

#ifdef __CUDACC__
#define RB200_HD __host__ __device__ __forceinline__
#else
#define RB200_HD inline
#endif

namespace rb200 {
namespace us {

// First of the two adjacent 64-k blocks whose group-32 scales one 8-byte load takes.  A decode group asks for
// its blocks of every chunk of four, and the last chunk may hold two only: kb == k_blocks there, and the
// scales belong to no block, so the row's last pair stands in (past it lies the next row, or nothing).
// kb and k_blocks are even.
RB200_HD int pair_in_row(int kb, int k_blocks) { return kb < k_blocks - 2 ? kb : k_blocks - 2; }

}  // namespace us
}  // namespace rb200
