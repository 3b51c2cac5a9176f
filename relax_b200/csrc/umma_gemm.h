// Host entry of the dense expert kernel (umma_gemm.cu).
#pragma once

#include "gemv.h"

namespace rb200 {

// Dense fp16 experts [E, N, K].  p.m = total rows of x / out; indptr = device int64[num_experts] of end
// offsets.  0 on launch, -1 on error (shapes outside the kernel's coverage are errors).
int umma_group_gemm_run(const GemvParams& p, int sm_count, const int64_t* indptr, int indptr_has_prev, int num_experts,
                        int64_t w_expert_bytes, cudaStream_t stream);

}  // namespace rb200
