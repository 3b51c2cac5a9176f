// Host side of the int4 kernel of one sequence of units per warp: which calls it takes, launch.
#include "gemv_flat.cuh"

namespace rb200 {
namespace fl {

int source(const rk::Params& pp, int bits, int zmode, int src) {
  const GemvParams& p = pp.g;
  const bool z = zmode == kZeroGeneral, tail = p.k % 256 != 0, experts = pp.indptr != nullptr;
  if (bits != 4 || (z && !p.z)) return -1;
  const uintptr_t addr = reinterpret_cast<uintptr_t>(p.s) | reinterpret_cast<uintptr_t>(p.z) | (uintptr_t)(pp.s_expert_stride * 2);
  const int64_t weights = (int64_t)p.n * p.k;
  const bool few = p.m <= 4 || experts;  // (an expert's rows are seldom more)
  const bool two = p.m > 8 && !experts;  // m-tiles
  // Groups of 32.  Five to eight rows, where two row blocks cannot share a load of x: eight rows with zero points k 4096 x
  // n 22016 21.3 / 16.9 us (here), k 11008 x n 4096 12.1 / 10.0, k = n = 4096 5.43 / 5.48, k 2048 x n 4096 3.53 / 4.17; without
  // k 5504 x n 4096 8.6 / 6.5 and 1152 x 1040 3.33 / 2.88, but whole chunks k = n = 4096 4.66 / 5.24, n 22016 15.5 / 15.6.
  if (p.group == 32 && p.s_g == 1 && p.s_n % 2 == 0 && (addr & 3u) == 0 && (tail || src == rk::kRow32)) {
    // Sixteen rows: k 5504 x n 4096 10.6 / 8.9, but whole chunks k 4096 x n 22016 20.2 / 22.2, with zero points k = n = 4096
    // 6.21 / 6.62.
    if (p.m <= 4 && !experts) return rk::kRow32;
    return tail || experts || (z && weights >= (16ll << 20) && !two) ? kRow32Wide : -1;
  }
  if (src == rk::kGeneral || src == rk::kRow32) return -1;
  if (!tail && p.s_g == 1 && p.group == 64 && p.s_n % 4 == 0 && (addr & 7u) == 0)
    // k 2048 x n 4096 without zero points 2.77 / 2.85 us (here), k = n = 4096 4.44 / 3.93; eight rows 3.13 / 3.5, 4.94 / 4.7
    // sixteen rows without zero points k 2048 x n 4096 4.23 / 4.07, k = n = 4096 7.0 / 5.7, k 11008 x n 4096 14.6 / 11.3, with
    // 4.39 / 4.88, 7.5 / 7.1, 16.3 / 13.6
    return experts || (two ? !z || weights >= (16ll << 20) : z || p.k >= 4096) ? kRow64 : -1;
  if (!tail && p.s_g == 1 && p.group == 128 && p.s_n % 2 == 0 && (addr & 3u) == 0)
    // eight rows: k 2048 x n 4096 with zero points 3.34 / 3.58, k = n = 4096 5.09 / 4.82, without 4.33 / 4.67
    // sixteen rows k = n = 4096 7.0 / 5.9 with them, 6.0 / 5.6 without, k 11008 x n 4096 16.7 / 11.4, 11.7 / 10.7
    return few || two || (z && p.k >= 4096) ? kRow128 : -1;
  if (src == rk::kChannel) return tail && !z && !two ? src : -1;  // whole chunks: k 8192 x n 28672 24.6 / 29
  if (src == rk::kTile && z) return -1;                   // spills 450 bytes: k 4096 x n 11008, one row 11.1 / 12.1
  if (tail) return src;
  // scales one by one, whole chunks: k = n = 4096 without zero points 3.88 / 4.06, x n 11008 7.77 / 6.88, eight rows
  // k 11008 x n 4096 8.28 / 8.59; groups of 64 with zero points k = n = 4096 5.34 / 5.81, x n 11008 11.0 / 10.4;
  // groups of 128 with zero points k = n = 4096 4.83 / 4.31, 1024 x 1024 2.49 / 2.41
  if (experts) return src;
  // sixteen rows: groups of 128 k 4096 x n 11008 11.4 / 10.4, 1024 x 1024 3.01 / 2.92, with zero points k 11008 x n 4096
  // 16.9 / 15.1, k 4096 x n 22016 25.4 / 26.9; groups of 64 k 4096 x n 11008 12.4 / 11.7, 1024 x 1024 3.01 / 3.18
  if (two) return src == rk::kHalf ? (!z || p.k >= 8192 ? src : -1) : (weights >= (4ll << 20) ? src : -1);
  if (src == rk::kHalf && z) return src;
  return few && weights >= (32ll << 20) ? src : -1;
}

template <int Z, int SRC, bool kTail>
int launch_form(const Params& pp, int grid, cudaStream_t stream) {
  const dim3 g((unsigned)grid);
  if (pp.indptr) {
    if constexpr (SRC != rk::kRow32) RB200_CUDA(launch_dependent(gemv_flat_experts_kernel<Z, SRC, kTail>, g, kWarps * 32, 0, stream, pp));
  } else {
    if (pp.g.m > 8) {
      if constexpr (SRC != rk::kRow32 && SRC != rk::kChannel) RB200_CUDA(launch_dependent(gemv_flat_kernel<Z, SRC, kTail, 2>, g, kWarps * 32, 0, stream, pp));
    } else {
      RB200_CUDA(launch_dependent(gemv_flat_kernel<Z, SRC, kTail, 1>, g, kWarps * 32, 0, stream, pp));
    }
  }
  return 0;
}
template <int Z, int SRC, bool kEither = true>
int launch_tail(const Params& pp, int grid, cudaStream_t stream) {
  if constexpr (kEither) {
    if (pp.g.k % 256) return launch_form<Z, SRC, true>(pp, grid, stream);
  }
  return launch_form<Z, SRC, false>(pp, grid, stream);
}
template <int SRC, bool kEither = true>
int launch_src(const Params& pp, int zmode, int grid, cudaStream_t stream) {
  return zmode == kZeroGeneral ? launch_tail<kZeroGeneral, SRC, kEither>(pp, grid, stream)
                               : launch_tail<kZeroConstInt, SRC, kEither>(pp, grid, stream);
}

int launch(const rk::Params& rp, int zmode, int src, int grid, cudaStream_t stream) {
  Params pp;
  static_cast<rk::Params&>(pp) = rp;
  pp.s_last = pp.g.group > 0 ? (unsigned)(pp.g.k / pp.g.group - 1) * (unsigned)pp.s_g : 0u;
  switch (src) {
    case rk::kRow32:
      return launch_src<rk::kRow32>(pp, zmode, grid, stream);
    case kRow32Wide:
      return launch_src<kRow32Wide>(pp, zmode, grid, stream);
    case kRow64:
      return launch_src<kRow64, false>(pp, zmode, grid, stream);
    case kRow128:
      return launch_src<kRow128, false>(pp, zmode, grid, stream);
    case rk::kHalf:
      return launch_src<rk::kHalf>(pp, zmode, grid, stream);
    case rk::kTile:
      return launch_tail<kZeroConstInt, rk::kTile>(pp, grid, stream);
  }
  return launch_form<kZeroConstInt, rk::kChannel, true>(pp, grid, stream);
}

}  // namespace fl
}  // namespace rb200
