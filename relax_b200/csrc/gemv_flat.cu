// Host side of the int4 kernel of one sequence of units per warp: which calls it takes, launch.
#include "gemv_flat.cuh"

namespace rb200 {
namespace fl {

// What decides beside the source of the scales, whose figures stand at each (us, other kernel / this one; graphs of launches
// over 300 MB of weights):
//   * a CTA's row blocks.  The other kernel takes two with one load of x: exactly two are its best case and this one's worst
//     (k 4096, n 6144 to 9472), an even number is ahead there where x counts, above twelve rows;
//   * the rows: a column without a row is not loaded here, so that sixteen rows cost more than nine;
//   * where k ends: a last chunk of one k block costs a whole one here, once for each row block, and chunks are dealt to eight
//     warps whole, where the other kernel leaves the last blocks to be added up by one warp.
int source(const rk::Params& pp, int bits, int zmode, int src, int sm_count) {
  const GemvParams& p = pp.g;
  const bool z = zmode == kZeroGeneral, tail = p.k % 256 != 0, experts = pp.indptr != nullptr;
  if (bits != 4 || (z && !p.z)) return -1;
  const uintptr_t addr = reinterpret_cast<uintptr_t>(p.s) | reinterpret_cast<uintptr_t>(p.z) | (uintptr_t)(pp.s_expert_stride * 2);
  const int64_t weights = (int64_t)p.n * p.k;
  const bool few = p.m <= 4 || experts;  // (an expert's rows are seldom more)
  const bool two = p.m > 8 && !experts;  // m-tiles
  const bool many = p.m > 12;            // rows of two m-tiles
  const int blocks = p.n / 16, ctas = 2 * sm_count;
  const int share = experts ? 3 : (blocks + ctas - 1) / ctas;  // row blocks of a CTA (experts: many pieces of any size)
  const bool pair = share == 2, odd = share % 2 == 1 && share <= 5;
  const int kb = p.k / 64, longest = ((kb + 3) / 4 + kWarps - 1) / kWarps * 4 * kWarps;  // k blocks, if each warp had the most
  const bool single = kb % 4 == 1;  // a last chunk of one
  const bool costs_little = (p.k < 2048 && share > 2) || (two && !z && share == 1 && longest * 10 <= kb * 13);  // and then
  // Groups of 32.  Five to eight rows, where two row blocks cannot share a load of x: eight rows with zero points k 4096 x
  // n 22016 21.9 / 18.6 us (here), k 11008 x n 4096 12.4 / 11.1, k = n = 4096 6.04 / 5.87, k 2048 x n 4096 3.53 / 4.17; without
  // k 5504 x n 4096 8.6 / 6.5 and 1152 x 1040 3.33 / 2.88, but whole chunks k = n = 4096 4.66 / 5.24, n 22016 15.5 / 15.6.
  if (p.group == 32 && p.s_g == 1 && p.s_n % 2 == 0 && (addr & 3u) == 0 && (tail || src == rk::kRow32)) {
    // Sixteen rows: k 11136 x n 4096 18.0 / 15.3, 8320 x 4096 1.08, but whole chunks k 4096 x n 22016 20.2 / 22.2; in pairs k 8256
    // x n 8192 18.9 / 22.1, 4224 x 8192 0.94, one last block k 2112 x n 12288 0.86, with zero points 2176 x 4096 0.94.
    if (p.m <= 4 && !experts) return rk::kRow32;
    if (two) return tail && !pair && (!single || costs_little) && (!z || share > 2 || longest * 2 <= kb * 3 || p.k < 1024) ? kRow32Wide : -1;
    return tail || experts || (z && weights >= (16ll << 20)) ? kRow32Wide : -1;
  }
  if (src == rk::kGeneral || src == rk::kRow32) return -1;
  if (!tail && p.s_g == 1 && p.group == 64 && p.s_n % 4 == 0 && (addr & 7u) == 0)
    // k 2048 x n 4096 without zero points 2.77 / 2.85 us (here), k = n = 4096 4.44 / 3.93; eight rows 3.13 / 3.5, 4.94 / 4.7
    // sixteen rows without zero points k 2048 x n 4096 4.23 / 4.07, k = n = 4096 7.0 / 5.7, k 11008 x n 4096 14.6 / 11.3, with
    // 4.39 / 4.88, 8.7 / 6.2, 16.7 / 12.3
    return experts || (two ? !z || weights >= (16ll << 20) : z || p.k >= 4096) ? kRow64 : -1;
  if (!tail && p.s_g == 1 && p.group == 128 && p.s_n % 2 == 0 && (addr & 3u) == 0) {
    // nine / sixteen rows without zero points k 4096 x n 4096 1.10 / 1.05 times as fast, n 12288 (three blocks) 1.22 / 1.11, n 14336
    // (four) 1.16 / 0.96, n 8192 (a pair) 1.06 / 0.97; with them 1.15 to 1.38 / 1.05 to 1.28
    if (two) return z || odd || p.m <= 14 ? kRow128 : -1;  // (thirteen / fourteen rows n 14336 1.11 / 1.04)
    // four rows in pairs without zero points k 4096 x n 6144 0.96, k 8192 1.02; eight rows with them k = n = 4096 5.12 / 4.83, n 14336
    // 1.09, in pairs 0.94 to 0.97, k 8192 1.02, k 2048 x n 4096 3.34 / 3.58; without them 4.33 / 4.67
    if (few) return z || !pair || p.k >= 8192 ? kRow128 : -1;
    return z && p.k >= 4096 && (!pair || p.k >= 8192) ? kRow128 : -1;
  }
  // whole chunks: k 8192 x n 28672 24.6 / 29; ungrouped short ones k 4224 x n 4096 5.1 / 6.1, 11136 x 4096 8.6 / 9.9, 1088 x 2048
  // 3.03 / 3.08; experts k 2944 x n 4096 1.11 to 1.17, 4160 x 4096 0.88
  if (src == rk::kChannel) return tail && !z && experts && (!single || p.k < 2048) ? src : -1;
  if (src == rk::kTile && z) return -1;  // spills 450 bytes: k 4096 x n 11008, one row 11.1 / 12.1
  if (experts) {
    // eight experts, k 4160 x n 4096, groups of 64: 2 rows 10.2 / 10.7, 16 rows 23.0 / 25.5; k 2048 x n 1024, 2 rows 5.07 / 5.53
    return src == rk::kTile && ((single && p.k >= 2048) || (int64_t)p.m * blocks <= ctas) ? -1 : src;
  }
  // Scales one by one.  A pair of row blocks: k 4096 x n 8192, groups of 128, eight rows with zero points 7.1 / 8.2, one row 6.7 / 7.2,
  // without them 6.1 / 6.7, sixteen rows 8.9 / 9.7; groups of 64 6.3 / 7.0, 9.3 / 10.9; short last chunks k 4224 x n 8192, eight
  // rows 0.95 and 0.96, sixteen 0.90 and 0.95, k 4160, groups of 64 8.2 / 10.2.
  if (pair) return two && !z && !tail && !many && src == rk::kHalf && p.k >= 8192 ? src : -1;  // (nine / twelve rows k 8192 x n 8192 1.06 / 1.02)
  if (tail) {
    // groups of 128: k 11136 x n 4096, one row with zero points 12.8 / 9.7, without 9.3 / 9.0, sixteen rows 18.7 / 16.6, 13.8 / 13.6
    if (src == rk::kHalf) return src;
    // groups of 64: k 11136 x n 4096 11.5 / 9.7, 2944 x 4096 5.1 / 4.8, but 2112 x 4096 3.8 / 4.6, 2176 x 4096, eight rows 0.91, sixteen
    // 1.0, 8256 x 2048 7.2 / 7.7 (nine rows 1.05); three row blocks k 2176 x n 12288 1.16 and 1.04, 1088 1.11 and 1.09, 2112 0.93 and 0.86
    if (single && !costs_little) return -1;
    return share > 2 || p.k < 1024 || longest * 10 <= kb * (two ? 19 : 14) ? src : -1;
  }
  if (src == rk::kHalf) {
    // nine / sixteen rows without zero points: k = n = 4096 1.09 / 1.0, n 12288 (three blocks) 1.17 / 1.06, n 14336 (four)
    // 1.12 / 0.92, k 8192 x n 28672 (seven) 1.05 / 0.94
    if (two && !z) return odd || !many ? src : -1;
    // with them (200 bytes of spills, 250 in the form for short last chunks) k 11008 x n 4096 16.8 / 14.6, k 8192 x n 10240 (three) 1.08 / 0.97, 14336 (four) 1.0 / 0.89, k 4096 x n 22016
    // 25.4 / 26.9
    if (two) return p.k >= 8192 && odd ? src : -1;
    // with them k = n = 4096 4.9 / 4.8, n 12288 1.20, 14336 1.12, k 2048 x n 4096 3.56 / 3.77, 1024 x 1024 3.25 / 3.03
    if (z) return share > 2 || p.k > 2048 || weights <= (4ll << 20) ? src : -1;
    // without them, up to four rows, k 8192 x n 4096 6.35 / 6.57, n 10240 1.11, k 4096 x n 11008 9.3 / 8.5
    return few && share > 2 && weights >= (32ll << 20) ? src : -1;
  }
  // groups of 64 without zero points: nine / sixteen rows k = n = 4096 1.07 / 1.01, k 4096 x n 12288 (three blocks) 1.15 / 1.05, 14336
  // (four) 1.08 / 0.91, k 8192 x n 14336 0.96 / 0.88, 1024 x 8192 0.95 / 0.94, 2048 x 4096 1.03 / 0.95, 4096 x 2048 1.08 / 1.04
  if (two) return weights >= (4ll << 20) && (p.k > 2048 || weights > (8ll << 20)) && (odd || (!many && p.k <= 4096)) ? src : -1;
  // up to four rows k 8192 x n 4096 7.5 / 6.9, k 4096 x n 12288 1.11, 14336 1.05, k = n = 4096 3.88 / 4.06
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
      if constexpr (SRC != rk::kChannel) RB200_CUDA(launch_dependent(gemv_flat_kernel<Z, SRC, kTail, 1>, g, kWarps * 32, 0, stream, pp));
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
