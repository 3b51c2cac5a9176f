// Host side of the small-batch kernel: scale source, grid, launch.
#include "gemv_flat.cuh"

#include <cstring>

namespace rb200 {

int gemv_rk_run(const GemvParams& p, int bits, int zmode, int sm_count, const int64_t* indptr, int has_prev,
                int num_experts, int64_t w_expert_bytes, int64_t s_expert_stride, cudaStream_t stream) {
  using namespace rk;
  const int frag = bits == 4 ? 64 : 32;
  RB200_CHECK((reinterpret_cast<uintptr_t>(p.x) & 15u) == 0 && p.ldx % 8 == 0,
              "x must be 16-byte aligned with a row pitch that is a multiple of 8 elements");
  RB200_CHECK(p.m >= 1 && p.m <= (indptr ? 32 : kMaxBatch), "small-batch kernel: m=%d out of range", p.m);
  Params pp;
  memset(&pp, 0, sizeof(pp));
  pp.g = p;
  pp.indptr = indptr;
  pp.has_prev = has_prev;
  pp.num_experts = num_experts;
  pp.w_expert_bytes = w_expert_bytes;
  pp.s_expert_stride = s_expert_stride;
  pp.early = launch_overlap_enabled() ? 1 : 0;
  int src = kChannel;
  pp.group_shift = -1;
  if (p.group > 0 && p.group < p.k) {
    RB200_CHECK(p.group % (frag / 4) == 0 && p.k % p.group == 0,
                "group_size=%d must divide k=%d and be a multiple of %d", p.group, p.k, frag / 4);
    src = p.group % (2 * frag) == 0 ? kHalf : (p.group % frag == 0 ? kTile : kGeneral);
    pp.per = p.group / (src == kHalf ? 2 * frag : frag);
    if ((p.group & (p.group - 1)) == 0)
      for (pp.group_shift = 0; (1 << pp.group_shift) < p.group;) ++pp.group_shift;
    const uintptr_t addr = reinterpret_cast<uintptr_t>(p.s) | reinterpret_cast<uintptr_t>(p.z) |
                           (uintptr_t)(s_expert_stride * 2);
    // whole 16-byte runs of eight group scales per chunk of 256 k
    if (bits == 4 && p.group == 32 && p.s_g == 1 && p.s_n % 8 == 0 && p.k % 256 == 0 && (addr & 15u) == 0) src = kRow32;
  }
  // 32-bit offsets of scales and activations
  if (p.s_n >= (1ll << 31) || p.s_g >= (1ll << 31) || (p.n + 16) * p.s_n + (p.k / frag) * 4 * p.s_g >= (1ll << 31) ||
      p.ldx * p.m >= (1ll << 31))
    return 1;
  pp.s_n = (int)p.s_n;
  pp.s_g = (int)p.s_g;
  const long long blocks = (long long)(p.n / 16) * (indptr ? num_experts : 1);
  const int flat = fl::source(pp, bits, zmode, src, sm_count);
  // Eight k slices while an SM has few row blocks (its 16 warps are two CTAs), four once there are
  // enough for four CTAs: half the passes per byte.  Measured: k 8192 x n 28672 int8 (12 row blocks
  // per SM) 44 -> 41 us, k 4096 x n 22016 int4 (9.3) 13.7 -> 13.9 us, k = n = 4096 (1.7) 3.9 -> 5.8 us.
  const int warps = flat < 0 && blocks >= (long long)sm_count * 12 ? 4 : 8;
  long long grid = (long long)sm_count * (16 / warps);
  if (grid > blocks) grid = blocks;
  // the kernel numbers row blocks entry by entry: an expert may have several, and most have none
  const long long numbered = indptr ? (long long)(p.n / 16) * kMaxEntries : blocks;
  RB200_CHECK(numbered * grid < (1ll << 32), "too many row blocks for the small-batch kernel (n=%d)", p.n);
  pp.per_cta = (unsigned)(blocks / grid);
  pp.extra = (unsigned)(blocks % grid);
  if (flat >= 0) return fl::launch(pp, zmode, flat, (int)grid, stream);
  return bits == 4 ? launch_i4(pp, zmode, src, warps, (int)grid, stream) : launch_i8(pp, zmode, src, warps, (int)grid, stream);
}

}  // namespace rb200
