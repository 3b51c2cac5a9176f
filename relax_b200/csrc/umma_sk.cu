// Host side of the medium-batch tensor-core kernel: coverage test, tile and pipeline plan, launch.
#include "umma_sk.cuh"

#include <cmath>
#include <cstring>

#include "tensormap.h"

namespace rb200 {

int umma_sk_run(const GemvParams& p, int bits, int zmode, int sm_count, uint32_t* vacant_words, size_t vacant_bytes,
                const int64_t* indptr, int has_prev, int num_experts, int64_t w_expert_bytes,
                int64_t s_expert_stride, cudaStream_t stream) {
  using namespace us;
  const bool grouped = indptr != nullptr;
  const int64_t per_expert_scales = p.group > 0 ? (int64_t)p.n * p.s_n + (int64_t)(p.k / p.group) * p.s_g : (int64_t)p.n * p.s_n;
  const bool covered = p.n % 16 == 0 && p.k % kKBlock == 0 && (reinterpret_cast<uintptr_t>(p.x) & 15u) == 0 && p.ldx % 8 == 0 &&
                       (reinterpret_cast<uintptr_t>(p.out) & 15u) == 0 && p.ldo % 8 == 0 && p.s_n < (1ll << 31) &&
                       p.s_g < (1ll << 31) && per_expert_scales < (1ll << 40);
  if (!covered) {
    RB200_CHECK(!grouped, "grouped GEMM needs n %% 16 == 0, k %% 64 == 0 and 16-byte aligned x / out rows (n=%d, k=%d)", p.n, p.k);
    return 1;
  }
  RB200_CHECK(!grouped || (num_experts >= 1 && num_experts <= kMaxExperts), "num_experts=%d outside [1, %d]", num_experts,
              kMaxExperts);
  Params pp;
  memset(&pp, 0, sizeof(pp));
  pp.g = p;
  pp.indptr = indptr;
  pp.has_prev = has_prev;
  pp.num_experts = num_experts;
  pp.w_expert_bytes = w_expert_bytes;
  pp.s_expert_stride = s_expert_stride;
  pp.s_n = (int)p.s_n;
  pp.s_g = (int)p.s_g;
  pp.early = launch_overlap_enabled() ? 1 : 0;
  pp.wait_limit_ms = wait_limit_ms();

  Launch l;
  memset(&l, 0, sizeof(l));
  l.zmode = zmode;
  const int lane_run = bits == 4 ? 16 : 8;
  if (p.group <= 0 || p.group >= p.k) {
    l.src = kChannel;
  } else {
    RB200_CHECK(p.group % lane_run == 0 && p.k % p.group == 0, "group_size=%d must divide k=%d and be a multiple of %d", p.group,
                p.k, lane_run);
    l.src = p.group % kKBlock == 0 ? kOne : (p.group == 32 ? kTwo : kAny);
    const uintptr_t addr = reinterpret_cast<uintptr_t>(p.s) | reinterpret_cast<uintptr_t>(p.z);
    pp.s_vec = p.s_g == 1 && p.s_n % 2 == 0 && (addr & 3u) == 0 && s_expert_stride % 2 == 0;
  }

  // Batch rows per tile.  Ungrouped: the batch in equal tiles of at most 256.  Grouped: the split of the
  // rows is known on the device only, so the width is an even share plus three standard deviations
  // of a uniform routing (an expert above it takes a second tile).
  if (grouped) {
    const double even = (double)p.m / num_experts;
    int nb = (int)(even + 3.0 * std::sqrt(even)) + 1;
    if (nb > p.m) nb = p.m;
    nb = (nb + 15) / 16 * 16;
    pp.nb = nb > kMaxNb ? kMaxNb : nb;
    pp.m_tiles = 1;
  } else {
    pp.m_tiles = (p.m + kMaxNb - 1) / kMaxNb;
    pp.nb = ((p.m + pp.m_tiles - 1) / pp.m_tiles + 15) / 16 * 16;
  }
  const bool small = pp.nb <= kSmallNb;
  l.groups = small ? 2 : 4;
  // tensor memory: one or two accumulators, then A slots of one or two 32-column blocks
  if (small) {
    pp.tmem_cols = 256;
    pp.d_stride = pp.nb <= 32 ? 32 : 64;
    pp.nd = 2;
  } else {
    pp.tmem_cols = 512;
    pp.d_stride = pp.nb <= 128 ? 128 : 256;
    pp.nd = pp.nb <= 128 ? 2 : 1;
  }
  pp.a_base = pp.nd * pp.d_stride;
  const int own = bits == 4 && small ? 2 : 1;  // blocks per A slot (kOwn of the kernel)
  pp.na = (pp.tmem_cols - pp.a_base) / (32 * own);
  if (pp.na > kMaxA) pp.na = kMaxA;
  // rings: x stages first (one 64-k block each), then as many weight stages as fit
  const size_t budget = small ? (size_t)(228 * 1024) / 2 - 1024 : (size_t)227 * 1024;
  pp.x_stages = 4;
  pp.w_stages = kMaxStages;
  while (pp.w_stages > 3 && smem_bytes(pp.nb, pp.x_stages, pp.w_stages, l.groups) > budget) --pp.w_stages;
  while (pp.x_stages < kMaxStages && smem_bytes(pp.nb, pp.x_stages + 1, pp.w_stages, l.groups) <= budget) ++pp.x_stages;
  l.smem = smem_bytes(pp.nb, pp.x_stages, pp.w_stages, l.groups);
  RB200_CHECK(l.smem <= budget, "medium-batch kernel: %zu bytes of shared memory for %d batch rows", l.smem, pp.nb);

  const int frag = bits == 4 ? 64 : 32;
  pp.cpt = (p.k / frag + 3) / 4;
  const long long n_tiles = (p.n + kTileRows - 1) / kTileRows;
  // most items a launch can have (grouped: every expert full tiles plus one ragged tile)
  const long long items = grouped ? n_tiles * ((long long)p.m / pp.nb + num_experts) : n_tiles * pp.m_tiles;
  const long long units = items * pp.cpt;
  long long grid = (long long)sm_count * (small ? 2 : 1);
  // a tile cut into many short ranges spends its time in the hand-over: at least three chunks per CTA
  // before a second CTA per SM
  if (small && units < 3 * grid) grid = sm_count;
  if (grid > units) grid = units;
  RB200_CHECK(items * pp.cpt * grid < (1ll << 31), "problem too large for the 32-bit work split (n=%d, k=%d, m=%d)", p.n, p.k, p.m);
  l.grid = (int)grid;
  RB200_CHECK((size_t)grid * pp.nb * kTileRows * sizeof(float) <= vacant_bytes, "split-k scratch too small for a grid of %d", l.grid);
  pp.partial = vacant_words;

  CUtensorMap tx;
  if (make_tensor_map_2d(&tx, p.x, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, (unsigned long long)p.k, (unsigned long long)p.m,
                         (unsigned long long)p.ldx * 2, kKBlock, (unsigned)pp.nb, CU_TENSOR_MAP_SWIZZLE_128B) != 0)
    return -1;
  return bits == 4 ? launch_i4(pp, l, tx, stream) : launch_i8(pp, l, tx, stream);
}

}  // namespace rb200
