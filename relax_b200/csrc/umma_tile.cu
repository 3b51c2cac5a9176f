// Host side of the tensor-core kernels over packed weights: coverage test, tile and pipeline plan, choice
// between the one-CTA form (umma_sk) and CTA pairs (umma_pair), launch.
#include "umma_pair.cuh"
#include "umma_sk.cuh"

#include <cmath>
#include <cstring>

#include "handover.h"
#include "tensormap.h"

namespace rb200 {

namespace {
using namespace us;

int x_map(CUtensorMap* tx, const GemvParams& p, int rows) {
  return make_tensor_map_2d(tx, p.x, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, (unsigned long long)p.k, (unsigned long long)p.m,
                            (unsigned long long)p.ldx * 2, kKBlock, (unsigned)rows, CU_TENSOR_MAP_SWIZZLE_128B);
}

// Batch tiles of the pair kernel: of the splits of m into equal tiles of at most 256 rows, the one that the
// clock counts below say is done first.  Per 64-k block the tensor pipe takes 2 nb clocks and the decode
// of a CTA's 128 rows by two groups of warps about 320 (the counts know neither the third group of tiles of 161 to
// 192 rows nor that two accumulators hide the drain up to 160), whichever is longer, so wide tiles win (2048 rows as 8 x 256 against
// 11 x 192 with two accumulators of that width, a form no longer here: 662 / 828 us for int8 k 8192 x
// n 28672) - unless there are too few of them for the pairs: a tile cut over c more pairs costs its owner about 1600 clocks per
// two parts and 48 columns (a trip to L2 each).
int pair_m_tiles(long long n_tiles, int m, int k_blocks, int pairs) {
  int best = 0;
  double best_clk = 0.0;
  const int least = (m + kMaxNb - 1) / kMaxNb;
  for (int t = least; t <= least + 8; ++t) {
    const int nb = ((m + t - 1) / t + 31) / 32 * 32;
    if (t > least && nb < 64) break;
    const long long items = n_tiles * ((m + nb - 1) / nb);
    const double tiles = (double)items / pairs;
    double clk = tiles * k_blocks * (nb * 2 > 320 ? nb * 2 : 320) + (tiles > 1.0 ? tiles : 1.0) * nb / 48.0 * 600.0;
    if (items % pairs) clk += std::ceil((tiles < 1.0 ? 1.0 / tiles : 1.0) / 2.0) * nb / 48.0 * 1600.0;
    if (best == 0 || clk < best_clk) {
      best = t;
      best_clk = clk;
    }
  }
  return best;
}

int run_pair(Params& pp, int bits, int zmode, int src, int sm_count, cudaStream_t stream) {
  const GemvParams& p = pp.g;
  const long long n_tiles = (p.n + 2 * kTileRows - 1) / (2 * kTileRows);
  if (!pp.indptr) {
    pp.m_tiles = pair_m_tiles(n_tiles, p.m, p.k / kKBlock, sm_count / 2);
    pp.nb = (p.m + pp.m_tiles - 1) / pp.m_tiles;
  }
  pp.nb = (pp.nb + 31) / 32 * 32;
  if (!pp.indptr) pp.m_tiles = (p.m + pp.nb - 1) / pp.nb;  // no tile without rows (an MMA of width 0 is illegal)
  // tensor memory: two accumulators of up to 160 columns or one of 256, then A slots of 64 columns (at least three:
  // int8 k 8192 x n 57344, 160 rows, two accumulators 139 us, one 142; int4 k 4096 x n 22016, group 32, 129 rows
  // 35.0 / 36.7)
  pp.tmem_cols = 512;
  pp.nd = pp.nb <= 160 ? 2 : 1;
  pp.d_stride = pp.nb <= 128 ? 128 : (pp.nb <= 160 ? 160 : (pp.nb <= 192 ? 192 : 256));
  pp.a_base = pp.nd * pp.d_stride;
  pp.na = (pp.tmem_cols - pp.a_base) / 64;
  if (pp.na > kMaxA) pp.na = kMaxA;
  const size_t budget = (size_t)227 * 1024;
  pp.x_stages = kMaxStages;
  pp.w_stages = kMaxStages;
  while (pp.w_stages > 4 && up::smem_bytes(pp.nb, pp.x_stages, pp.w_stages) > budget) --pp.w_stages;
  while (pp.x_stages > 2 && up::smem_bytes(pp.nb, pp.x_stages, pp.w_stages) > budget) --pp.x_stages;
  up::Launch l;
  memset(&l, 0, sizeof(l));
  l.zmode = zmode;
  l.src = src;
  l.smem = up::smem_bytes(pp.nb, pp.x_stages, pp.w_stages);
  RB200_CHECK(l.smem <= budget, "pair kernel: %zu bytes of shared memory for %d batch rows", l.smem, pp.nb);
  // most items a launch can have (grouped: every expert full tiles plus one ragged tile)
  const long long items = pp.indptr ? n_tiles * ((long long)p.m / pp.nb + pp.num_experts) : n_tiles * pp.m_tiles;
  RB200_CHECK(items < (1ll << 30), "too many tiles (n=%d, m=%d)", p.n, p.m);
  l.most_pairs = items * pp.cpt;
  pp.partial = handover_words(stream, sm_count, (size_t)sm_count * pp.nb * kTileRows * sizeof(float));
  CUtensorMap tx;  // x as [64-k block][row][64 k]
  {
    const unsigned long long dims[3] = {64ull, (unsigned long long)p.m, (unsigned long long)(p.k / 64)};
    const unsigned long long strides[2] = {(unsigned long long)p.ldx * 2ull, 128ull};
    const unsigned box[3] = {64u, (unsigned)(pp.nb / 2), 2u};
    if (make_tensor_map(&tx, p.x, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 3, dims, strides, box, CU_TENSOR_MAP_SWIZZLE_128B) != 0)
      return -1;
  }
  return bits == 4 ? up::launch_i4(pp, l, tx, stream) : up::launch_i8(pp, l, tx, stream);
}

int run_single(Params& pp, int bits, int zmode, int src, int sm_count, cudaStream_t stream) {
  const GemvParams& p = pp.g;
  if (!pp.indptr) {
    pp.m_tiles = (p.m + kSmallNb - 1) / kSmallNb;
    pp.nb = (p.m + pp.m_tiles - 1) / pp.m_tiles;
  }
  pp.nb = (pp.nb + 15) / 16 * 16;
  if (!pp.indptr) pp.m_tiles = (p.m + pp.nb - 1) / pp.nb;
  // tensor memory: two accumulators, then A slots
  pp.tmem_cols = 256;
  pp.d_stride = pp.nb <= 32 ? 32 : 64;
  pp.nd = 2;
  pp.a_base = pp.nd * pp.d_stride;
  const int own = bits == 4 ? 2 : 1;  // blocks per A slot (kOwn of the kernel)
  pp.na = (pp.tmem_cols - pp.a_base) / (32 * own);
  if (pp.na > kMaxA) pp.na = kMaxA;
  // rings: x stages first (one 64-k block each), then as many weight stages as fit
  const size_t budget = kCtaSmem;
  pp.x_stages = 4;
  pp.w_stages = kMaxStages;
  while (pp.w_stages > 3 && smem_bytes(pp.nb, pp.x_stages, pp.w_stages) > budget) --pp.w_stages;
  while (pp.x_stages < kMaxStages && smem_bytes(pp.nb, pp.x_stages + 1, pp.w_stages) <= budget) ++pp.x_stages;
  Launch l;
  memset(&l, 0, sizeof(l));
  l.zmode = zmode;
  l.src = src;
  l.smem = smem_bytes(pp.nb, pp.x_stages, pp.w_stages);
  RB200_CHECK(l.smem <= budget, "medium-batch kernel: %zu bytes of shared memory for %d batch rows", l.smem, pp.nb);
  const long long n_tiles = (p.n + kTileRows - 1) / kTileRows;
  const long long items = pp.indptr ? n_tiles * ((long long)p.m / pp.nb + pp.num_experts) : n_tiles * pp.m_tiles;
  const long long units = items * pp.cpt;
  // Split: when the tiles leave room for two or more CTAs each, every tile is cut into the same number of
  // ranges - no CTA then drains two pieces (k 4096 x n 12288, 24 rows: 13.2 us in 96 x 3 ranges, 15.1 in
  // 296 equal runs; n 4096: 9.7 / 11.3) - of at least ten 64-k blocks, or sixteen where the hand-over of a
  // part is twice as large.  Otherwise equal runs over the tiles (n 22016, 172 tiles).
  long long grid = (long long)sm_count * 2;
  if (!pp.indptr) {
    long long ranges = grid / items;
    const long long longest = (p.k / kKBlock) / (pp.nb <= 32 ? 10 : 16);
    if (ranges > longest) ranges = longest;
    if (ranges > 8) ranges = 8;
    if (ranges >= 2 || items <= sm_count) grid = items * (ranges > 1 ? ranges : 1);
    // Where the parts of a tile are many or large they are added inside a cluster: one exchange through shared memory in
    // place of a trip to memory per part.  Without overlap of launches, us without / with: k 4096 x n 4096 int4 group 32,
    // 32 rows 12.2 / 11.5, 64 rows 14.8 / 13.3; k 14336 x n 4096 32 rows 20.3 / 18.5; k 11008 x n 4096 64 rows 23.4 / 18.7;
    // k 8192 x n 1024 64 rows 18.6 / 11.7; int8 per row k 8192 x n 4096 64 rows 22.7 / 17.6.  Nine to sixteen rows come here with
    // groups of 32 and zero points: sixteen, k 14336 x n 4096 23.1 / 21.8, k 28672 x n 2048 32.0 / 31.4, k 57344 x n 1024
    // 48.3 / 37.4.  Fewer or smaller parts lose to the two cluster barriers (32 rows, k 2048 x n 4096 in three CTAs a tile
    // 9.3 / 11.1; 48 rows of int8 in four 1 % slower), and clusters that do not all run at once to the second wave (k 4096 x
    // n 12288, 96 x 3: 15.0 / 27.3).  Overlapped launches of up to 32 rows start late in an SM that is full of them: there only
    // up to a CTA per SM (k 4096 x n 2048 9.6 / 8.3; n 4096, 256 CTAs, 10.4 / 11.0).
    const int k_blocks = p.k / kKBlock;
    int wide = k_blocks / 8 < 8 ? k_blocks / 8 : 8;
    while (wide >= 4 && cluster_places(wide) < items) --wide;
    if (pp.nb <= 32 ? wide == 8 && (!pp.early || items * wide <= sm_count)
                    : (wide > 4 || (wide == 4 && k_blocks >= 64)) && wide * pp.nb >= (bits == 4 ? 192 : 256)) {
      l.ranges = wide;
      grid = items * wide;
    }
  } else if (units < 3 * grid) {
    grid = sm_count;  // a tile cut into many short ranges spends its time in the hand-over
  }
  if (grid > units) grid = units;
  RB200_CHECK(units * grid < (1ll << 31), "problem too large for the 32-bit work split (n=%d, k=%d, m=%d)", p.n, p.k, p.m);
  // (one CTA per tile cuts none)
  if (!l.ranges && (pp.indptr || grid != items)) pp.partial = handover_words(stream, sm_count, (size_t)grid * pp.nb * kTileRows * sizeof(float));
  // A tile per SM is not cut: its first CTA makes one, the second a run of the rest.  That saves a quarter of the pieces
  // where the tiles come near two per SM; with fewer the second CTA is done before the first, by more or less as the equal
  // runs' cuts fall.  k 4096, us in equal runs / so, 32 and 64 rows: int4 group 32 n 20480 (160 tiles) 21.9 / 24.5 and 24.9 / 29.1,
  // n 22016 (172) 23.1 / 21.9 and 26.1 / 28.9, n 26624 (208) 26.4 / 28.3 and 29.4 / 29.7, n 30208 (236) 28.0 / 29.0 and 31.1 /
  // 30.4, n 31616 (247) 29.6 / 29.6 and 32.7 / 31.1, n 32016 (251) 29.9 / 29.7 and 32.9 / 31.2, n 36000 (282) 32.1 / 32.0 and 34.8 /
  // 34.5; int8 per row n 22016 25.5 / 27.0 and 28.8 / 31.3, n 26624 30.0 / 28.9 and 33.5 / 33.5, n 32016 33.1 / 32.2 and 37.2 / 35.4,
  // n 36000 35.9 / 35.2 and 39.7 / 38.5.
  // (More CTAs than tiles, so two chunks a tile at least, and no fewer chunks are left than second CTAs.)
  if (!pp.indptr && pp.partial && grid == 2ll * sm_count && items < grid && (pp.nb > 32 ? items * 5 >= sm_count * 8ll : items * 3 >= sm_count * 5ll))
    pp.whole = sm_count;
  l.grid = (int)grid;
  CUtensorMap tx;
  if (x_map(&tx, p, pp.nb) != 0) return -1;
  return bits == 4 ? launch_i4(pp, l, tx, stream) : launch_i8(pp, l, tx, stream);
}
}  // namespace

int umma_run(const GemvParams& p, int bits, int zmode, int sm_count, const int64_t* indptr, int has_prev, int num_experts,
             int64_t w_expert_bytes, int64_t s_expert_stride, cudaStream_t stream) {
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
  // (what the switch promises about weights it promises for decode batches only)
  pp.early = launch_overlap_enabled() && !grouped && p.m <= 32 ? 1 : 0;
  pp.wait_limit_ms = wait_limit_ms();

  const int lane_run = bits == 4 ? 16 : 8;
  int src;
  if (p.group <= 0 || p.group >= p.k) {
    src = kChannel;
  } else {
    RB200_CHECK(p.group % lane_run == 0 && p.k % p.group == 0, "group_size=%d must divide k=%d and be a multiple of %d", p.group,
                p.k, lane_run);
    src = p.group % kKBlock == 0 ? kOne : (p.group == 32 ? kTwo : kAny);
    pp.blk_shift = -1;
    const int blocks = p.group / kKBlock;
    if (src == kOne && (blocks & (blocks - 1)) == 0)
      for (pp.blk_shift = 0; (1 << pp.blk_shift) < blocks;) ++pp.blk_shift;
    const uintptr_t addr = reinterpret_cast<uintptr_t>(p.s) | reinterpret_cast<uintptr_t>(p.z);
    auto words_of = [&](int halves) {
      return p.s_g == 1 && p.s_n % halves == 0 && (addr & (uintptr_t)(2 * halves - 1)) == 0 && s_expert_stride % halves == 0;
    };
    pp.s_vec = words_of(4) && pairs_fit_rows(p.k, bits) ? 2 : (words_of(2) ? 1 : 0);
  }

  const int frag = bits == 4 ? 64 : 32;
  pp.cpt = (p.k / frag + 3) / 4;
  if (grouped) {
    // The split of the rows over the experts is known on the device only: the tile is an even share plus
    // three standard deviations of a uniform routing (rows drawn one by one) wide; an expert above it takes a second
    // tile.  With the deviation of a Poisson count 1024 rows over 8 experts had tiles of 192 columns, one accumulator,
    // instead of 160, two: int4 group 128, k 4096 x n 14336 143.8 -> 131.5 us, int8 k 4096 x n 8192 96.9 -> 90.6.
    const double even = (double)p.m / num_experts;
    int nb = (int)(even + 3.0 * std::sqrt(even * (1.0 - 1.0 / num_experts))) + 1;
    if (nb > p.m) nb = p.m;
    pp.nb = nb > kMaxNb ? kMaxNb : nb;
    pp.m_tiles = 1;
  }
  const bool single = (grouped ? pp.nb : p.m) <= kSmallNb;
  return single ? run_single(pp, bits, zmode, src, sm_count, stream) : run_pair(pp, bits, zmode, src, sm_count, stream);
}

}  // namespace rb200
