// Medium batches (17 to 64 rows, and expert layers with as few rows per expert) on the 5th-generation
// tensor cores, with the work split evenly over the SMs.
//
//   out^T tile [128 weight rows x nb batch rows] = W_tile [128 x K] * x_tile^T [K x nb]
//
// Bound: HBM (the packed weight once) and the decode arithmetic; one tcgen05.mma of width N with A
// in tensor memory takes N / 2 clocks (9 at N = 16, 32 at 64, 128 at 256), so up to about 90 rows the
// tensor pipe waits for the weights.  Dequantised weights go from registers straight to tensor
// memory (thread = weight row = TMEM lane), never through shared memory; the batch is the MMA's N,
// padded to 16 only.
//
// Work split: all (tile, chunk of k) units in one line, cut into equal contiguous ranges, one per CTA
// (stream-k), so that neither the number of tiles nor a short last wave leaves SMs idle.  A CTA that
// starts inside a tile publishes its partial accumulator (fp32, global scratch); the CTA that holds
// the tile's first chunk adds the others' parts in CTA order at the end of its own range - they were
// published at the start of theirs.  The result does not depend on timing.  The scratch words are
// their own flags: at rest they hold a NaN pattern that no sum has (kVacant), the owner polls them -
// several contributors' words requested together, one trip to memory per try - and puts the pattern
// back.  (A fence, a flag and a second trip per contributor cost 6 us at k = n = 4096.)
// Where a tile is cut into equal parts that are many or large, its CTAs form a cluster instead and each adds up its
// share of the columns (kCluster; the rule and its figures are beside the split in umma_tile.cu): the owner's trips to
// memory, one per part, were up to a third of such a launch, and the registers for several parts a trip spill.
//
//   warp 0  packed weights, one 16 KB bulk copy per chunk (128 rows x 256 | 128 k)
//   warp 1  MMA: four per 64-k block, by an elected thread
//   warp 2  x: one TMA tile [nb rows x 64 k] per block, 128-byte swizzle = K-major operand
//   warps 4-11  two groups of four warps decode a share of each chunk's blocks, then drain the
//           accumulator: bias / activation / residual, one rounding, transpose through shared memory,
//           whole-line stores.
// 256 TMEM columns and half the shared memory per CTA, so two CTAs share an SM and one's decode covers
// the other's waits.
// Every wait is bounded and reports through the device status word.
//
// Stands in for fastertransformer::gemm_fp16_int_bias_act[_residual]
// (python/tvm/contrib/cutlass/gemm_operation.py:441-458) and, grouped, the expert form of
// src/runtime/contrib/cutlass/fp16_group_gemm.cu:39-64 over quantised weights.
#pragma once

#include "umma_tile.cuh"

namespace rb200 {
namespace us {

constexpr int kSmallNb = 64;            // up to here two CTAs share an SM
constexpr int kGroups = 2;              // decode groups of four warps
constexpr size_t kCtaSmem = 228 * 1024 / 2 - 1024;  // the most for two CTAs per SM

inline size_t bar_bytes() { return (size_t)(4 * kMaxStages + 2 * kMaxA + 4 + kGroups) * 8 + 16 + (3 * kMaxExperts + 4) * sizeof(int); }
inline size_t smem_bytes(int nb, int x_stages, int w_stages) {
  return 1024 + (size_t)x_stages * nb * 128 + (size_t)w_stages * kWBytes + kGroups * kStageBytes + bar_bytes();
}

// How the tiles are cut: equal runs of chunks, a tile each for the first CTAs and runs of the rest (Params::whole), or
// every tile over a cluster.
enum Split { kRuns, kWholeFirst, kCluster };
struct Launch {
  int grid, zmode, src;
  int ranges;  // every tile is shared by a cluster of as many CTAs, 0: parts go through global scratch
  size_t smem;
};
int launch_i4(const Params& pp, const Launch& l, const CUtensorMap& tx, cudaStream_t stream);
int cluster_places(int ranges);  // clusters of so many CTAs that run at a time
int launch_i8(const Params& pp, const Launch& l, const CUtensorMap& tx, cudaStream_t stream);

#ifdef __CUDACC__

using ug::tc_commit;
using ug::tc_mma_ts;

__device__ __forceinline__ void tma_load_x(void* smem_dst, const CUtensorMap* map, int c0, int c1, uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(
          smem_u32(smem_dst)),
      "l"(map), "r"(c0), "r"(c1), "r"(smem_u32(bar))
      : "memory");
}

__device__ __forceinline__ uint32_t cluster_nctarank() {
  uint32_t r;
  asm("mov.u32 %0, %%cluster_nctaid.x;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void cluster_sync() {
  __syncwarp();
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// An address of this CTA's shared memory in that of the cluster's CTA `rank`.
__device__ __forceinline__ uint32_t map_to(uint32_t addr, int rank) {
  uint32_t to;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(to) : "r"(addr), "r"(rank));
  return to;
}

// Parts of a tile in one cluster: each CTA sends column c of its accumulator to the CTA that adds it up, in place of that
// CTA's ring of weights (at most 64 + 7 columns of 512 bytes; the ring has at least three stages of 16 KB).  Columns and not
// weight rows: a thread's sixteen values go to few CTAs, 128 bytes a warp each.
__device__ __forceinline__ void exchange_send(uint32_t ring, uint32_t d, int cols, int rank, int ranks, int grp, int gj) {
  const int most = (cols + ranks - 1) / ranks;
  for (int c0 = grp * 16; c0 < cols; c0 += kGroups * 16) {
    float v[16];
    tc_ld16(d + (uint32_t)c0, v);
    int to = ((c0 + 1) * ranks - 1) / cols, lo = cols * to / ranks, hi = cols * (to + 1) / ranks;
    uint32_t dst = map_to(ring, to);
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      const int c = c0 + i;
      if (c >= cols) break;
      if (c >= hi) {
        do {
          ++to;
          lo = hi;
          hi = cols * (to + 1) / ranks;
        } while (c >= hi);
        dst = map_to(ring, to);
      }
      asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(dst + (uint32_t)(((rank * most + c - lo) * kTileRows + gj) * 4)),
                   "f"(v[i])
                   : "memory");
    }
  }
}
// This CTA's columns, half of them each group's, a weight row per thread; parts in the order of the CTAs as in drain_store.
template <bool SCALED>
__device__ __forceinline__ void exchange_store(const Params& pp, const float* parts, const float* scales, int n0, int m0, int cols, int rank,
                                               int ranks, int grp, int row) {
  const GemvParams& p = pp.g;
  const int most = (cols + ranks - 1) / ranks, lo = cols * rank / ranks, hi = cols * (rank + 1) / ranks, half = (hi - lo + 1) / 2;
  const int first = lo + grp * half, end = grp ? hi : lo + half;
  // where the sending thread of this weight row put it: its tensor-memory lane
  const int blk = row >> 4, lane = (((row >> 3) & 1) + 2 * (blk >> 2)) * 32 + (blk & 3) * 8 + (row & 7);
  const float scale = SCALED ? scales[lane] : 1.0f;
  const int n = n0 + row;
  for (int c = first; c < end; c += 4) {
    float v[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) v[i] = parts[(min(c + i, end - 1) - lo) * kTileRows + lane];
    for (int s = 1; s < ranks; ++s)
#pragma unroll
      for (int i = 0; i < 4; ++i) v[i] += parts[(s * most + min(c + i, end - 1) - lo) * kTileRows + lane];
    if (SCALED) {
#pragma unroll
      for (int i = 0; i < 4; ++i) v[i] *= scale;
    }
    const int m = m0 + c, m_end = m0 + end;
    if (p.epi.act == kActSwiglu) {
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float up = __shfl_down_sync(0xffffffffu, v[i], 8);
        if (m + i < m_end && n < p.n && !(row & 8))
          p.out[(int64_t)(m + i) * p.ldo + n0 / 2 + blk * 8 + (row & 7)] = __float2half_rn(silu_mul(v[i], up));
      }
    } else {
#pragma unroll
      for (int i = 0; i < 4; ++i)
        if (m + i < m_end && n < p.n) p.out[(int64_t)(m + i) * p.ldo + n] = __float2half_rn(apply_epilogue(v[i], p.epi, m + i, n));
    }
  }
}

template <int BITS, int ZMODE, int SRC, int SPLIT>
__global__ void __launch_bounds__((4 + 4 * kGroups) * 32, 2)
    umma_sk_kernel(const Params pp, const __grid_constant__ CUtensorMap tmap_x) {
  constexpr int kBlkPerChunk = BITS == 8 ? 2 : 4;   // 64-k blocks per weight stage
  constexpr int kTilesPerBlk = BITS == 8 ? 2 : 1;
  constexpr int kFragK = BITS == 8 ? 32 : 64;
  constexpr int kOwn = kBlkPerChunk / kGroups;  // adjacent blocks of a chunk one group decodes: an A slot
  constexpr bool kExchange = SPLIT == kCluster;
  extern __shared__ uint8_t smem_raw[];
  const GemvParams& p = pp.g;
  // 1 KB alignment as an offset from the array (a pointer rebuilt from an integer would turn every
  // shared-memory access of the decode warps into a generic one)
  uint8_t* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
  const int nb = pp.nb, x_stages = pp.x_stages, w_stages = pp.w_stages;
  const int x_stage_bytes = nb * 128;
  uint8_t* x_ring = smem;
  uint8_t* w_ring = x_ring + (size_t)x_stages * x_stage_bytes;
  uint8_t* e_stage = w_ring + (size_t)w_stages * kWBytes;
  uint64_t* w_full = reinterpret_cast<uint64_t*>(e_stage + kGroups * kStageBytes);
  uint64_t* w_empty = w_full + kMaxStages;
  uint64_t* x_full = w_empty + kMaxStages;
  uint64_t* x_empty = x_full + kMaxStages;
  uint64_t* a_full = x_empty + kMaxStages;
  uint64_t* a_empty = a_full + kMaxA;
  uint64_t* d_full = a_empty + kMaxA;
  uint64_t* d_empty = d_full + 2;
  uint64_t* e_bar = d_empty + 2;
  uint32_t* tmem_holder = reinterpret_cast<uint32_t*>(e_bar + kGroups);
  volatile uint32_t* const gave_up = tmem_holder + 1;  // kCluster: a wait of one of its CTAs ran out
  Tables& tt = *reinterpret_cast<Tables*>(tmem_holder + 4);

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const bool grouped = !kExchange && pp.indptr != nullptr;
  bool fine = true;
  if (tid == 0) {
    for (int s = 0; s < w_stages; ++s) {
      mbar_init(&w_full[s], 1);
      mbar_init(&w_empty[s], 4 * kGroups);
    }
    for (int s = 0; s < x_stages; ++s) {
      mbar_init(&x_full[s], 1);
      mbar_init(&x_empty[s], 1);
    }
    for (int i = 0; i < pp.na; ++i) {
      mbar_init(&a_full[i], 4);
      mbar_init(&a_empty[i], 1);
    }
    for (int i = 0; i < pp.nd; ++i) {
      mbar_init(&d_full[i], 1);
      mbar_init(&d_empty[i], 4 * kGroups);
    }
    for (int i = 0; i < kGroups; ++i) mbar_init(&e_bar[i], 4);
    mbar_fence_init();
    *gave_up = 0u;
  }
  if (warp == 1) {
    ug::tmem_alloc(tmem_holder, (uint32_t)pp.tmem_cols);
    ug::tmem_relinquish();
  }
  const int n_tiles = (p.n + kTileRows - 1) / kTileRows;
  if (grouped) {
    griddep_wait();  // the row table is the routing kernel's output
    if (tid < pp.num_experts) {
      const int r0 = (tid || pp.has_prev) ? (int)pp.indptr[tid - 1] : 0;
      const int r1 = min((int)pp.indptr[tid], p.m);  // never past the rows x / out hold
      tt.row_begin[tid] = r0;
      tt.row_end[tid] = max(r1, r0);
    }
    __syncthreads();
    if (tid == 0) {
      int acc = 0;
      for (int e = 0; e < pp.num_experts; ++e) {
        tt.base[e] = acc;
        acc += n_tiles * ((tt.row_end[e] - tt.row_begin[e] + nb - 1) / nb);
      }
      tt.base[pp.num_experts] = acc;
    }
  }
  fence_proxy_async();
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  // only now, with this CTA's tensor memory in hand: a dependent CTA that took it first would hold it
  // until this grid has ended
  griddep_launch_dependents();
  const uint32_t tmem = *tmem_holder;

  const int NB = p.n / 16, KT = p.k / kFragK, cpt = pp.cpt;
  const unsigned items = grouped ? (unsigned)tt.base[pp.num_experts] : (unsigned)(n_tiles * pp.m_tiles);
  const unsigned total = items * (unsigned)cpt;  // total * grid fits 31 bits (checked by the host)
  // what the cuts fall between: chunks, or tiles where there are no words to hand over a part of one
  const unsigned step = kExchange || pp.partial ? 1u : (unsigned)cpt, units = kExchange || pp.partial ? total : items;
  // (experts without rows can leave fewer units than CTAs: the surplus CTAs stay out of the split)
  const unsigned ctas = min(gridDim.x, units);
  unsigned u_begin = blockIdx.x < ctas ? blockIdx.x * units / ctas * step : 0u;
  unsigned u_end = blockIdx.x < ctas ? (blockIdx.x + 1) * units / ctas * step : 0u;
  [[maybe_unused]] unsigned whole = 0u, base = 0u, rest = 0u, takers = 0u;
  if constexpr (SPLIT == kWholeFirst) {
    // (rest >= takers: see the rule in umma_tile.cu; a CTA without a chunk inside an owner's range would be waited for)
    whole = (unsigned)pp.whole, base = whole * (unsigned)cpt, rest = total - base, takers = ctas - whole;
    const unsigned idx = blockIdx.x - whole;
    u_begin = blockIdx.x < whole ? blockIdx.x * (unsigned)cpt : base + idx * rest / takers;
    u_end = blockIdx.x < whole ? u_begin + (unsigned)cpt : base + (idx + 1) * rest / takers;
  }

  auto get_item = [&](int item) {
    Item it;
    if (grouped) {
      int e = 0;
      while (e + 1 < pp.num_experts && item >= tt.base[e + 1]) ++e;
      const int rows = tt.row_end[e] - tt.row_begin[e];
      const int mt = (rows + nb - 1) / nb, local = item - tt.base[e];
      it.e = e;
      it.n_tile = local / mt;
      it.m0 = tt.row_begin[e] + (local - it.n_tile * mt) * nb;
      it.m_end = tt.row_end[e];
    } else {
      it.e = 0;
      it.n_tile = item / pp.m_tiles;
      it.m0 = (item - it.n_tile * pp.m_tiles) * nb;
      it.m_end = p.m;
    }
    return it;
  };
  // The CTA's pieces in order: item, chunks [c0, c1).
  struct Walk {
    unsigned u;
    int item, c0, c1;
  };
  auto begin = [&](Walk& w) {
    w.u = u_begin;
    if (u_begin >= u_end) return false;
    w.item = (int)(u_begin / (unsigned)cpt);
    w.c0 = (int)(u_begin - (unsigned)w.item * (unsigned)cpt);
    w.c1 = min(cpt, w.c0 + (int)(u_end - u_begin));
    return true;
  };
  auto next = [&](Walk& w) {
    w.u += (unsigned)(w.c1 - w.c0);
    if (w.u >= u_end) return false;
    ++w.item;
    w.c0 = 0;
    w.c1 = min(cpt, (int)(u_end - w.u));
    return true;
  };
  // 64-k blocks of chunk c
  auto blocks_of = [&](int c) { return min(4, KT - c * 4) / kTilesPerBlk; };

  if (warp == 0) {
    // ============================================================ producer: packed weights
    Walk w;
    bool have = begin(w), ok = true;
    if (have && !pp.early && !grouped) {
      // only into L2 before the wait: a prefetch returns nothing to this kernel, so it is safe
      // whatever the previous one still writes
      if (lane == 0) {
        const Item it = get_item(w.item);
        for (int c = w.c0; c < min(w.c1, w.c0 + w_stages); ++c)
          asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(p.w + frag_stage_offset(it.n_tile, c, NB, KT)),
                       "r"(min(4, KT - c * 4) * min(8, NB - it.n_tile * 8) * 512)
                       : "memory");
      }
      griddep_wait();
    }
    int ws = 0;
    uint32_t ph = 1;
    for (; ok && have; have = next(w)) {
      const Item it = get_item(w.item);
      const uint8_t* w_e = p.w + it.e * pp.w_expert_bytes;
      for (int c = w.c0; c < w.c1; ++c) {
        if (!mbar_wait_parked(&w_empty[ws], ph, p.status)) {
          ok = false;
          break;
        }
        if (lane == 0) {
          const uint32_t bytes = (uint32_t)(min(4, KT - c * 4) * min(8, NB - it.n_tile * 8)) * 512u;
          mbar_arrive_expect_tx(&w_full[ws], bytes);
          bulk_g2s(w_ring + (size_t)ws * kWBytes, w_e + frag_stage_offset(it.n_tile, c, NB, KT), bytes, &w_full[ws]);
        }
        __syncwarp();
        if (++ws == w_stages) {
          ws = 0;
          ph ^= 1u;
        }
      }
    }
  } else if (warp == 1) {
    // ============================================================ MMA issuer (elected thread)
    const uint32_t idesc = (1u << 4) | ((uint32_t)(nb >> 3) << 17) | ((uint32_t)(128 >> 4) << 24);
    const bool leader = elect_one();
    const uint64_t x_desc0 = make_b_desc(smem_u32(x_ring));
    uint64_t x_desc = x_desc0;
    int xs = 0, ab = 0, db = 0;
    uint32_t xph = 0, aph = 0, dph = 1;
    Walk w;
    bool ok = true;
    for (bool have = begin(w); ok && have; have = next(w)) {
      if (!mbar_wait_parked(&d_empty[db], dph, p.status)) break;
      tc_fence_after();
      const uint32_t d = tmem + (uint32_t)(db * pp.d_stride);
      uint32_t acc = 0u;
      for (int c = w.c0; c < w.c1 && ok; ++c) {
        const int nblk = blocks_of(c);
        for (int b0 = 0; b0 < nblk; b0 += kOwn) {
          if (!mbar_wait_parked(&a_full[ab], aph, p.status)) {
            ok = false;
            break;
          }
          uint32_t a = tmem + (uint32_t)(pp.a_base + ab * (kOwn * 32));
          for (int i = 0; i < min(kOwn, nblk - b0); ++i, a += 32) {
            if (!mbar_wait_parked(&x_full[xs], xph, p.status)) {
              ok = false;
              break;
            }
            tc_fence_after();
            if (leader) {
              tc_mma_ts(d, a, x_desc, idesc, acc);
#pragma unroll
              for (int j = 1; j < 4; ++j) tc_mma_ts(d, a + j * 8, x_desc + j * 2, idesc, 1u);
              tc_commit(&x_empty[xs]);
            }
            __syncwarp();
            acc = 1u;
            x_desc += (uint64_t)(x_stage_bytes >> 4);
            if (++xs == x_stages) {
              xs = 0;
              xph ^= 1u;
              x_desc = x_desc0;
            }
          }
          if (!ok) break;
          if (leader) tc_commit(&a_empty[ab]);
          __syncwarp();
          if (++ab == pp.na) {
            ab = 0;
            aph ^= 1u;
          }
        }
      }
      if (ok && leader) tc_commit(&d_full[db]);
      __syncwarp();
      if (++db == pp.nd) {
        db = 0;
        dph ^= 1u;
      }
    }
  } else if (warp == 2) {
    // ============================================================ x tiles (TMA)
    if (!grouped) griddep_wait();
    int xs = 0;
    uint32_t ph = 1;
    Walk w;
    bool ok = true;
    for (bool have = begin(w); ok && have; have = next(w)) {
      const int m0 = get_item(w.item).m0;
      const int kb_end = min(w.c1 * kBlkPerChunk, p.k / kKBlock);
      for (int kb = w.c0 * kBlkPerChunk; kb < kb_end; ++kb) {
        if (!mbar_wait_parked(&x_empty[xs], ph, p.status)) {
          ok = false;
          break;
        }
        if (lane == 0) {
          mbar_arrive_expect_tx(&x_full[xs], (uint32_t)x_stage_bytes);
          tma_load_x(x_ring + (size_t)xs * x_stage_bytes, &tmap_x, kb * kKBlock, m0, &x_full[xs]);
        }
        __syncwarp();
        if (++xs == x_stages) {
          xs = 0;
          ph ^= 1u;
        }
      }
    }
  } else if (warp >= 4) {
    // ============================================================ decode + epilogue warps
    const int grp = (warp - 4) >> 2, w4 = warp & 3;
    const int hi = w4 & 1;
    const int bl = (w4 >> 1) * 4 + (lane >> 3), g = lane & 7;
    const int row = 16 * bl + g + 8 * hi;      // weight row held by this thread's TMEM lane
    const int gj = w4 * 32 + lane;             // thread index inside the group = TMEM lane
    const uint32_t lane_taddr = (uint32_t)(32 * w4) << 16;
    const ZeroConsts zc = make_zero_consts(ZMODE, p.zero_const);
    uint32_t off[4];
#pragma unroll
    for (int t = 0; t < 4; ++t) off[t] = (uint32_t)(t * 128 + ((g + 2 * t) & 7) * 16);
    if (!grouped && !pp.early) griddep_wait();  // scales may be the previous kernel's output
    bool waited = grouped || !pp.early;

    const int k_blocks = p.k / kKBlock;
    ScaleFeed<BITS, ZMODE, SRC, kOwn, BITS == 8> feed;
    feed.init(pp, hi);
    auto fetch = [&](int c) {
      const int kb = c * kBlkPerChunk + grp * kOwn;
      if (kOwn == 2) feed.fetch_two(pp, kb, k_blocks);
      else feed.fetch(pp, 0, min(kb, k_blocks - 1));
    };

    bool ok = true;
    uint32_t e_phase = 0;
    auto group_sync = [&]() -> bool {  // the four warps of this group (bounded, unlike a named barrier)
      __syncwarp();
      if (lane == 0) mbar_arrive(&e_bar[grp]);
      const bool fine = mbar_wait_parked(&e_bar[grp], e_phase, p.status);
      e_phase ^= 1u;
      return fine;
    };

    int ws = 0, ab0 = 0, db = 0;
    uint32_t wph = 0, aph0 = 1, dph = 0;
    unsigned step = 0;
    Walk w;
    for (bool have = begin(w); ok && have; have = next(w)) {
      const Item it = get_item(w.item);
      feed.row(pp, it.e, it.n_tile * kTileRows + row);
      fetch(w.c0);
      for (int c = w.c0; c < w.c1; ++c) {
        feed.advance();
        if (c + 1 < w.c1) fetch(c + 1);
        if (!mbar_wait_parked(&w_full[ws], wph, p.status)) {
          ok = false;
          break;
        }
        const int nft = min(4, KT - c * 4), nblk = nft / kTilesPerBlk;
        const uint8_t* blk0 = w_ring + (size_t)ws * kWBytes + bl * (nft * 512);
        const int first = grp * kOwn;
        if (first < nblk) {
          int ab = ab0 + first / kOwn;
          uint32_t aph = aph0;
          if (ab >= pp.na) {
            ab -= pp.na;
            aph ^= 1u;
          }
          const uint32_t a_taddr = lane_taddr | (tmem + (uint32_t)(pp.a_base + ab * (kOwn * 32)));
          ok = mbar_wait_parked(&a_empty[ab], aph, p.status);
          if (!ok) break;
          tc_fence_after();
#pragma unroll
          for (int i = 0; i < kOwn; ++i) {
            const int b = first + i;
            if (i > 0 && b >= nblk) break;
            decode_own<BITS, ZMODE, SRC>(pp, feed, i, c * kBlkPerChunk + b, blk0 + b * (kTilesPerBlk * 512), off, zc,
                                    a_taddr + (uint32_t)(i * 32));
          }
          tc_wait_st();
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(&a_full[ab]);
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(&w_empty[ws]);
        if (++ws == w_stages) {
          ws = 0;
          wph ^= 1u;
        }
        ab0 += (nblk + kOwn - 1) / kOwn;
        if (ab0 >= pp.na) {
          ab0 -= pp.na;
          aph0 ^= 1u;
        }
      }
      if (!ok) break;
      // ---------------------------------------------------------- this piece's accumulator
      if (!mbar_wait_parked(&d_full[db], dph, p.status)) {
        ok = false;
        break;
      }
      tc_fence_after();
      if (kExchange) {
        if (folds<ZMODE, SRC>()) reinterpret_cast<float*>(e_stage)[gj] = drain_scale<BITS>(feed.s_row, hi);  // (both groups the same)
        break;
      }
      if (!waited) {
        griddep_wait();  // outputs and scratch may be in use by the previous kernel until it has ended
        waited = true;
      }
      const DrainTile dt = {lane_taddr | (tmem + (uint32_t)(db * pp.d_stride)), grp * 16, kGroups * 16, min(nb, it.m_end - it.m0),
                            it.n_tile * kTileRows, it.m0, it.m_end, row, gj,
                            folds<ZMODE, SRC>() ? drain_scale<BITS>(feed.s_row, hi) : 1.0f};
      const int me = (int)blockIdx.x;
      if (w.c0 > 0) {
        drain_publish(pp, dt, me);
      } else {
        int last = me;
        if (w.c1 < cpt) {
          // this CTA owns the tile, later ones hold the rest
          const unsigned hi_u = (unsigned)w.item * (unsigned)cpt + (unsigned)cpt - 1u;
          if constexpr (SPLIT == kWholeFirst) last = (int)(whole + ((hi_u - base + 1u) * takers - 1u) / rest);
          else last = (int)(((hi_u + 1u) * ctas - 1u) / total);
        }
        ok = drain_store<false, folds<ZMODE, SRC>()>(pp, dt, me, last, 1, e_stage + grp * kStageBytes, step, group_sync);
        if (!ok) break;
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&d_empty[db]);
      if (++db == pp.nd) {
        db = 0;
        dph ^= 1u;
      }
    }
    fine = ok;
  }

  if (kExchange) {
    const int grp = (warp - 4) >> 2, w4 = warp & 3, ranks = (int)cluster_nctarank(), rank = (int)blockIdx.x % ranks;
    const Item it = get_item((int)blockIdx.x / ranks);
    const int cols = min(nb, it.m_end - it.m0);
    cluster_sync();  // no CTA reads its ring of weights any more
    if (warp >= 4) {
      // After a wait that ran out bulk copies may still be on their way into a ring: the cluster's CTAs leave the tile unwritten.
      // (Told before the first barrier, which takes one more for the flags to be at rest, it cost 3 to 6 % at 256 CTAs.)
      if (!__all_sync(0xffffffffu, fine) && lane < ranks)
        asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(map_to(smem_u32(tmem_holder + 1), lane)), "r"(1u) : "memory");
      exchange_send(smem_u32(w_ring), ((uint32_t)(32 * w4) << 16) | tmem, cols, rank, ranks, grp, w4 * 32 + lane);
      tc_fence_before();
      if (pp.early) griddep_wait();  // outputs may be in use by the previous kernel until it has ended
    }
    cluster_sync();
    if (warp >= 4 && *gave_up == 0u)
      exchange_store<folds<ZMODE, SRC>()>(pp, reinterpret_cast<const float*>(w_ring), reinterpret_cast<const float*>(e_stage),
                                          it.n_tile * kTileRows, it.m0, cols, rank, ranks, grp, w4 * 32 + lane);
  }
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    ug::tmem_dealloc(tmem, (uint32_t)pp.tmem_cols);
  }
}

template <int BITS, int ZMODE, int SRC, int SPLIT>
int launch_split(const Params& pp, const Launch& l, const CUtensorMap& tx, cudaStream_t stream) {
  auto kern = umma_sk_kernel<BITS, ZMODE, SRC, SPLIT>;
  static thread_local int configured_device = -1;
  int dev = 0;
  RB200_CUDA(cudaGetDevice(&dev));
  if (configured_device != dev) {
    RB200_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024));
    configured_device = dev;
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)l.grid, 1, 1);
  cfg.blockDim = dim3((4 + 4 * kGroups) * 32, 1, 1);
  cfg.dynamicSmemBytes = l.smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  if (SPLIT == kCluster) {
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = (unsigned)l.ranges;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    cfg.numAttrs = 1;
  }
  // always a programmatic dependent: before its wait the kernel only prefetches, unless the host
  // switched launch overlap on
  attr[cfg.numAttrs].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[cfg.numAttrs].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  ++cfg.numAttrs;
  RB200_CUDA(cudaLaunchKernelEx(&cfg, kern, pp, tx));
  return 0;
}
template <int BITS, int ZMODE, int SRC>
int launch_inst(const Params& pp, const Launch& l, const CUtensorMap& tx, cudaStream_t stream) {
  if (l.ranges > 1) return launch_split<BITS, ZMODE, SRC, kCluster>(pp, l, tx, stream);
  if (pp.whole) return launch_split<BITS, ZMODE, SRC, kWholeFirst>(pp, l, tx, stream);
  return launch_split<BITS, ZMODE, SRC, kRuns>(pp, l, tx, stream);
}

template <int BITS, int ZMODE>
int launch_src(const Params& pp, const Launch& l, const CUtensorMap& tx, cudaStream_t stream) {
  switch (l.src) {
    case kChannel: return launch_inst<BITS, ZMODE, kChannel>(pp, l, tx, stream);
    case kOne: return launch_inst<BITS, ZMODE, kOne>(pp, l, tx, stream);
    case kTwo: return launch_inst<BITS, ZMODE, kTwo>(pp, l, tx, stream);
    default: return launch_inst<BITS, ZMODE, kAny>(pp, l, tx, stream);
  }
}
template <int BITS>
int launch_bits(const Params& pp, const Launch& l, const CUtensorMap& tx, cudaStream_t stream) {
  return l.zmode == kZeroGeneral ? launch_src<BITS, kZeroGeneral>(pp, l, tx, stream)
                                 : launch_src<BITS, kZeroConstInt>(pp, l, tx, stream);
}

#endif  // __CUDACC__

}  // namespace us

}  // namespace rb200
