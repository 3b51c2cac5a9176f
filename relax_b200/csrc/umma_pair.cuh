// Large batches (more than 64 rows, expert layers included) over packed weights: CTA pairs on the
// 5th-generation tensor cores.
//
//   out^T tile [256 weight rows x nb batch rows] = W_tile [256 x K] * x_tile^T [K x nb]
//
// Bound: the tensor pipe (and the 1000 W power cap behind it).  One CTA per 128-row tile had to stream
// nb x 128 bytes of x per 64-k block through its own L2 port: at nb = 256 that is 32 KB per 512 clocks of
// MMA, the port's whole 64 bytes per clock.  Here the two CTAs of a pair (tcgen05 cta_group::2, M = 256)
// hold half of the x tile each and the tensor cores read both halves: 16 KB per CTA and block.
//
//   every CTA decodes its own 128 weight rows straight into its tensor memory (A, thread = weight row);
//   rank 0 issues the MMAs of the pair and commits to both CTAs' barriers;
//   everything is handed over in steps of two 64-k blocks: with one block a step the barriers, commits and
//   tensor-memory store waits of a step took longer than its MMAs (int8, m 256, k 8192 x n 57344: 191 us
//   without any arithmetic, 118 us without arithmetic, stores and three of the four MMAs);
//   accumulators: two of up to 160 columns, so that one drains while the next tile runs, or one of up to 256.
//
//   warp 0        packed weights, one 16 KB bulk copy per chunk (128 rows x 256 | 128 k)
//   warp 1        MMA issue (rank 0)
//   warp 2        x: one TMA tile [nb/2 rows x 128 k] per step, completing on rank 0's barrier
//   warps 4-15    three groups of four warps.  With two accumulators two of them decode alternate steps and
//                 the third drains: epilogue, one rounding, transpose through shared memory, whole-line
//                 stores (the others help it with the last tile).  With a single accumulator there is nothing
//                 to drain while a tile is made: all three decode in turn and then drain in shares, up to a tile
//                 of 192 rows.  Above, a block's MMAs take longer than two groups take to decode it, and a third
//                 only gets in their way (int8 per row, k 4096 x n 22016, 256 rows 53.7 us with three, 52.1 with
//                 two; int4 group 32 47.9 / 46.6, group 64 with zero points 51.6 / 50.4).  At 192 and fewer three
//                 are ahead by up to 3 % (int8 per row, k 28672 x n 8192, 192 rows 110.3 us with two, 108.3 with
//                 three), and an expert layer's tiles, whose MMAs are narrower than the tile, gain most.
//
// Work split: whole waves of tiles go round robin over the pairs, neighbours sharing a weight tile in L2;
// the remainder - between one and two waves - is cut into equal runs of (tile, chunk) units that the
// pairs do first (stream-k), handing partial accumulators over as in umma_sk.cuh.  So no wave is partly
// empty, and the hand-over hides behind the whole tiles.
// Every wait is bounded and reports through the device status word.
//
// Stands in for fastertransformer::gemm_fp16_int_bias_act[_residual] at large m
// (python/tvm/contrib/cutlass/gemm_operation.py:441-458), the reference's tensor-core matmul schedule
// (python/tvm/dlight/gpu/matmul.py:316-535) and, grouped, the expert form of
// src/runtime/contrib/cutlass/fp16_group_gemm.cu:39-64 over quantised weights.
#pragma once

#include "umma_tile.cuh"

namespace rb200 {
namespace up {

using namespace us;

constexpr int kThreads = 16 * 32;
constexpr int kDrainGroups = 3;

inline size_t smem_bytes(int nb, int x_stages, int w_stages) {
  return 1024 + (size_t)x_stages * nb * 128 + (size_t)w_stages * kWBytes + kDrainGroups * kStageBytes +
         (size_t)(4 * kMaxStages + 2 * kMaxA + 5 + kDrainGroups) * 8 + 16 + (3 * kMaxExperts + 4) * sizeof(int);
}

struct Launch {
  int zmode, src;
  long long most_pairs;  // pairs the problem can use
  size_t smem;
};
int launch_i4(const Params& pp, const Launch& l, const CUtensorMap& tx, cudaStream_t stream);
int launch_i8(const Params& pp, const Launch& l, const CUtensorMap& tx, cudaStream_t stream);

#ifdef __CUDACC__

// ---------------------------------------------------------------- pair forms of the PTX wrappers
__device__ __forceinline__ uint32_t cluster_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ uint32_t at_rank0(const void* p) {  // the same shared-memory object in rank 0
  uint32_t a;
  asm volatile("mapa.shared::cluster.u32 %0, %1, 0;" : "=r"(a) : "r"(smem_u32(p)));
  return a;
}
// What these barriers order is tensor memory (through the tcgen05 fences) and TMA data, never generic
// writes, so the default scope does: an acquire of cluster scope drops the L1 cache, which holds the
// scales, on every wait (1300 instead of 400 clocks per 64-k block).
__device__ __forceinline__ void arrive_cluster(uint32_t bar) {
  asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(bar) : "memory");
}
// x tile of this CTA's half (64-k blocks kb, kb + 1; a block past k reads as zero), completion counted on rank 0's barrier
__device__ __forceinline__ void tma_load_half(void* smem_dst, const CUtensorMap* map, int row, int kb, uint32_t bar0) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes.cta_group::2 [%0], [%1, {%2, %3, %4}], "
      "[%5];" ::"r"(smem_u32(smem_dst)),
      "l"(map), "r"(0), "r"(row), "r"(kb), "r"(bar0)
      : "memory");
}
__device__ __forceinline__ void tmem_alloc2(uint32_t* smem_holder, uint32_t cols) {
  asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(smem_holder)), "r"(cols) : "memory");
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc2(uint32_t taddr, uint32_t cols) {
  asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(cols) : "memory");
}
__device__ __forceinline__ void mma_ts2(uint32_t d, uint32_t a, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], [%1], %2, %3, p;\n\t}" ::"r"(d),
      "r"(a), "l"(b_desc), "r"(idesc), "r"(accumulate)
      : "memory");
}
__device__ __forceinline__ void commit2(uint64_t* bar) {  // arrives at both CTAs' barrier
  asm volatile(
      "tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(smem_u32(bar)),
      "h"((uint16_t)3)
      : "memory");
}

template <int BITS, int ZMODE, int SRC>
__global__ void __launch_bounds__(kThreads, 1)
    umma_pair_kernel(const Params pp, const __grid_constant__ CUtensorMap tmap_x) {
  constexpr int kBlkPerChunk = BITS == 8 ? 2 : 4;  // 64-k blocks per weight stage
  constexpr int kTilesPerBlk = BITS == 8 ? 2 : 1;
  constexpr int kFragK = BITS == 8 ? 32 : 64;
  constexpr int kStepBlk = 2;                      // blocks of a step
  extern __shared__ uint8_t smem_raw[];
  const GemvParams& p = pp.g;
  uint8_t* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
  const int nb = pp.nb, x_stages = pp.x_stages, w_stages = pp.w_stages;
  const int x_block_bytes = (nb / 2) * 128, x_stage_bytes = kStepBlk * x_block_bytes;
  uint8_t* x_ring = smem;
  uint8_t* w_ring = x_ring + (size_t)x_stages * x_stage_bytes;
  uint8_t* e_stage = w_ring + (size_t)w_stages * kWBytes;
  uint64_t* w_full = reinterpret_cast<uint64_t*>(e_stage + kDrainGroups * kStageBytes);
  uint64_t* w_empty = w_full + kMaxStages;
  uint64_t* x_full = w_empty + kMaxStages;   // rank 0's are used
  uint64_t* x_empty = x_full + kMaxStages;
  uint64_t* a_full = x_empty + kMaxStages;   // rank 0's are used
  uint64_t* a_empty = a_full + kMaxA;
  uint64_t* d_full = a_empty + kMaxA;
  uint64_t* d_empty = d_full + 2;            // rank 0's are used
  uint64_t* d_last = d_empty + 2;            // the last accumulator, for the helping groups
  uint64_t* e_bar = d_last + 1;
  uint32_t* tmem_holder = reinterpret_cast<uint32_t*>(e_bar + kDrainGroups);
  Tables& tt = *reinterpret_cast<Tables*>(tmem_holder + 4);

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const uint32_t rank = cluster_rank();
  const unsigned pair = blockIdx.x >> 1, pairs = gridDim.x >> 1;
  const bool grouped = pp.indptr != nullptr;
  const bool all_drain = pp.nd == 1;  // nothing to drain while a tile is made
  // groups that decode (na >= 3 A slots: with fewer, three would meet in a slot's phase)
  const int decoders = all_drain && nb <= 192 ? 3 : 2;
  if (tid == 0) {
    for (int s = 0; s < w_stages; ++s) {
      mbar_init(&w_full[s], 1);
      mbar_init(&w_empty[s], 4 * decoders);
    }
    for (int s = 0; s < x_stages; ++s) {
      mbar_init(&x_full[s], 1);
      mbar_init(&x_empty[s], 1);
    }
    for (int i = 0; i < pp.na; ++i) {
      mbar_init(&a_full[i], 8);  // a group's four warps, in both CTAs
      mbar_init(&a_empty[i], 1);
    }
    for (int i = 0; i < pp.nd; ++i) {
      mbar_init(&d_full[i], 1);
      mbar_init(&d_empty[i], all_drain ? 24 : 8);
    }
    mbar_init(d_last, 1);
    for (int i = 0; i < kDrainGroups; ++i) mbar_init(&e_bar[i], 4);
    mbar_fence_init();
  }
  if (warp == 1) tmem_alloc2(tmem_holder, (uint32_t)pp.tmem_cols);
  const int n_tiles = (p.n + 2 * kTileRows - 1) / (2 * kTileRows);
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
  cluster_sync();  // both CTAs' barriers exist before any remote arrival
  tc_fence_after();
  // only now, with this pair's tensor memory in hand: a dependent CTA that took it first would hold it
  // until this grid has ended
  griddep_launch_dependents();
  const uint32_t tmem = *tmem_holder;

  const int NB = p.n / 16, KT = p.k / kFragK, cpt = pp.cpt, k_blocks = p.k / kKBlock;
  const unsigned items = grouped ? (unsigned)tt.base[pp.num_experts] : (unsigned)(n_tiles * pp.m_tiles);
  // the first `split` items are shared out in equal runs of chunks, the others in whole waves
  const unsigned waves = items / pairs, rem = items - waves * pairs;
  // (none of them where there are no words to hand over a part of a tile)
  const unsigned split = rem == 0 || !pp.partial ? 0u : (waves >= 1 ? pairs + rem : rem);
  const unsigned total = split * (unsigned)cpt;
  const unsigned takers = min(pairs, total);  // pairs with a run
  const unsigned u_begin = pair < takers ? (unsigned)((unsigned long long)pair * total / takers) : 0u;
  const unsigned u_end = pair < takers ? (unsigned)((unsigned long long)(pair + 1) * total / takers) : 0u;

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
    it.n_tile = 2 * it.n_tile + (int)rank;  // this CTA's 128-row tile
    return it;
  };
  // MMA width of an item: its batch rows, not the tile's width (an expert's share of the rows is usually
  // well below the width that leaves room for an uneven routing, and padding costs as much power as work)
  auto width_of = [&](const Item& it) { return max(32, min(nb, (it.m_end - it.m0 + 31) / 32 * 32)); };
  // The pair's pieces in order: item, chunks [c0, c1); whole items from `split` on.
  struct Walk {
    unsigned u;
    int item, c0, c1;
  };
  auto whole = [&](Walk& w, unsigned item) {
    w.u = u_end;
    w.item = (int)item;
    w.c0 = 0;
    w.c1 = cpt;
    return item < items;
  };
  auto begin = [&](Walk& w) {
    w.u = u_begin;
    if (u_begin >= u_end) return whole(w, split + pair);
    w.item = (int)(u_begin / (unsigned)cpt);
    w.c0 = (int)(u_begin - (unsigned)w.item * (unsigned)cpt);
    w.c1 = min(cpt, w.c0 + (int)(u_end - u_begin));
    return true;
  };
  auto next = [&](Walk& w) {
    if (w.u >= u_end) return whole(w, (unsigned)w.item + pairs);
    w.u += (unsigned)(w.c1 - w.c0);
    if (w.u >= u_end) return whole(w, split + pair);
    ++w.item;
    w.c0 = 0;
    w.c1 = min(cpt, (int)(u_end - w.u));
    return true;
  };
  auto is_last = [&](Walk w) { return !next(w); };
  // 64-k blocks of chunk c, bytes of it in this CTA's 128-row tile
  auto blocks_of = [&](int c) { return min(4, KT - c * 4) / kTilesPerBlk; };

  if (warp == 0) {
    // ============================================================ producer: packed weights
    Walk w;
    bool have = begin(w), ok = true;
    auto bytes_of = [&](const Item& it, int c) { return (uint32_t)(min(4, KT - c * 4) * max(0, min(8, NB - it.n_tile * 8))) * 512u; };
    if (have && !pp.early && !grouped) {
      // only into L2 before the wait: a prefetch returns nothing to this kernel, so it is safe
      // whatever the previous one still writes
      const Item it = get_item(w.item);
      if (lane == 0)
        for (int c = w.c0; c < min(w.c1, w.c0 + w_stages); ++c)
          if (bytes_of(it, c))
            asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(p.w + frag_stage_offset(it.n_tile, c, NB, KT)),
                         "r"(bytes_of(it, c))
                         : "memory");
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
          const uint32_t bytes = bytes_of(it, c);
          if (bytes) {
            mbar_arrive_expect_tx(&w_full[ws], bytes);
            bulk_g2s(w_ring + (size_t)ws * kWBytes, w_e + frag_stage_offset(it.n_tile, c, NB, KT), bytes, &w_full[ws]);
          } else {
            mbar_arrive(&w_full[ws]);  // a tile past the last row: decoded from stale bytes, never stored
          }
        }
        __syncwarp();
        if (++ws == w_stages) {
          ws = 0;
          ph ^= 1u;
        }
      }
    }
  } else if (warp == 1) {
    // ============================================================ MMA issue (rank 0, elected thread)
    if (rank == 0) {
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
        const uint32_t idesc = (1u << 4) | ((uint32_t)(width_of(get_item(w.item)) >> 3) << 17) | ((uint32_t)(256 >> 4) << 24);
        uint32_t acc = 0u;
        for (int c = w.c0; c < w.c1 && ok; ++c) {
          const int nblk = blocks_of(c);
          for (int b0 = 0; b0 < nblk; b0 += kStepBlk) {
            if (!mbar_wait_parked(&x_full[xs], xph, p.status) || !mbar_wait_parked(&a_full[ab], aph, p.status)) {
              ok = false;
              break;
            }
            tc_fence_after();
            const uint32_t a = tmem + (uint32_t)(pp.a_base + ab * (kStepBlk * 32));
            if (leader) {
              mma_ts2(d, a, x_desc, idesc, acc);
#pragma unroll
              for (int j = 1; j < 4; ++j) mma_ts2(d, a + j * 8, x_desc + j * 2, idesc, 1u);
              if (b0 + 1 < nblk) {
                const uint64_t x_desc1 = x_desc + (uint64_t)(x_block_bytes >> 4);
#pragma unroll
                for (int j = 0; j < 4; ++j) mma_ts2(d, a + 32 + j * 8, x_desc1 + j * 2, idesc, 1u);
              }
              commit2(&a_empty[ab]);
              commit2(&x_empty[xs]);
            }
            __syncwarp();
            acc = 1u;
            x_desc += (uint64_t)(x_stage_bytes >> 4);
            if (++xs == x_stages) {
              xs = 0;
              xph ^= 1u;
              x_desc = x_desc0;
            }
            if (++ab == pp.na) {
              ab = 0;
              aph ^= 1u;
            }
          }
        }
        if (ok && leader) {
          commit2(&d_full[db]);
          if (!all_drain && is_last(w)) commit2(d_last);
        }
        __syncwarp();
        if (++db == pp.nd) {
          db = 0;
          dph ^= 1u;
        }
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
      const Item it = get_item(w.item);
      const int m0 = it.m0 + (int)rank * (width_of(it) / 2);
      const int kb_end = min(w.c1 * kBlkPerChunk, k_blocks);
      for (int kb = w.c0 * kBlkPerChunk; kb < kb_end; kb += kStepBlk) {
        if (!mbar_wait_parked(&x_empty[xs], ph, p.status)) {
          ok = false;
          break;
        }
        if (lane == 0) {
          if (rank == 0) mbar_arrive_expect_tx(&x_full[xs], (uint32_t)x_stage_bytes * 2u);
          tma_load_half(x_ring + (size_t)xs * x_stage_bytes, &tmap_x, m0, kb, at_rank0(&x_full[xs]));
        }
        __syncwarp();
        if (++xs == x_stages) {
          xs = 0;
          ph ^= 1u;
        }
      }
    }
    // every commit to this CTA's barriers has arrived before it may leave
    for (int i = 0; ok && i < x_stages; ++i) {
      ok = mbar_wait_parked(&x_empty[xs], ph, p.status);
      if (++xs == x_stages) {
        xs = 0;
        ph ^= 1u;
      }
    }
  } else if (warp >= 4) {
    // ============================================================ decode (groups 0, 1 or all three) and drain
    const int grp = (warp - 4) >> 2, w4 = warp & 3;
    const int hi = w4 & 1;
    const int bl = (w4 >> 1) * 4 + (lane >> 3), g = lane & 7;
    const int row = 16 * bl + g + 8 * hi;  // weight row held by this thread's TMEM lane
    const int gj = w4 * 32 + lane;         // thread index inside the group = TMEM lane
    const uint32_t lane_taddr = (uint32_t)(32 * w4) << 16;
    if (!grouped && !pp.early) griddep_wait();  // scales may be the previous kernel's output
    bool waited = grouped || !pp.early;

    bool ok = true;
    uint32_t e_phase = 0;
    unsigned parity = 0;
    auto group_sync = [&]() -> bool {  // the four warps of this group (bounded, unlike a named barrier)
      __syncwarp();
      if (lane == 0) mbar_arrive(&e_bar[grp]);
      const bool fine = mbar_wait_parked(&e_bar[grp], e_phase, p.status);
      e_phase ^= 1u;
      return fine;
    };
    // this group's share of a finished accumulator
    auto drain = [&](const Walk& w, const Item& it, int db, int share, int shares, uint32_t s_row) -> bool {
      if (!waited) {
        griddep_wait();  // outputs and scratch may be in use by the previous kernel until it has ended
        waited = true;
      }
      if (it.n_tile * kTileRows >= p.n) return true;
      const DrainTile dt = {lane_taddr | (tmem + (uint32_t)(db * pp.d_stride)), share * 16, shares * 16, min(nb, it.m_end - it.m0),
                            it.n_tile * kTileRows, it.m0, it.m_end, row, gj, folds<ZMODE, SRC>() ? drain_scale<BITS>(s_row, hi) : 1.0f};
      const int me = (int)blockIdx.x;
      if (w.c0 > 0) {
        drain_publish(pp, dt, me);
        return true;
      }
      int last = me;
      if (w.c1 < cpt) {
        // this pair owns the tile, later ones hold the rest
        const unsigned hi_u = (unsigned)w.item * (unsigned)cpt + (unsigned)cpt - 1u;
        last = 2 * (int)((((unsigned long long)hi_u + 1u) * takers - 1u) / total) + (int)rank;
      }
      return drain_store<true, folds<ZMODE, SRC>()>(pp, dt, me, last, 2, e_stage + grp * kStageBytes, parity, group_sync);
    };

    ScaleFeed<BITS, ZMODE, SRC, kStepBlk, true> feed;
    feed.init(pp, hi);
    int db = 0;
    uint32_t dph = 0;
    Walk w;
    if (grp >= decoders) {
      for (bool have = begin(w); ok && have; have = next(w)) {
        const Item it = get_item(w.item);
        feed.row(pp, it.e, it.n_tile * kTileRows + row);
        ok = mbar_wait_parked(&d_full[db], dph, p.status);
        if (!ok) break;
        tc_fence_after();
        ok = drain(w, it, db, 0, all_drain || is_last(w) ? kDrainGroups : 1, feed.s_row);
        if (!ok) break;
        tc_fence_before();
        __syncwarp();
        if (lane == 0) arrive_cluster(at_rank0(&d_empty[db]));
        if (++db == pp.nd) {
          db = 0;
          dph ^= 1u;
        }
      }
    } else {
      const ZeroConsts zc = make_zero_consts(ZMODE, p.zero_const);
      uint32_t off[4];
#pragma unroll
      for (int t = 0; t < 4; ++t) off[t] = (uint32_t)(t * 128 + ((g + 2 * t) & 7) * 16);
      int own = grp;  // the groups take the steps in turn: this group's next one, counted from the current chunk's first
      auto fetch = [&](int c, int own) {
        // (on every path, a group without a step in the chunk too: a load under a branch is waited for where the paths meet)
        const int j = min(own, kBlkPerChunk / kStepBlk - 1);
        feed.fetch_two(pp, min(c * kBlkPerChunk + j * kStepBlk, (k_blocks - 1) & ~1), k_blocks);
      };
      int ws = 0, ab0 = 0;
      uint32_t wph = 0, aph0 = 1;
      for (bool have = begin(w); ok && have; have = next(w)) {
        const Item it = get_item(w.item);
        feed.row(pp, it.e, it.n_tile * kTileRows + row);
        fetch(w.c0, own);
        for (int c = w.c0; c < w.c1; ++c) {
          const int nft = min(4, KT - c * 4), nblk = nft / kTilesPerBlk, steps = (nblk + kStepBlk - 1) / kStepBlk;
          const int j = own;
          feed.advance();
          own -= steps;
          if (own < 0) own += decoders;
          fetch(min(c + 1, w.c1 - 1), own);
          // (a group without a step in this chunk waits all the same: its arrival must not run ahead)
          if (!mbar_wait_parked(&w_full[ws], wph, p.status)) {
            ok = false;
            break;
          }
          if (j < steps) {
            int ab = ab0 + j;
            uint32_t aph = aph0;
            if (ab >= pp.na) {
              ab -= pp.na;
              aph ^= 1u;
            }
            const uint8_t* blk = w_ring + (size_t)ws * kWBytes + bl * (nft * 512) + j * (kStepBlk * kTilesPerBlk * 512);
            const int kb = c * kBlkPerChunk + j * kStepBlk;
            const uint32_t a_taddr = lane_taddr | (tmem + (uint32_t)(pp.a_base + ab * (kStepBlk * 32)));
            ok = mbar_wait_parked(&a_empty[ab], aph, p.status);
            if (!ok) break;
            tc_fence_after();
#pragma unroll
            for (int i = 0; i < kStepBlk; ++i) {
              if (i > 0 && j * kStepBlk + i >= nblk) break;
              decode_own<BITS, ZMODE, SRC>(pp, feed, i, kb + i, blk + i * (kTilesPerBlk * 512), off, zc, a_taddr + (uint32_t)(i * 32));
            }
            tc_wait_st();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) arrive_cluster(at_rank0(&a_full[ab]));
          }
          __syncwarp();
          if (lane == 0) mbar_arrive(&w_empty[ws]);
          if (++ws == w_stages) {
            ws = 0;
            wph ^= 1u;
          }
          ab0 += steps;
          if (ab0 >= pp.na) {
            ab0 -= pp.na;
            aph0 ^= 1u;
          }
        }
        if (!ok) break;
        const bool last = is_last(w);
        if (all_drain || last) {
          ok = all_drain ? mbar_wait_parked(&d_full[db], dph, p.status) : mbar_wait_parked(d_last, 0, p.status);
          if (!ok) break;
          tc_fence_after();
          ok = drain(w, it, db, grp == 2 ? 0 : grp + 1, kDrainGroups, feed.s_row);
          if (!ok) break;
          tc_fence_before();
          __syncwarp();
          if (all_drain && lane == 0) arrive_cluster(at_rank0(&d_empty[db]));
        }
        if (++db == pp.nd) {
          db = 0;
          dph ^= 1u;
        }
      }
      // every commit to this CTA's barriers has arrived before it may leave
      for (int i = 0; ok && i < pp.na; ++i) {
        ok = mbar_wait_parked(&a_empty[ab0], aph0, p.status);
        if (++ab0 == pp.na) {
          ab0 = 0;
          aph0 ^= 1u;
        }
      }
    }
  }

  tc_fence_before();
  __syncthreads();
  cluster_sync();  // the other CTA may still have been reading this one's x tiles, or arriving here
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc2(tmem, (uint32_t)pp.tmem_cols);
  }
}

template <int BITS, int ZMODE, int SRC>
int launch_inst(const Params& pp, const Launch& l, const CUtensorMap& tx, cudaStream_t stream) {
  auto kern = umma_pair_kernel<BITS, ZMODE, SRC>;
  static thread_local int configured_device = -1, pairs_fit = 0;
  int dev = 0;
  RB200_CUDA(cudaGetDevice(&dev));
  cudaLaunchConfig_t cfg = {};
  cfg.blockDim = dim3(kThreads, 1, 1);
  cfg.dynamicSmemBytes = l.smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 2;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  if (configured_device != dev) {
    RB200_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024));
    // pairs that wait on one another have to be resident together
    cfg.gridDim = dim3((unsigned)sm_count_current() / 2 * 2, 1, 1);
    cfg.dynamicSmemBytes = 227 * 1024;
    RB200_CUDA(cudaOccupancyMaxActiveClusters(&pairs_fit, kern, &cfg));
    cfg.dynamicSmemBytes = l.smem;
    RB200_CHECK(pairs_fit >= 1, "no CTA pair fits the device");
    configured_device = dev;
  }
  long long pairs = l.most_pairs < pairs_fit ? l.most_pairs : pairs_fit;
  cfg.gridDim = dim3((unsigned)pairs * 2, 1, 1);
  // always a programmatic dependent: before its wait the kernel only prefetches, unless the host
  // switched launch overlap on
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.numAttrs = 2;
  RB200_CUDA(cudaLaunchKernelEx(&cfg, kern, pp, tx));
  return 0;
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

}  // namespace up
}  // namespace rb200
