// Medium batches (9 to 256 rows, and expert layers above the decode size) on the 5th-generation
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
//
//   warp 0  packed weights, one 16 KB bulk copy per chunk (128 rows x 256 | 128 k)
//   warp 1  MMA: four per 64-k block, by an elected thread
//   warp 2  x: one TMA tile [nb rows x 64 k] per block, 128-byte swizzle = K-major operand
//   warps 4 .. 4 + 4G - 1: G groups of four warps decode a share of each chunk's blocks, then drain the
//           accumulator, G x 16 batch columns at a time: bias / activation / residual, one rounding,
//           transpose through shared memory, whole-line stores.
//   G = 2, at most 64 batch rows: 256 TMEM columns and half the shared memory, so two CTAs share an SM
//           and one's decode covers the other's waits; G = 4 above that, one CTA per SM.
// Every wait is bounded and reports through the device status word.
//
// Stands in for fastertransformer::gemm_fp16_int_bias_act[_residual]
// (python/tvm/contrib/cutlass/gemm_operation.py:441-458) and, grouped, for the expert form of
// src/runtime/contrib/cutlass/fp16_group_gemm.cu:39-64 over quantised weights.
#pragma once

#include <cuda.h>

#include "dequant.cuh"
#include "gemv.h"
#include "umma_common.cuh"

namespace rb200 {
namespace us {

constexpr int kTileRows = 128;
constexpr int kKBlock = 64;
constexpr int kWBytes = 8 * 4 * 512;
constexpr int kMaxExperts = 64;
constexpr int kMaxStages = 8;
constexpr int kMaxA = 8;
constexpr uint32_t kVacant = 0xffffffffu;  // a NaN; sums that are NaN are published as 0x7fffffff
constexpr int kMaxNb = 256;
constexpr int kSmallNb = 64;            // up to here two CTAs share an SM
constexpr int kStageBytes = 16 * kTileRows * 4;  // per group: two 16 x 128 fp16 buffers, or one fp32
constexpr int kMaxGroups = 4;

enum ScaleSrc : int {
  kChannel = 0,  // one per row
  kOne = 1,      // groups of whole 64-k blocks
  kTwo = 2,      // group 32
  kAny = 3,      // any other group size
};

struct Params {
  GemvParams g;
  int nb, m_tiles;             // batch rows per tile (multiple of 16), batch tiles (ungrouped)
  int cpt;                     // chunks per tile
  int x_stages, w_stages;
  int nd, d_stride, a_base, na, tmem_cols;  // accumulators and A slots in tensor memory
  int s_n, s_g;                // scale strides in elements
  int s_vec;                   // kTwo: the two groups of a block are one aligned 32-bit word
  int early;                   // weights / scales were not written by the previous kernel
  const int64_t* indptr;       // grouped form: end rows (device), else nullptr
  int has_prev, num_experts;
  int64_t w_expert_bytes, s_expert_stride;
  uint32_t* partial;           // [grid][nb / 4][128][4] fp32 words, kVacant at rest
  unsigned wait_limit_ms;
};

inline size_t bar_bytes() { return (size_t)(4 * kMaxStages + 2 * kMaxA + 4 + kMaxGroups) * 8 + 16 + (3 * kMaxExperts + 4) * sizeof(int); }
inline size_t smem_bytes(int nb, int x_stages, int w_stages, int groups) {
  return 1024 + (size_t)x_stages * nb * 128 + (size_t)w_stages * kWBytes + (size_t)groups * kStageBytes + bar_bytes();
}

struct Launch {
  int grid, groups, zmode, src;
  size_t smem;
};
int launch_i4(const Params& pp, const Launch& l, const CUtensorMap& tx, cudaStream_t stream);
int launch_i8(const Params& pp, const Launch& l, const CUtensorMap& tx, cudaStream_t stream);

#ifdef __CUDACC__

using ug::elect_one;
using ug::make_b_desc;
using ug::tc_commit;
using ug::tc_fence_after;
using ug::tc_fence_before;
using ug::tc_ld16;
using ug::tc_mma_ts;
using ug::tc_st32;
using ug::tc_wait_st;

struct Tables {
  int base[kMaxExperts + 1];  // first item of an expert
  int row_begin[kMaxExperts];
  int row_end[kMaxExperts];
};
struct Item {
  int e, n_tile, m0, m_end;
};

__device__ __forceinline__ void tma_load_x(void* smem_dst, const CUtensorMap* map, int c0, int c1, uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(
          smem_u32(smem_dst)),
      "l"(map), "r"(c0), "r"(c1), "r"(smem_u32(bar))
      : "memory");
}

__device__ __forceinline__ void st_relaxed_v4(uint4* p, const uint4& v) {
  asm volatile("st.volatile.global.v4.u32 [%0], {%1, %2, %3, %4};" ::"l"(p), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w) : "memory");
}
__device__ __forceinline__ uint4 ld_relaxed_v4(const uint4* p) {
  uint4 v;
  asm volatile("ld.volatile.global.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ bool arrived(const uint4& v) {
  return v.x != kVacant && v.y != kVacant && v.z != kVacant && v.w != kVacant;
}
// v += the 16 columns of one contributor and, when `second` is not zero, of the one `second` words of
// 16 bytes further on, in that order; leaves the words vacant.  False when the wait ran out.
__device__ __forceinline__ bool add_parts(float (&v)[16], uint4* part, int second, unsigned limit_ms, int* status) {
  uint4 a[4], b[4];
  unsigned long long t0 = 0ull;
  for (;;) {
    bool all = true;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      a[i] = ld_relaxed_v4(part + i * kTileRows);
      b[i] = second ? ld_relaxed_v4(part + second + i * kTileRows) : make_uint4(0u, 0u, 0u, 0u);
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) all = all && arrived(a[i]) && arrived(b[i]);
    if (all) break;
    unsigned long long t1;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t1));
    if (t0 == 0ull) t0 = t1;
    if (t1 - t0 > (limit_ms ? limit_ms : 2000u) * 1000000ull) {  // give up, report, leave the tile unwritten
      if (status) atomicExch(status, kStatusWaitTimeout);
      return false;
    }
  }
  const uint4 vacant = make_uint4(kVacant, kVacant, kVacant, kVacant);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    v[4 * i] += __uint_as_float(a[i].x);
    v[4 * i + 1] += __uint_as_float(a[i].y);
    v[4 * i + 2] += __uint_as_float(a[i].z);
    v[4 * i + 3] += __uint_as_float(a[i].w);
    part[i * kTileRows] = vacant;
    if (second) {
      v[4 * i] += __uint_as_float(b[i].x);
      v[4 * i + 1] += __uint_as_float(b[i].y);
      v[4 * i + 2] += __uint_as_float(b[i].z);
      v[4 * i + 3] += __uint_as_float(b[i].w);
      part[second + i * kTileRows] = vacant;
    }
  }
  return true;
}

// One 64-k block of this thread's weight row -> 32 packed fp16 pairs in k order.  `blk`: this thread's
// row block inside the stage, `off`: its unit offsets, HI: rows g + 8 of the 16-row block.
// s / z: f16x2 scale and zero point of (tile, lane run): index ti * 4 + t for int8, t for int4.
template <int BITS, int ZMODE, int HI, class SFn, class ZFn>
__device__ __forceinline__ void decode_block(const uint8_t* blk, const uint32_t (&off)[4], const ZeroConsts& zc, SFn s_of, ZFn z_of,
                                             uint32_t (&regs)[32]) {
  if constexpr (BITS == 4) {
    constexpr uint32_t kMagic = 0x64006400u, kSixteenth = 0x2C002C00u;
    constexpr uint32_t kMask = HI ? 0x00f000f0u : 0x000f000fu;
#pragma unroll
    for (int t = 0; t < 4; ++t) {
      const uint4 u = *reinterpret_cast<const uint4*>(blk + off[t]);
      const uint32_t s2 = s_of(t), z2 = z_of(t);
      const uint32_t ww[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        uint32_t e0 = and_or(ww[j], kMask, kMagic), e1 = and_or(ww[j] >> 8, kMask, kMagic);
        if (HI) {
          e0 = h2_fma(e0, kSixteenth, zc.add_hi);
          e1 = h2_fma(e1, kSixteenth, zc.add_hi);
        } else {
          e0 = h2_sub(e0, zc.sub_lo);
          e1 = h2_sub(e1, zc.sub_lo);
        }
        if (ZMODE == kZeroGeneral) {
          e0 = h2_sub(e0, z2);
          e1 = h2_sub(e1, z2);
        }
        regs[8 * t + 2 * j] = h2_mul(e0, s2);
        regs[8 * t + 2 * j + 1] = h2_mul(e1, s2);
      }
    }
  } else {
    constexpr uint32_t kMagicBytes = 0x64646464u;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int ti = i >> 2, t = i & 3;
      const uint4 u = *reinterpret_cast<const uint4*>(blk + ti * 512 + off[t]);
      const uint32_t s2 = s_of(i), z2 = z_of(i);
      const uint32_t ww[2] = {HI ? u.y : u.x, HI ? u.w : u.z};
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        uint32_t e0 = h2_sub(prmt(ww[j], kMagicBytes, 0x4140u), zc.sub_lo);
        uint32_t e1 = h2_sub(prmt(ww[j], kMagicBytes, 0x4342u), zc.sub_lo);
        if (ZMODE == kZeroGeneral) {
          e0 = h2_sub(e0, z2);
          e1 = h2_sub(e1, z2);
        }
        regs[16 * ti + 4 * t + 2 * j] = h2_mul(e0, s2);
        regs[16 * ti + 4 * t + 2 * j + 1] = h2_mul(e1, s2);
      }
    }
  }
}

template <int BITS, int ZMODE, int SRC, int G>
__global__ void __launch_bounds__((4 + 4 * G) * 32, G == 2 ? 2 : 1)
    umma_sk_kernel(const Params pp, const __grid_constant__ CUtensorMap tmap_x) {
  constexpr int kBlkPerChunk = BITS == 8 ? 2 : 4;   // 64-k blocks per weight stage
  constexpr int kTilesPerBlk = BITS == 8 ? 2 : 1;
  constexpr int kFragK = BITS == 8 ? 32 : 64;
  constexpr int kOwn = kBlkPerChunk >= G ? kBlkPerChunk / G : 1;  // adjacent blocks of a chunk one group decodes: an A slot
  constexpr int kSlots = kBlkPerChunk / kOwn;                      // A slots of a whole chunk
  constexpr bool kZ = ZMODE == kZeroGeneral;
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
  uint64_t* w_full = reinterpret_cast<uint64_t*>(e_stage + G * kStageBytes);
  uint64_t* w_empty = w_full + kMaxStages;
  uint64_t* x_full = w_empty + kMaxStages;
  uint64_t* x_empty = x_full + kMaxStages;
  uint64_t* a_full = x_empty + kMaxStages;
  uint64_t* a_empty = a_full + kMaxA;
  uint64_t* d_full = a_empty + kMaxA;
  uint64_t* d_empty = d_full + 2;
  uint64_t* e_bar = d_empty + 2;
  uint32_t* tmem_holder = reinterpret_cast<uint32_t*>(e_bar + kMaxGroups);
  Tables& tt = *reinterpret_cast<Tables*>(tmem_holder + 4);

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const bool grouped = pp.indptr != nullptr;
  if (tid == 0) {
    for (int s = 0; s < w_stages; ++s) {
      mbar_init(&w_full[s], 1);
      mbar_init(&w_empty[s], 4 * G);
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
      mbar_init(&d_empty[i], 4 * G);
    }
    for (int i = 0; i < G; ++i) mbar_init(&e_bar[i], 4);
    mbar_fence_init();
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
  // (experts without rows can leave fewer units than CTAs: the surplus CTAs stay out of the split)
  const unsigned ctas = min(gridDim.x, total);
  const unsigned u_begin = blockIdx.x < ctas ? blockIdx.x * total / ctas : 0u;
  const unsigned u_end = blockIdx.x < ctas ? (blockIdx.x + 1) * total / ctas : 0u;

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
    const uint32_t zconst_h2 = h2_bcast(__float2half_rn(p.zero_const));
    const bool has_zeros = kZ && p.z != nullptr;
    uint32_t off[4];
#pragma unroll
    for (int t = 0; t < 4; ++t) off[t] = (uint32_t)(t * 128 + ((g + 2 * t) & 7) * 16);
    if (!grouped && !pp.early) griddep_wait();  // scales may be the previous kernel's output
    bool waited = grouped || !pp.early;

    const int k_blocks = p.k / kKBlock;
    // scales of this group's blocks of a chunk, fetched one chunk ahead
    uint32_t sv[kOwn], zv[kOwn], sn[kOwn], zn[kOwn];
    uint32_t s_row = 0u, z_row = zconst_h2;
    const __half *sp = nullptr, *zp = nullptr;
    // first block of the chunk this group decodes (kOwn of them), or -1
    auto own_first = [&](unsigned seq) -> int {
      if (kBlkPerChunk >= G) return grp * kOwn;
      return (int)(seq % (G / kBlkPerChunk)) == grp / kBlkPerChunk ? grp % kBlkPerChunk : -1;
    };
    auto fetch = [&](unsigned seq, int c, uint32_t (&s)[kOwn], uint32_t (&z)[kOwn]) {
      if (SRC != kOne && SRC != kTwo) return;
      const int first = own_first(seq);
      if (first < 0) return;
#pragma unroll
      for (int i = 0; i < kOwn; ++i) {
        const int kb = min(c * kBlkPerChunk + first + i, k_blocks - 1);
        if (SRC == kOne) {
          const int64_t o = (int64_t)((unsigned)(kb * kKBlock) / (unsigned)p.group) * pp.s_g;
          s[i] = ld_nc_u16(sp + o) * 0x10001u;
          if (has_zeros) z[i] = ld_nc_u16(zp + o) * 0x10001u;
        } else if (pp.s_vec) {
          s[i] = __ldg(reinterpret_cast<const uint32_t*>(sp + kb * 2));
          if (has_zeros) z[i] = __ldg(reinterpret_cast<const uint32_t*>(zp + kb * 2));
        } else {
          const int64_t o = (int64_t)(kb * 2) * pp.s_g;
          s[i] = ld_nc_u16(sp + o) | (ld_nc_u16(sp + o + pp.s_g) << 16);
          if (has_zeros) z[i] = ld_nc_u16(zp + o) | (ld_nc_u16(zp + o + pp.s_g) << 16);
        }
      }
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
    unsigned seq = 0, step = 0;
    Walk w;
    for (bool have = begin(w); ok && have; have = next(w)) {
      const Item it = get_item(w.item);
      const int n_row = it.n_tile * kTileRows + row;
      {
        const int n_s = min(n_row, p.n - 1);
        const int64_t o = it.e * pp.s_expert_stride + (int64_t)n_s * pp.s_n;
        sp = p.s + o;
        zp = p.z + o;
        if (SRC == kChannel) {
          s_row = ld_nc_u16(sp) * 0x10001u;
          if (has_zeros) z_row = ld_nc_u16(zp) * 0x10001u;
        }
      }
      fetch(seq, w.c0, sn, zn);
      for (int c = w.c0; c < w.c1; ++c, ++seq) {
#pragma unroll
        for (int i = 0; i < kOwn; ++i) {
          sv[i] = sn[i];
          zv[i] = zn[i];
        }
        if (c + 1 < w.c1) fetch(seq + 1, c + 1, sn, zn);
        if (!mbar_wait_parked(&w_full[ws], wph, p.status)) {
          ok = false;
          break;
        }
        const int nft = min(4, KT - c * 4), nblk = nft / kTilesPerBlk;
        const uint8_t* blk0 = w_ring + (size_t)ws * kWBytes + bl * (nft * 512);
        const int first = own_first(seq);
        if (first >= 0 && first < nblk) {
          int ab = ab0 + first / kOwn;
          uint32_t aph = aph0;
          if (ab >= pp.na) {
            ab -= pp.na;
            aph ^= 1u;
          }
          const uint32_t a_taddr = lane_taddr | (tmem + (uint32_t)(pp.a_base + ab * (kOwn * 32)));
#pragma unroll
          for (int i = 0; i < kOwn; ++i) {
            const int b = first + i;
            uint32_t regs[32];
            const uint8_t* blk = blk0 + b * (kTilesPerBlk * 512);
            auto s_of = [&](int t) -> uint32_t {  // t: lane run (int8: tile * 4 + lane run)
              if (SRC == kChannel) return s_row;
              if (SRC == kOne) return sv[i];
              if (SRC == kTwo) return prmt(sv[i], sv[i], (BITS == 4 ? t >> 1 : t >> 2) ? 0x3232u : 0x1010u);
              const unsigned k = (unsigned)((c * kBlkPerChunk + b) * kKBlock + (BITS == 4 ? t * 16 : t * 8));
              return ld_nc_u16(sp + (int64_t)(k / (unsigned)p.group) * pp.s_g) * 0x10001u;
            };
            auto z_of = [&](int t) -> uint32_t {
              if (!kZ || !has_zeros) return zconst_h2;
              if (SRC == kChannel) return z_row;
              if (SRC == kOne) return zv[i];
              if (SRC == kTwo) return prmt(zv[i], zv[i], (BITS == 4 ? t >> 1 : t >> 2) ? 0x3232u : 0x1010u);
              const unsigned k = (unsigned)((c * kBlkPerChunk + b) * kKBlock + (BITS == 4 ? t * 16 : t * 8));
              return ld_nc_u16(zp + (int64_t)(k / (unsigned)p.group) * pp.s_g) * 0x10001u;
            };
            if (i > 0 && b >= nblk) break;
            if (hi) decode_block<BITS, ZMODE, 1>(blk, off, zc, s_of, z_of, regs);
            else decode_block<BITS, ZMODE, 0>(blk, off, zc, s_of, z_of, regs);
            if (i == 0) {  // the first block is decoded before the slot has to be free
              ok = mbar_wait_parked(&a_empty[ab], aph, p.status);
              if (!ok) break;
              tc_fence_after();
            }
            tc_st32(a_taddr + (uint32_t)(i * 32), regs);
          }
          if (ok) {
            tc_wait_st();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&a_full[ab]);
          }
        }
        if (!ok) break;
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
      if (!waited) {
        griddep_wait();  // outputs and scratch may be in use by the previous kernel until it has ended
        waited = true;
      }
      const uint32_t d = lane_taddr | (tmem + (uint32_t)(db * pp.d_stride));
      const int cols = min(nb, it.m_end - it.m0);
      if (w.c0 > 0) {
        // the tile began in an earlier CTA: publish
        uint4* slot = reinterpret_cast<uint4*>(pp.partial) + (size_t)blockIdx.x * (nb / 4) * kTileRows + gj;
        for (int c0 = grp * 16; c0 < cols; c0 += G * 16) {
          float v[16];
          tc_ld16(d + (uint32_t)c0, v);
          uint32_t u[16];
#pragma unroll
          for (int i = 0; i < 16; ++i) {
            u[i] = __float_as_uint(v[i]);
            if (u[i] == kVacant) u[i] = 0x7fffffffu;
          }
#pragma unroll
          for (int i = 0; i < 4; ++i)
            st_relaxed_v4(slot + (size_t)(c0 / 4 + i) * kTileRows, make_uint4(u[4 * i], u[4 * i + 1], u[4 * i + 2], u[4 * i + 3]));
        }
      } else {
        int last_cta = (int)blockIdx.x;
        if (w.c1 < cpt) {
          // this CTA owns the tile, later ones hold the rest
          const unsigned hi_u = (unsigned)w.item * (unsigned)cpt + (unsigned)cpt - 1u;
          last_cta = (int)(((hi_u + 1u) * ctas - 1u) / total);
        }
        const int n_read = min(n_row, p.n - 1);  // rows past n are computed on stale bytes and never stored
        for (int c0 = grp * 16; c0 < cols; c0 += G * 16, ++step) {
          float v[16];
          tc_ld16(d + (uint32_t)c0, v);
          for (int c = (int)blockIdx.x + 1; c <= last_cta && ok; c += 2)  // fixed CTA order, two at a time
            ok = add_parts(v, reinterpret_cast<uint4*>(pp.partial) + ((size_t)c * (nb / 4) + c0 / 4) * kTileRows + gj,
                           c < last_cta ? (nb / 4) * kTileRows : 0, pp.wait_limit_ms, p.status);
          if (!__all_sync(0xffffffffu, ok)) {
            ok = false;
            break;
          }
          const int mrow0 = it.m0 + c0;
          if (p.epi.act == kActSwiglu) {
            // gate and up rows of one f sit in different warps: fp32 through shared memory
            float* st = reinterpret_cast<float*>(e_stage + grp * kStageBytes);
            if (!group_sync()) {
              ok = false;
              break;
            }
#pragma unroll
            for (int i = 0; i < 16; ++i) st[i * kTileRows + row] = v[i];
            if (!group_sync()) {
              ok = false;
              break;
            }
            const int mi = gj >> 3, q = gj & 7;  // batch row, 16-row block = eight f
            const int m = mrow0 + mi;
            if (m < it.m_end && it.n_tile * kTileRows + q * 16 < p.n) {
              const float4* src = reinterpret_cast<const float4*>(st + mi * kTileRows + q * 16);
              const float4 g0 = src[0], g1 = src[1], u0 = src[2], u1 = src[3];
              __half2 res[4];
              res[0] = __floats2half2_rn(silu_mul(g0.x, u0.x), silu_mul(g0.y, u0.y));
              res[1] = __floats2half2_rn(silu_mul(g0.z, u0.z), silu_mul(g0.w, u0.w));
              res[2] = __floats2half2_rn(silu_mul(g1.x, u1.x), silu_mul(g1.y, u1.y));
              res[3] = __floats2half2_rn(silu_mul(g1.z, u1.z), silu_mul(g1.w, u1.w));
              *reinterpret_cast<uint4*>(p.out + (int64_t)m * p.ldo + it.n_tile * (kTileRows / 2) + q * 8) =
                  *reinterpret_cast<const uint4*>(res);
            }
          } else {
            // transpose through shared memory: 16 batch rows x 128 weight rows, rounded once
            __half* st = reinterpret_cast<__half*>(e_stage + grp * kStageBytes) + (step & 1u) * 16 * kTileRows;
            apply_epilogue16(v, p.epi, mrow0, it.m_end, n_read);
#pragma unroll
            for (int i = 0; i < 16; ++i) st[i * kTileRows + row] = __float2half_rn(v[i]);
            if (!group_sync()) {
              ok = false;
              break;
            }
#pragma unroll
            for (int pass = 0; pass < 2; ++pass) {
              const int mi = pass * 8 + (gj >> 4), ch = gj & 15;
              const int m = mrow0 + mi;
              if (m < it.m_end && it.n_tile * kTileRows + ch * 8 < p.n)
                *reinterpret_cast<uint4*>(p.out + (int64_t)m * p.ldo + it.n_tile * kTileRows + ch * 8) =
                    *reinterpret_cast<const uint4*>(st + mi * kTileRows + ch * 8);
            }
          }
        }
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
  }

  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    ug::tmem_dealloc(tmem, (uint32_t)pp.tmem_cols);
  }
}

template <int BITS, int ZMODE, int SRC, int G>
int launch_inst(const Params& pp, const Launch& l, const CUtensorMap& tx, cudaStream_t stream) {
  auto kern = umma_sk_kernel<BITS, ZMODE, SRC, G>;
  static thread_local int configured_device = -1;
  int dev = 0;
  RB200_CUDA(cudaGetDevice(&dev));
  if (configured_device != dev) {
    RB200_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024));
    configured_device = dev;
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)l.grid, 1, 1);
  cfg.blockDim = dim3((4 + 4 * G) * 32, 1, 1);
  cfg.dynamicSmemBytes = l.smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  // always a programmatic dependent: before its wait the kernel only prefetches, unless the host
  // switched launch overlap on
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  RB200_CUDA(cudaLaunchKernelEx(&cfg, kern, pp, tx));
  return 0;
}

template <int BITS, int ZMODE>
int launch_src(const Params& pp, const Launch& l, const CUtensorMap& tx, cudaStream_t stream) {
#define RB200_US(S)                                                                      \
  if (l.src == (S))                                                                      \
    return l.groups == 2 ? launch_inst<BITS, ZMODE, S, 2>(pp, l, tx, stream) : launch_inst<BITS, ZMODE, S, 4>(pp, l, tx, stream)
  RB200_US(kChannel);
  RB200_US(kOne);
  RB200_US(kTwo);
  RB200_US(kAny);
#undef RB200_US
  RB200_CHECK(false, "no medium-batch kernel for scale source %d", l.src);
  return -1;
}
template <int BITS>
int launch_bits(const Params& pp, const Launch& l, const CUtensorMap& tx, cudaStream_t stream) {
  return l.zmode == kZeroGeneral ? launch_src<BITS, kZeroGeneral>(pp, l, tx, stream)
                                 : launch_src<BITS, kZeroConstInt>(pp, l, tx, stream);
}

#endif  // __CUDACC__

}  // namespace us

// Host entry: 1 when the problem is outside this kernel's coverage (ungrouped only), 0 on launch, -1 on error.
// Grouped (indptr != nullptr): p.m = total rows; shapes outside the coverage are errors.
int umma_sk_run(const GemvParams& p, int bits, int zmode, int sm_count, uint32_t* vacant_words, size_t vacant_bytes,
                const int64_t* indptr, int has_prev, int num_experts, int64_t w_expert_bytes,
                int64_t s_expert_stride, cudaStream_t stream);

}  // namespace rb200
