// What the tensor-core kernels over packed weights share (umma_sk.cuh: one CTA per tile row block;
// umma_pair.cuh: CTA pairs): parameters, the bit-exact decode of a 64-k block of a weight row, the
// scale feed, the hand-over of partial accumulators between CTAs, and the drain of an accumulator.
#pragma once

#include <cuda.h>

#include "dequant.cuh"
#include "gemv.h"
#include "umma_common.cuh"
#include "umma_index.h"

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
constexpr int kStageBytes = 16 * kTileRows * 4;  // per drain group: two 16 x 128 fp16 buffers, or one fp32

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
  int whole;                   // umma_sk: CTAs that take a whole tile each
  int x_stages, w_stages;
  int nd, d_stride, a_base, na, tmem_cols;  // accumulators and A slots in tensor memory
  int s_n, s_g;                // scale strides in elements
  int blk_shift;               // kOne: log2 of a group's 64-k blocks, or -1
  int s_vec;                   // kTwo: the two groups of a block are one aligned 32-bit word (1), those of two
                               // adjacent blocks one 64-bit word (2; pairs_fit_rows)
  int early;                   // weights / scales were not written by the previous kernel
  const int64_t* indptr;       // grouped form: end rows (device), else nullptr
  int has_prev, num_experts;
  int64_t w_expert_bytes, s_expert_stride;
  uint32_t* partial;           // [grid][nb / 4][128][4] fp32 words, kVacant at rest; nullptr: no tile is cut
  unsigned wait_limit_ms;
};

#ifdef __CUDACC__

// One scale per row and an integer zero point: the MMA takes u - z as it is, in the codes' units (fp16
// subnormals, codes_int4_word in dequant.cuh, and a subtraction that is exact), and the drain multiplies
// the fp32 sums by the scale: 2.5 (int8: 2) instead of 3.5 (3) instructions per pair of weights, and one
// rounding less.  Measured for int8 k 8192 x n 57344: 24 rows 92.4 -> 85.7 us, 64 rows 109 -> 104, 256 rows
// 193 -> 185, 4096 rows 2880 -> 2736 (under the power cap: less arithmetic, higher clocks); int4 k 4096 x
// n 22016: 24 rows 20.2 -> 18.8, 64 rows 23.5 -> 21.8, 512 rows 76.3 -> 73.1.
constexpr int kCodes = 3;
template <int ZMODE, int SRC>
constexpr bool folds() {
  return SRC == kChannel && ZMODE == kZeroConstInt;
}
// one over the unit of a row's codes
template <int BITS>
__device__ __forceinline__ float code_scale(bool hi) {
  return BITS == 4 && hi ? 1048576.0f : 16777216.0f;
}
template <int BITS>
__device__ __forceinline__ float drain_scale(uint32_t s2, bool hi) {
  return __half2float(__ushort_as_half((unsigned short)(s2 & 0xffffu))) * code_scale<BITS>(hi);
}

using ug::elect_one;
using ug::make_b_desc;
using ug::tc_fence_after;
using ug::tc_fence_before;
using ug::tc_ld16;
using ug::tc_st8;
using ug::tc_wait_st;

struct Tables {
  int base[kMaxExperts + 1];  // first item of an expert
  int row_begin[kMaxExperts];
  int row_end[kMaxExperts];
};
struct Item {
  int e, n_tile, m0, m_end;
};

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
template <bool TWO>
__device__ __forceinline__ bool add_parts(float (&v)[16], uint4* part, int second, unsigned limit_ms, int* status) {
  uint4 a[4], b[4];
  if (!TWO) second = 0;
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

// One 64-k block of this thread's weight row -> 32 columns of tensor memory at `taddr`, packed fp16 pairs
// in k order.  `blk`: this thread's row block inside the stage, `off`: its unit offsets, HI: rows g + 8 of
// the 16-row block.  s / z: f16x2 scale and zero point of (tile, lane run): index ti * 4 + t for int8, t
// for int4.  Stored eight columns at a time while the next eight are decoded: a store holds on to its
// registers for 150 to 340 clocks, which one store of all 32 per block exposed in full.
template <int BITS, int ZMODE, int HI, class SFn, class ZFn>
__device__ __forceinline__ void decode_block(const uint8_t* blk, const uint32_t (&off)[4], const ZeroConsts& zc, SFn s_of, ZFn z_of,
                                             uint32_t taddr) {
  if constexpr (BITS == 4) {
    constexpr uint32_t kMagic = 0x64006400u, kSixteenth = 0x2C002C00u;
    constexpr uint32_t kMask = HI ? 0x00f000f0u : 0x000f000fu;
#pragma unroll
    for (int t = 0; t < 4; ++t) {
      const uint4 u = *reinterpret_cast<const uint4*>(blk + off[t]);
      const uint32_t s2 = s_of(t), z2 = z_of(t);
      const uint32_t ww[4] = {u.x, u.y, u.z, u.w};
      uint32_t regs[8];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        if (ZMODE == kCodes) {
          regs[2 * j] = h2_sub(ww[j] & kMask, z2);
          regs[2 * j + 1] = h2_sub((ww[j] >> 8) & kMask, z2);
          continue;
        }
        uint32_t e0 = and_or(ww[j], kMask, kMagic), e1 = and_or(ww[j] >> 8, kMask, kMagic);
        if (HI) {
          e0 = h2_fma(e0, kSixteenth, ZMODE == kZeroExact ? z2 : zc.add_hi);
          e1 = h2_fma(e1, kSixteenth, ZMODE == kZeroExact ? z2 : zc.add_hi);
        } else {
          e0 = h2_sub(e0, ZMODE == kZeroExact ? z2 : zc.sub_lo);
          e1 = h2_sub(e1, ZMODE == kZeroExact ? z2 : zc.sub_lo);
        }
        if (ZMODE == kZeroGeneral) {
          e0 = h2_sub(e0, z2);
          e1 = h2_sub(e1, z2);
        }
        regs[2 * j] = h2_mul(e0, s2);
        regs[2 * j + 1] = h2_mul(e1, s2);
      }
      tc_st8(taddr + (uint32_t)(8 * t), regs);
    }
  } else {
    constexpr uint32_t kMagicBytes = 0x64646464u;
#pragma unroll
    for (int h = 0; h < 4; ++h) {
      uint32_t regs[8];
#pragma unroll
      for (int o = 0; o < 2; ++o) {
        const int i = 2 * h + o, ti = i >> 2, t = i & 3;
        const uint4 u = *reinterpret_cast<const uint4*>(blk + ti * 512 + off[t]);
        const uint32_t s2 = s_of(i), z2 = z_of(i);
        const uint32_t ww[2] = {HI ? u.y : u.x, HI ? u.w : u.z};
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          if (ZMODE == kCodes) {
            regs[4 * o + 2 * j] = h2_sub(prmt(ww[j], 0u, 0x4140u), z2);
            regs[4 * o + 2 * j + 1] = h2_sub(prmt(ww[j], 0u, 0x4342u), z2);
            continue;
          }
          uint32_t e0 = h2_sub(prmt(ww[j], kMagicBytes, 0x4140u), ZMODE == kZeroExact ? z2 : zc.sub_lo);
          uint32_t e1 = h2_sub(prmt(ww[j], kMagicBytes, 0x4342u), ZMODE == kZeroExact ? z2 : zc.sub_lo);
          if (ZMODE == kZeroGeneral) {
            e0 = h2_sub(e0, z2);
            e1 = h2_sub(e1, z2);
          }
          regs[4 * o + 2 * j] = h2_mul(e0, s2);
          regs[4 * o + 2 * j + 1] = h2_mul(e1, s2);
        }
      }
      tc_st8(taddr + (uint32_t)(8 * h), regs);
    }
  }
}

// The same with the scales and zero points of `feed`'s own block i (64-k block kb).
template <int BITS, int ZMODE, int SRC, class Feed>
__device__ __forceinline__ void decode_own(const Params& pp, const Feed& feed, int i, int kb, const uint8_t* blk,
                                           const uint32_t (&off)[4], const ZeroConsts& zc, uint32_t taddr) {
  if constexpr (folds<ZMODE, SRC>()) {
    auto none = [](int) { return 0u; };
    auto z_of = [&](int) { return feed.z_row_o; };
    if (feed.hi) decode_block<BITS, kCodes, 1>(blk, off, zc, none, z_of, taddr);
    else decode_block<BITS, kCodes, 0>(blk, off, zc, none, z_of, taddr);
    return;
  }
  auto s_of = [&](int t) { return feed.scale(pp, i, kb, t); };
  if (ZMODE == kZeroGeneral && !feed.block_exact(i)) {
    auto z_of = [&](int t) { return feed.zero(pp, i, kb, t); };
    if (feed.hi) decode_block<BITS, ZMODE, 1>(blk, off, zc, s_of, z_of, taddr);
    else decode_block<BITS, ZMODE, 0>(blk, off, zc, s_of, z_of, taddr);
  } else {
    constexpr int kMode = ZMODE == kZeroGeneral ? kZeroExact : ZMODE;
    auto z_of = [&](int t) { return ZMODE == kZeroGeneral ? feed.zero_exact(i, t) : 0u; };
    if (feed.hi) decode_block<BITS, kMode, 1>(blk, off, zc, s_of, z_of, taddr);
    else decode_block<BITS, kMode, 0>(blk, off, zc, s_of, z_of, taddr);
  }
}

// Scales and zero points of the blocks one group of warps decodes, fetched a chunk ahead.
// APART: where a kTwo block's two groups are no word, they are put together when their chunk's turn comes and not
// where they are loaded, which would wait for the loads there (int8 in groups of 32: k 8192 x n 8192, 256 rows 87 us
// put together at the load, 53 apart, k 4096 x n 22016, 32 rows 33.6 / 28.4; int4 with scales [K/32, N], 128 rows,
// k 4096 x n 22016 41.4 / 31.8).  Int4 on one CTA a tile has no registers for it, and would lose 2 % where the groups
// are words (k 4096 x n 22016, 32 rows).
template <int BITS, int ZMODE, int SRC, int OWN, bool APART>
struct ScaleFeed {
  static constexpr bool kZ = ZMODE == kZeroGeneral;
  const __half *sp, *zp;
  uint32_t s_row, s_row2, z_row;                // kChannel (s_row2, int4: twice, for the current chunk)
  uint32_t sv[OWN], zv[OWN], sn[OWN], zn[OWN];  // current chunk, next chunk
  uint32_t sn2[OWN], zn2[OWN];                  // APART: the next chunk's second groups, 0 beside words
  uint32_t zconst_h2;
  bool has_zeros, hi;
  uint32_t zo[OWN], z_row_o;                    // offset zero points (kZeroExact; kCodes: in the codes' units) ...
  bool exact[OWN], row_exact;                   // ... where they are exact

  __device__ __forceinline__ uint32_t offset(uint32_t z2, bool& ok) const {
    return BITS == 4 && hi ? zero_offset_hi(z2, ok) : zero_offset_lo(z2, ok);
  }
  __device__ __forceinline__ void init(const Params& pp, bool hi_rows) {
    hi = hi_rows;
    row_exact = SRC != kAny;
    zconst_h2 = h2_bcast(__float2half_rn(pp.g.zero_const));
    has_zeros = kZ && pp.g.z != nullptr;
#pragma unroll
    for (int i = 0; i < OWN; ++i) sn2[i] = zn2[i] = 0u;
    s_row = 0u;
    z_row = zconst_h2;
    if (kZ) z_row_o = offset(zconst_h2, row_exact);
    else if (folds<ZMODE, SRC>()) z_row_o = h2_bcast(__float2half_rn(pp.g.zero_const / code_scale<BITS>(hi)));
  }
  __device__ __forceinline__ void row(const Params& pp, int e, int n_row) {
    const int64_t o = e * pp.s_expert_stride + (int64_t)min(n_row, pp.g.n - 1) * pp.s_n;
    sp = pp.g.s + o;
    zp = pp.g.z + o;
    if (SRC == kChannel) {
      // doubled for a chunk or where it is used, not to wait for it here (int4 with zero points, k 4096 x n 22016, 24
      // rows: 22.6 us doubled at each use, 22.2 for a chunk; int8 has no register for it and loses 1 %)
      s_row = ld_nc_u16(sp);
      if (has_zeros) {
        z_row = ld_nc_u16(zp) * 0x10001u;
        row_exact = true;
        z_row_o = offset(z_row, row_exact);
      }
    }
  }
  // the i-th own block of the next chunk is 64-k block kb
  __device__ __forceinline__ void fetch(const Params& pp, int i, int kb) {
    if (SRC == kOne) {
      const int64_t o = (int64_t)(pp.blk_shift >= 0 ? (unsigned)kb >> pp.blk_shift : (unsigned)(kb * kKBlock) / (unsigned)pp.g.group) * pp.s_g;
      sn[i] = ld_nc_u16(sp + o);
      if (has_zeros) zn[i] = ld_nc_u16(zp + o);
    } else if (SRC == kTwo && pp.s_vec) {
      sn[i] = __ldg(reinterpret_cast<const uint32_t*>(sp + kb * 2));
      if (has_zeros) zn[i] = __ldg(reinterpret_cast<const uint32_t*>(zp + kb * 2));
    } else if (SRC == kTwo) {
      const int64_t o = (int64_t)(kb * 2) * pp.s_g;
      const uint32_t a = ld_nc_u16(sp + o), b = ld_nc_u16(sp + o + pp.s_g);
      sn[i] = APART ? a : a | (b << 16);
      sn2[i] = b;
      if (has_zeros) {
        const uint32_t za = ld_nc_u16(zp + o), zb = ld_nc_u16(zp + o + pp.s_g);
        zn[i] = APART ? za : za | (zb << 16);
        zn2[i] = zb;
      }
    }
  }
  // own blocks 0, 1 of the next chunk are the adjacent 64-k blocks kb, kb + 1 (kb even): their four group-32
  // scales are one 8-byte load when the rows allow it
  __device__ __forceinline__ void fetch_two(const Params& pp, int kb, int k_blocks) {
    if (SRC == kTwo && pp.s_vec == 2) {
      const uint2 s = __ldg(reinterpret_cast<const uint2*>(sp + kb * 2));
      sn[0] = s.x;
      sn[OWN - 1] = s.y;
      if (has_zeros) {
        const uint2 z = __ldg(reinterpret_cast<const uint2*>(zp + kb * 2));
        zn[0] = z.x;
        zn[OWN - 1] = z.y;
      }
      return;
    }
#pragma unroll
    for (int i = 0; i < OWN; ++i) fetch(pp, i, min(kb + i, k_blocks - 1));
  }
  __device__ __forceinline__ void advance() {
    if (SRC == kChannel && BITS == 4 && !folds<ZMODE, SRC>()) s_row2 = s_row * 0x10001u;
#pragma unroll
    for (int i = 0; i < OWN; ++i) {
      // (kOne: doubled here and not where it is loaded, which would wait for the load there: an expert layer's
      // matmul of 1024 rows, k 4096 x n 14336, group 128, spent 1400 of 2900 clocks a step on that)
      sv[i] = SRC == kOne ? sn[i] * 0x10001u : (SRC == kTwo && APART ? sn[i] | (sn2[i] << 16) : sn[i]);
      zv[i] = SRC == kOne ? zn[i] * 0x10001u : (SRC == kTwo && APART ? zn[i] | (zn2[i] << 16) : zn[i]);
      if (kZ && (SRC == kOne || SRC == kTwo) && has_zeros) {
        exact[i] = true;
        zo[i] = offset(zv[i], exact[i]);
      }
    }
  }
  // all lanes' zero points of own block i allow kZeroExact
  __device__ __forceinline__ bool block_exact(int i) const {
    return __all_sync(0xffffffffu, !has_zeros || SRC == kChannel ? row_exact : (SRC == kAny ? false : exact[i]));
  }
  __device__ __forceinline__ uint32_t zero_exact(int i, int t) const {
    if (!has_zeros || SRC == kChannel) return z_row_o;
    return SRC == kTwo ? prmt(zo[i], zo[i], (BITS == 4 ? t >> 1 : t >> 2) ? 0x3232u : 0x1010u) : zo[i];
  }
  // run t (int8: fragment tile * 4 + lane run) of own block i = 64-k block kb
  __device__ __forceinline__ uint32_t scale(const Params& pp, int i, int kb, int t) const {
    if (SRC == kChannel) return BITS == 4 ? s_row2 : prmt(s_row, s_row, 0x1010u);
    if (SRC == kOne) return sv[i];
    if (SRC == kTwo) return prmt(sv[i], sv[i], (BITS == 4 ? t >> 1 : t >> 2) ? 0x3232u : 0x1010u);
    const unsigned k = (unsigned)(kb * kKBlock + (BITS == 4 ? t * 16 : t * 8));
    return ld_nc_u16(sp + (int64_t)(k / (unsigned)pp.g.group) * pp.s_g) * 0x10001u;
  }
  __device__ __forceinline__ uint32_t zero(const Params& pp, int i, int kb, int t) const {
    if (!kZ || !has_zeros) return zconst_h2;
    if (SRC == kChannel) return z_row;
    if (SRC == kOne) return zv[i];
    if (SRC == kTwo) return prmt(zv[i], zv[i], (BITS == 4 ? t >> 1 : t >> 2) ? 0x3232u : 0x1010u);
    const unsigned k = (unsigned)(kb * kKBlock + (BITS == 4 ? t * 16 : t * 8));
    return ld_nc_u16(zp + (int64_t)(k / (unsigned)pp.g.group) * pp.s_g) * 0x10001u;
  }
};

// Drain of one accumulator by a group of four warps (128 TMEM lanes): columns first, first + step, ...
// below `cols`, sixteen at a time.
struct DrainTile {
  uint32_t d;             // tensor-memory address of the accumulator, this warp's lanes
  int first, step, cols;  // columns
  int n0, m0, m_end;      // first weight row of the tile, first batch row, end of the batch rows
  int row, gj;            // weight row of this thread inside the tile, thread index in the group
  float scale;            // SCALED: of this weight row, fetched when the piece began
};

// the partial accumulator of a tile that began in an earlier CTA -> hand-over slot `me`
__device__ __forceinline__ void drain_publish(const Params& pp, const DrainTile& t, int me) {
  uint4* slot = reinterpret_cast<uint4*>(pp.partial) + (size_t)me * (pp.nb / 4) * kTileRows + t.gj;
  for (int c0 = t.first; c0 < t.cols; c0 += t.step) {
    float v[16];
    tc_ld16(t.d + (uint32_t)c0, v);
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
}

// epilogue and store; parts of slots me + slot_step, me + 2 slot_step, ... last are added first (fixed
// order; TWO: two at a time, for 16 registers more), SCALED: the sums are in the units of the codes.  `sync`: barrier of the group, false when its wait ran out.
template <bool TWO, bool SCALED, class Sync>
__device__ __forceinline__ bool drain_store(const Params& pp, const DrainTile& t, int me, int last, int slot_step, uint8_t* stage,
                                            unsigned& parity, Sync sync) {
  const GemvParams& p = pp.g;
  const int n_read = min(t.n0 + t.row, p.n - 1);  // rows past n are computed on stale bytes and never stored
  for (int c0 = t.first; c0 < t.cols; c0 += t.step, parity ^= 1u) {
    float v[16];
    tc_ld16(t.d + (uint32_t)c0, v);
    bool ok = true;
    for (int c = me + slot_step; c <= last && ok; c += (TWO ? 2 : 1) * slot_step)
      ok = add_parts<TWO>(v, reinterpret_cast<uint4*>(pp.partial) + ((size_t)c * (pp.nb / 4) + c0 / 4) * kTileRows + t.gj,
                     c + slot_step <= last ? slot_step * (pp.nb / 4) * kTileRows : 0, pp.wait_limit_ms, p.status);
    if (!__all_sync(0xffffffffu, ok)) return false;
    if (SCALED) {
#pragma unroll
      for (int i = 0; i < 16; ++i) v[i] *= t.scale;
    }
    const int mrow0 = t.m0 + c0;
    if (p.epi.act == kActSwiglu) {
      // gate and up rows of one f sit in different warps: fp32 through shared memory
      float* st = reinterpret_cast<float*>(stage);
      if (!sync()) return false;
#pragma unroll
      for (int i = 0; i < 16; ++i) st[i * kTileRows + t.row] = v[i];
      if (!sync()) return false;
      const int mi = t.gj >> 3, q = t.gj & 7;  // batch row, 16-row block = eight f
      const int m = mrow0 + mi;
      if (m < t.m_end && t.n0 + q * 16 < p.n) {
        const float4* src = reinterpret_cast<const float4*>(st + mi * kTileRows + q * 16);
        const float4 g0 = src[0], g1 = src[1], u0 = src[2], u1 = src[3];
        __align__(16) __half2 res[4];
        res[0] = __floats2half2_rn(silu_mul(g0.x, u0.x), silu_mul(g0.y, u0.y));
        res[1] = __floats2half2_rn(silu_mul(g0.z, u0.z), silu_mul(g0.w, u0.w));
        res[2] = __floats2half2_rn(silu_mul(g1.x, u1.x), silu_mul(g1.y, u1.y));
        res[3] = __floats2half2_rn(silu_mul(g1.z, u1.z), silu_mul(g1.w, u1.w));
        *reinterpret_cast<uint4*>(p.out + (int64_t)m * p.ldo + t.n0 / 2 + q * 8) = *reinterpret_cast<const uint4*>(res);
      }
    } else {
      // transpose through shared memory: 16 batch rows x 128 weight rows, rounded once
      __half* st = reinterpret_cast<__half*>(stage) + (parity & 1u) * 16 * kTileRows;
      apply_epilogue16(v, p.epi, mrow0, t.m_end, n_read);
#pragma unroll
      for (int i = 0; i < 16; ++i) st[i * kTileRows + t.row] = __float2half_rn(v[i]);
      if (!sync()) return false;
#pragma unroll
      for (int pass = 0; pass < 2; ++pass) {
        const int mi = pass * 8 + (t.gj >> 4), ch = t.gj & 15;
        const int m = mrow0 + mi;
        if (m < t.m_end && t.n0 + ch * 8 < p.n)
          *reinterpret_cast<uint4*>(p.out + (int64_t)m * p.ldo + t.n0 + ch * 8) =
              *reinterpret_cast<const uint4*>(st + mi * kTileRows + ch * 8);
      }
    }
  }
  return true;
}

#endif  // __CUDACC__

}  // namespace us

// Host entry of the tensor-core kernels over packed weights: 1 when the problem is outside their coverage
// (ungrouped only), 0 on launch, -1 on error.  Grouped (indptr != nullptr): p.m = total rows; shapes
// outside the coverage are errors.
int umma_run(const GemvParams& p, int bits, int zmode, int sm_count, const int64_t* indptr, int has_prev, int num_experts,
             int64_t w_expert_bytes, int64_t s_expert_stride, cudaStream_t stream);

}  // namespace rb200
