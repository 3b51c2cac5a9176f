// Decode-path kernel for at most sixteen batch rows: row blocks per CTA, k split over its warps.  (Most int4 calls are
// taken by gemv_flat.cuh; the rules, with the figures of both, are in gemv_flat.cu.)
//
//   out[m, n] = epilogue(sum_k x[m, k] * wq[n, k]),  m <= 8 or 16 (one or two m16n8k16 MMAs wide)
//
// Bound: HBM (the packed weight once) and, close behind, instruction issue: the exact two-rounding
// decode is 52 of the 61 instructions a 512-byte tile needs (4 MMAs, 3 loads, 2 scale selects), 36
// where the scale is left to the sums.
// So nothing else is in the loop: no shared memory, no barriers, no copies through the async
// engine.  A warp reads fragment tiles with 128-bit loads that are whole 512-byte lines in the
// fragment layout, straight into the registers the MMA takes them from, one chunk (four tiles)
// ahead of the arithmetic; activations come from L1 / L2 once per chunk and serve all row blocks
// of the pass.  The first chunks are prefetched into L2 before the wait on the previous kernel: a
// prefetch returns no data to this kernel, so it is safe whatever that kernel still writes.
//
// Measured (graph of launches over 400 MB of weights, launch overlap on, one row): int4 group 32
// k 4096 x n 4096 3.9 us (8.1 in the stream-k kernel), x 12288 9.0 (13.6), x 22016 13.9 (19.1),
// k 11008 x n 4096 8.0 (13.4); int8 k 8192 x n 28672, eight rows, 37.7 us = 6.2 TB/s (48.6).
// What bounds int4: about 155 clocks per tile and SM sub-partition, of which the 32 fp16 and 35
// integer instructions take two each and overlap only in part (a loop of alternating lop3 and
// mul.f16x2 issues one per 1.7 clocks where either alone takes 2.0).
//
// Work split: a row block (16 output rows) belongs to one CTA, its k range to the CTA's eight warps,
// whose partial sums meet in shared memory in warp order: no partial ever leaves the SM, there is
// no flag, fence or second pass, and the result does not depend on the grid.
//
// Grouped (expert) form: the row blocks of all experts that have rows form one list, read from
// indptr on the device, so that a whole expert layer is one launch.
#pragma once

#include <type_traits>

#include "dequant.cuh"
#include "gemv.h"

namespace rb200 {
namespace rk {

constexpr int kMaxBatch = 16;   // two m-tiles of eight rows
constexpr int kEntryRows = 8;   // grouped form: batch rows of one entry
constexpr int kLeadChunks = 2;   // chunks between an L2 prefetch and the load
constexpr int kMaxEntries = 32;  // grouped form: (expert, eight batch rows) pairs that 32 rows in all can make

// where a lane gets its scales / zero points from
enum ScaleSrc : int {
  kChannel = 0,  // one per output row
  kRow32 = 1,    // int4, group 32, [N, K/32]: the eight groups of a chunk are one 16-byte load
  kHalf = 2,     // groups of whole chunk halves (two tiles), any strides: one 16-bit load per row and half
  kGeneral = 3,  // any strides and group size: one 16-bit load per row and tile
  kTile = 4,     // as kGeneral, groups of whole tiles
};

// Where u - z goes into the MMA in the codes' units and the scale is applied to its fp32 sums (kFold below),
// which also rounds less: a group has to be whole tiles, since an MMA's sum runs over a quarter of a tile.
// The difference comes before the product, as in the decode: sums of u x and of z x kept apart cancel when
// the activations have a mean (int8 per row, k 28672, mean 4: relative error 1.3e-3 against 2.1e-4 here and
// 2.5e-4 with decoded weights) and turn an infinite activation into NaN.  Nine instructions per code word of
// int4 instead of 13, or 17 with zero points.  Measured at k 4096 x n 11008 int4, four rows, decoded against
// this: group 128 with zero points 12.9 / 10.3 us, without 10.7 / 9.3, group 64 12.0 / 10.1, one scale per row
// 8.8 / 8.2.  Two m-tiles decode (measured only for the form that kept the sums apart, which was slower
// there: 16 rows, group 128 12.8 / 14.6) except with one scale per row and an integer zero point: sixteen rows of int4
// k 4096 x n 22016 18.1 / 16.1, k 8192 x n 57344 66.7 / 57.5, k = n = 4096 5.81 / 5.51; of int8, run for a quarter of a
// second at a time, k 28672 x n 8192 52.6 / 47.6, k 8192 x n 57344 96.9 / 92.6, k 4096 x n 22016 22.0 / 21.7, k = n = 4096
// 5.81 / 5.85 (alone, before the power cap is felt, 4 % slower to 4 % faster: what counts is the arithmetic's power).  With
// zero points int4 is 3 % slower to 19 % faster, int8 10 % to 16 %: those decode.  Group 32 decodes here; gemv_flat.cuh
// keeps its two groups of a tile apart.
constexpr bool folds(int zmode, int src, int m_tiles) {
  if (m_tiles == 2) return src == kChannel && zmode == kZeroConstInt;
  return src != kRow32 && src != kGeneral;
}

// Row blocks of one pass: activations fetched once serve both.  With a scale and a zero point per group of 32 the two
// need more registers than there are (384 to 640 bytes spilled), and one is faster (three layers of hidden 4096, ffn
// 11008: one row 166 -> 149 us, eight 182 -> 157; k 4096 x n 22016, eight rows 24.0 -> 21.4).
constexpr int pass_rows(int src, int zmode) { return src == kRow32 && zmode == kZeroGeneral ? 1 : 2; }

struct Params {
  GemvParams g;
  int group_shift;         // log2 of the group size, or -1
  unsigned per_cta, extra; // ungrouped: row blocks per CTA, and how many CTAs take one more
  int per;                 // kHalf / kTile: halves / tiles of a group
  int s_n, s_g;            // scale strides in elements
  int early;               // the host promises that weights were not written by the previous kernel
  const int64_t* indptr;   // grouped form: end rows per expert (device), else nullptr
  int has_prev, num_experts;
  int64_t w_expert_bytes, s_expert_stride;
};

int launch_i4(const Params& pp, int zmode, int src, int warps, int grid, cudaStream_t stream);
int launch_i8(const Params& pp, int zmode, int src, int warps, int grid, cudaStream_t stream);

#ifdef __CUDACC__

__device__ __forceinline__ uint4 ld_stream_v4(const void* p) {
  uint4 v;
  asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0, %1, %2, %3}, [%4];"
               : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
               : "l"(p));
  return v;
}
// Activations: not .nc, which is for memory that nothing writes while the kernel runs.  This kernel may be
// resident before they are written - by the kernel it waits for, or, behind two small grids, while the one
// before that still reads the same buffer on this SM.  Weights, scales and zero points are written by kernels
// that let no dependent start early.
__device__ __forceinline__ uint4 ld_x_v4(const void* p) {
  uint4 v;
  asm volatile("ld.global.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
  return v;
}
__device__ __forceinline__ uint2 ld_nc_v2(const void* p) {
  uint2 v;
  asm volatile("ld.global.nc.v2.u32 {%0, %1}, [%2];" : "=r"(v.x), "=r"(v.y) : "l"(p));
  return v;
}
__device__ __forceinline__ void prefetch_l2(const void* p) {
  asm volatile("prefetch.global.L2 [%0];" ::"l"(p));
}

// Grouped form: the (expert, up to eight batch rows) pairs that have rows.
struct Entries {
  int count, m_lo[kMaxEntries], m_n[kMaxEntries], expert[kMaxEntries];
};
// ... from indptr (the whole CTA).
__device__ __forceinline__ void list_entries(const Params& pp, Entries& tab) {
  const int lane = threadIdx.x & 31;
  if (threadIdx.x < 32) {
    int n_e = 0;
    for (int e0 = 0; e0 < pp.num_experts; e0 += 32) {
      const int e = e0 + lane;
      int r0 = 0, r1 = 0;
      if (e < pp.num_experts) {
        r0 = (e || pp.has_prev) ? (int)pp.indptr[e - 1] : 0;
        r1 = min((int)pp.indptr[e], pp.g.m);  // never past the rows x / out hold
      }
      const int mine = r1 > r0 ? (r1 - r0 + kEntryRows - 1) / kEntryRows : 0;
      int incl = mine;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += v;
      }
      for (int i = 0; i < mine; ++i) {
        const int slot = n_e + incl - mine + i;
        if (slot < kMaxEntries) {
          tab.m_lo[slot] = r0 + i * kEntryRows;
          tab.m_n[slot] = min(kEntryRows, r1 - r0 - i * kEntryRows);
          tab.expert[slot] = e;
        }
      }
      n_e += __shfl_sync(0xffffffffu, incl, 31);
    }
    if (lane == 0) tab.count = min(n_e, kMaxEntries);
  }
  __syncthreads();
}

template <int kXV, int MT>
struct XHalf {
  uint4 v[2][MT][kXV];
};

// kWarps: warps per CTA = k slices of a row block (16 warps per SM either way)
// MT: m-tiles of eight batch rows (MMA n)
template <int BITS, int ZMODE, int SRC, bool GROUPED, int kWarps, int MT>
__global__ void __launch_bounds__(kWarps * 32, 16 / kWarps) gemv_rk_kernel(const Params pp) {
  constexpr int kFrag = BITS == 4 ? 64 : 32;
  constexpr int kLaneK = kFrag / 4;
  constexpr int kXV = BITS == 4 ? 2 : 1;  // 16-byte pieces of x per lane and tile
  constexpr bool kZ = ZMODE == kZeroGeneral;
  constexpr int kRows = pass_rows(SRC, ZMODE);
  constexpr bool kFold = folds(ZMODE, SRC, MT);
  constexpr bool kFoldAll = kFold && SRC == kChannel;  // the sums run over all of k
  __shared__ __align__(16) float4 red[2][kWarps][kRows * MT][32];
  __shared__ Entries tab;
  const GemvParams& p = pp.g;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int g = lane >> 2, t = lane & 3;
  const int NB = p.n / 16, KB = p.k / kFrag;
  constexpr bool grouped = GROUPED;

  griddep_launch_dependents();
  int entries = 1;
  if (grouped) {
    griddep_wait();  // the row table is the routing kernel's output
    list_entries(pp, tab);
    entries = tab.count;
  }
  // this CTA's row blocks, numbered entry by entry
  unsigned pos, pos_end;
  if (grouped) {
    const unsigned total = (unsigned)entries * (unsigned)NB;  // total * grid fits 32 bits (checked by the host)
    pos = blockIdx.x * total / gridDim.x;
    pos_end = (blockIdx.x + 1) * total / gridDim.x;
  } else {
    pos = blockIdx.x * pp.per_cta + min(blockIdx.x, pp.extra);
    pos_end = pos + pp.per_cta + (blockIdx.x < pp.extra ? 1u : 0u);
  }
  if (pos >= pos_end) return;

  const ZeroConsts zc = make_zero_consts(ZMODE, p.zero_const);
  const uint32_t zconst_h2 = h2_bcast(__float2half_rn(p.zero_const));
  const uint32_t half_sel = (t >> 1) ? 0x3232u : 0x1010u;
  const int unit16 = frag_unit_pos(lane) * 16;
  const bool has_zeros = kZ && p.z != nullptr;
  // kFold: the codes' units, and what the MMA's codes are reduced by (f16x2 of rows g, g + 8)
  constexpr float kUnitLo = 1.0f / (1 << 24), kUnitHi = BITS == 4 ? 16.0f * kUnitLo : kUnitLo;
  struct Zeros {
    uint32_t z[kRows];
    bool codes;  // in the codes' units, for all lanes and row blocks; else the zero points as they are
  };
  auto zeros_of = [&](const uint32_t (&z2)[kRows]) {
    Zeros z;
    bool fit = true;
#pragma unroll
    for (int r = 0; r < kRows; ++r) {
      bool f;
      z.z[r] = zero_in_codes<BITS>(z2[r], f);
      fit = fit && f;
    }
    z.codes = !kZ || __all_sync(0xffffffffu, fit);  // (kZeroConstInt: an integer)
    if (kZ && !z.codes)
#pragma unroll
      for (int r = 0; r < kRows; ++r) z.z[r] = z2[r];
    return z;
  };
  using CodeUnits = std::true_type;
  using PlainUnits = std::false_type;

  // this warp's whole chunks (four fragment tiles); the tiles of a short last chunk go to the last warp
  const int full_chunks = KB / 4;
  const int c0 = warp * full_chunks / kWarps, c1 = (warp + 1) * full_chunks / kWarps;

  // What a pass works on: up to two row blocks of one entry.
  struct Pass {
    int nb0, rn, m_lo, m_n, e;
  };
  auto get_pass = [&](unsigned at) {
    Pass q;
    const int entry = grouped ? (int)(at / (unsigned)NB) : 0;
    q.nb0 = (int)(at - (unsigned)entry * (unsigned)NB);
    // a short last row tile has another chunk stride: a pass stays on one side of it
    const int to_tile_end = 8 - (q.nb0 & 7);
    q.rn = min(min(kRows, (int)(pos_end - at)), min(NB - q.nb0, to_tile_end));
    q.e = grouped ? tab.expert[entry] : 0;
    q.m_lo = grouped ? tab.m_lo[entry] : 0;
    q.m_n = grouped ? tab.m_n[entry] : p.m;
    return q;
  };
  const int row8 = pp.s_n * 8;  // elements from row g's scale to row g + 8's

  // Two register sets, one per half of a chunk (two tiles of each row block); a set is loaded for the
  // next chunk as soon as it has been decoded, so a chunk per row block is always on its way.  The
  // row blocks of a pass lie in one 128-row tile, so one pointer and immediate offsets reach all of
  // a chunk's tiles.
  uint4 w[2][kRows][2];
  uint2 sv[2][kRows][2], zv[2][kRows][2];      // kRow32: rows g, g + 8: the half's four groups
  // kHalf, kTile, kGeneral: per half or tile, rows g, g + 8; a word each where registers allow it (as
  // one word they are waited for soon after their loads: int4 k 4096 x n 57344, group 128 36.6 -> 35.0 us)
  uint32_t sg[2][kRows][2][2], zg[2][kRows][2];
  // kChannel: rows g, g + 8.  They are loaded before a pass's first weights and, as one word, waited for there, so
  // without zero points they are a word each (int4 k 4096 x n 22016, one row: 12.2 us as one word, 12.0 apart).  Beside
  // zero points that is so for int4 at nine to sixteen rows only (k = n = 4096, sixteen rows 6.37 / 6.16); int8 spills
  // 28 bytes there (k 4096 x n 22016, twelve rows 23.1 / 23.9; k 11008 x n 4096, sixteen 12.6 / 13.0), and at up to
  // eight rows one word is as fast or faster (int4 k = n = 4096, one row 4.24 / 4.33, n 22016 13.7 / 13.8).
  constexpr bool kApart = !kZ || (BITS == 4 && MT == 2);
  uint32_t ch_s[kRows][2], ch_z[kRows][2];  // kApart: rows g, g + 8; else both in the first
  // of row g (i = 0) or g + 8, twice; of both
  auto ch_twice = [](const uint32_t (&v)[2], int i) {
    const uint32_t w = kApart ? v[i] : v[0];
    return prmt(w, w, kApart || i == 0 ? 0x1010u : 0x3232u);
  };
  auto ch_both = [](const uint32_t (&v)[2]) { return kApart ? prmt(v[0], v[1], 0x5410u) : v[0]; };
  const uint8_t* wp = nullptr;                 // next chunk to load
  const __half *sp[kRows][2], *zp[kRows][2];   // scales of rows g, g + 8 (kRow32: of the next chunk)
  int stride = 0;                              // bytes from a chunk to the next
  unsigned s_at = 0u;                          // kHalf, kTile: offset of the next group's scales, and what
  int s_left = 0;                              // is left of that group

  auto load_set = [&](auto set_tag, auto rn_tag, int c) {
    constexpr int S = decltype(set_tag)::value, RN = decltype(rn_tag)::value;
    unsigned at[2];  // offsets of the groups' scales
    if (SRC == kHalf || SRC == kTile) {
#pragma unroll
      for (int j = 0; j < (SRC == kHalf ? 1 : 2); ++j) {
        at[j] = s_at;
        if (--s_left == 0) {
          s_left = pp.per;
          s_at += (unsigned)pp.s_g;
        }
      }
    }
#pragma unroll
    for (int r = 0; r < RN; ++r) {
      w[S][r][0] = ld_stream_v4(wp + r * 2048 + S * 1024);
      w[S][r][1] = ld_stream_v4(wp + r * 2048 + S * 1024 + 512);
      if (SRC == kRow32) {
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          sv[S][r][i] = ld_nc_v2(sp[r][i] + S * 4);
          if (has_zeros) zv[S][r][i] = ld_nc_v2(zp[r][i] + S * 4);
        }
      } else if (SRC == kHalf || SRC == kGeneral || SRC == kTile) {
#pragma unroll
        for (int j = 0; j < (SRC == kHalf ? 1 : 2); ++j) {
          unsigned o = 0u;
          if (SRC != kGeneral) {
            o = at[j];
          } else {
            const unsigned k = (unsigned)((c * 4 + S * 2 + j) * kFrag + t * kLaneK);
            o = (pp.group_shift >= 0 ? k >> pp.group_shift : k / (unsigned)p.group) * (unsigned)pp.s_g;
          }
          const uint32_t a = ld_nc_u16(sp[r][0] + o), b = ld_nc_u16(sp[r][1] + o);
          sg[S][r][j][0] = kFold ? a : a | (b << 16);
          sg[S][r][j][1] = b;
          if (has_zeros) {
            const uint32_t za = ld_nc_u16(zp[r][0] + o), zb = ld_nc_u16(zp[r][1] + o);
            zg[S][r][j] = za | (zb << 16);
          }
        }
      }
    }
    if (S == 1) {
      wp += stride;
      if (SRC == kRow32) {
#pragma unroll
        for (int r = 0; r < RN; ++r)
#pragma unroll
          for (int i = 0; i < 2; ++i) {
            sp[r][i] += 8;
            if (has_zeros) zp[r][i] += 8;
          }
      }
    }
  };
  using I0 = std::integral_constant<int, 0>;
  using I1 = std::integral_constant<int, 1>;
  using I2 = std::integral_constant<int, 2>;
  auto start_pass = [&](const Pass& q) {
    stride = min(8, NB - (q.nb0 & ~7)) * 2048;
    wp = p.w + (grouped ? q.e * pp.w_expert_bytes : 0) + 
         (int64_t)((q.nb0 & ~7) * KB + c0 * (stride >> 9) + (q.nb0 & 7) * 4) * 512 + unit16;
#pragma unroll
    for (int r = 0; r < kRows; ++r) {
      const int nb = q.nb0 + min(r, q.rn - 1);
      const int64_t o = (grouped ? q.e * pp.s_expert_stride : 0) + (nb * 16 + g) * pp.s_n + (SRC == kRow32 ? c0 * 8 : 0);
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        sp[r][i] = p.s + o + i * row8;
        zp[r][i] = p.z + o + i * row8;
      }
      if (SRC == kChannel) {
        const uint32_t a = ld_nc_u16(sp[r][0]), b = ld_nc_u16(sp[r][1]);
        ch_s[r][0] = kApart ? a : a | (b << 16);
        ch_s[r][1] = b;
        if (has_zeros) {
          const uint32_t za = ld_nc_u16(zp[r][0]), zb = ld_nc_u16(zp[r][1]);
          ch_z[r][0] = kApart ? za : za | (zb << 16);
          ch_z[r][1] = zb;
        }
      }
    }
    if (SRC == kHalf || SRC == kTile) {
      const unsigned unit = (unsigned)c0 * (SRC == kHalf ? 2u : 4u), grp = unit / (unsigned)pp.per;
      s_at = grp * (unsigned)pp.s_g;
      s_left = pp.per - (int)(unit - grp * (unsigned)pp.per);
    }
    if (c0 < c1) {
      if constexpr (kRows == 2) {
        if (q.rn == 2) {
          load_set(I0{}, I2{}, c0);
          load_set(I1{}, I2{}, c0);
          return;
        }
      }
      load_set(I0{}, I1{}, c0);
      load_set(I1{}, I1{}, c0);
    }
  };

  // L2 prefetch: a lane asks for one of the 16 lines of either row block's chunk.  int8 tiles take a
  // third of the arithmetic of int4 tiles per byte, so there the loads need this lead to keep HBM
  // busy (k 8192 x n 28672: 54 -> 38 us).  For int4 it only costs instructions in one matmul (14.8 against
  // 13.7 us at k 4096 x n 22016), but an expert layer's weights are many times that, and its passes jump between
  // experts: eight experts, 16 rows, k 4096 x n 28672, one scale per row 80.5 -> 78.0 us.
  constexpr bool kLead = BITS == 8 || (GROUPED && kFoldAll && !kZ);
  const int ahead = min(kLeadChunks, c1 - c0);
  auto line_of = [&](const Pass& q, int c) -> const uint8_t* {
    const int st = min(8, NB - (q.nb0 & ~7)) * 4;
    return p.w + (grouped ? q.e * pp.w_expert_bytes : 0) +
           (int64_t)((q.nb0 & ~7) * KB + c * st + (q.nb0 & 7) * 4) * 512 + lane * 128;
  };
  uint32_t zconst_of[kRows];
#pragma unroll
  for (int r = 0; r < kRows; ++r) zconst_of[r] = zconst_h2;
  const Zeros zeros_const = zeros_of(zconst_of);
  Pass q = get_pass(pos);
  if (!grouped && pp.early) start_pass(q);
  if (kLead || !pp.early) {
    // before the wait: a prefetch returns nothing to this kernel, so it is safe whatever the previous
    // kernel still writes
    const uint8_t* line = line_of(q, c0);
    for (int c = 0; c < ahead; ++c, line += min(8, NB - (q.nb0 & ~7)) * 2048)
      if (lane < 16 * q.rn) prefetch_l2(line);
  }
  if (!grouped) griddep_wait();
  if (grouped || !pp.early) start_pass(q);

  // lanes of absent batch rows fetch row 0: their columns of the result are never stored
  auto x_of = [&](const Pass& q) { return p.x + (q.m_lo + (g < q.m_n ? g : 0)) * (unsigned)p.ldx + t * kLaneK; };
  // elements to the second m-tile's row
  auto x_next_of = [&](const Pass& q) { return MT > 1 && g + 8 < q.m_n ? 8u * (unsigned)p.ldx : 0u; };
  auto load_x_at = [&](XHalf<kXV, MT>& xv, const __half* at, unsigned x_next) {
#pragma unroll
    for (int j = 0; j < 2; ++j)
#pragma unroll
      for (int mt = 0; mt < MT; ++mt)
#pragma unroll
        for (int i = 0; i < kXV; ++i) xv.v[j][mt][i] = ld_x_v4(at + mt * x_next + j * kFrag + i * 8);
  };
  // int8, one scale per row: the first x of a pass leaves with its first weights (unlike read-only loads they
  // are not moved ahead of the barrier and the stores of the pass before: k 8192 x n 28672, eight rows,
  // 40.9 -> 38.0 us; the other forms have no registers for it)
  constexpr bool kXEarly = BITS == 8 && SRC == kChannel;
  XHalf<kXV, MT> x_first;
  if (kXEarly && c0 < c1) load_x_at(x_first, x_of(q) + c0 * (kFrag * 4), x_next_of(q));

  int buf = 0;
  for (;;) {
    constexpr int kChains = MT == 1 && (!kFold || kFoldAll) ? 2 : 1;  // independent MMA chains (two m-tiles are two already)
    float acc[kRows][kChains][MT][4];
#pragma unroll
    for (int r = 0; r < kRows; ++r)
#pragma unroll
      for (int i = 0; i < kChains; ++i)
#pragma unroll
        for (int mt = 0; mt < MT; ++mt)
#pragma unroll
          for (int c = 0; c < 4; ++c) acc[r][i][mt][c] = 0.0f;
    const __half* x0 = x_of(q);
    const unsigned x_next = x_next_of(q);

    auto mma_tile = [&](int r, const uint4& wv, uint32_t s_g, uint32_t s_g8, uint32_t z_g, uint32_t z_g8,
                        const uint4 (&xv)[MT][kXV]) {
      const uint32_t ww[4] = {wv.x, wv.y, wv.z, wv.w};
#pragma unroll
      for (int j = 0; j < 2 * kXV; ++j) {  // MMAs of the tile: four int4 words, two int8 word pairs
        uint32_t a[4];
        if (BITS == 4) decode_int4_word<ZMODE>(ww[j], zc, s_g, s_g8, z_g, z_g8, a);
        else decode_int8_pair<ZMODE>(ww[2 * (j & 1)], ww[2 * (j & 1) + 1], zc, s_g, s_g8, z_g, z_g8, a);
#pragma unroll
        for (int mt = 0; mt < MT; ++mt) {
          const uint4& x = xv[mt][j >> 1];
          mma_16816(acc[r][j % kChains][mt], a, (j & 1) ? x.z : x.x, (j & 1) ? x.w : x.y);
        }
      }
    };
    // kFold: d (+)= (u - z) x
    auto code_step = [&](auto units, float (&d)[MT][4], const uint4& wv, uint32_t z2, const uint4 (&xv)[MT][kXV], int j, bool first) {
      const uint32_t ww[4] = {wv.x, wv.y, wv.z, wv.w};
      const uint32_t z_g = prmt(z2, z2, 0x1010u), z_g8 = prmt(z2, z2, 0x3232u);
      uint32_t a[4];
      if (units) {
        if (BITS == 4) codes_int4_word(ww[j], z_g, z_g8, a);
        else codes_int8_pair(ww[2 * (j & 1)], ww[2 * (j & 1) + 1], z_g, z_g8, a);
      } else {
        constexpr uint32_t kOne = 0x3c003c00u;
        if (BITS == 4) decode_int4_word<ZMODE>(ww[j], zc, kOne, kOne, z_g, z_g8, a);
        else decode_int8_pair<ZMODE>(ww[2 * (j & 1)], ww[2 * (j & 1) + 1], zc, kOne, kOne, z_g, z_g8, a);
      }
#pragma unroll
      for (int mt = 0; mt < MT; ++mt) {
        const uint4& x = xv[mt][j >> 1];
        if (first && j == 0) mma_16816_first(d[mt], a, x.x, x.y);
        else mma_16816(d[mt], a, (j & 1) ? x.z : x.x, (j & 1) ? x.w : x.y);
      }
    };
    // acc += s * d, in the codes' units
    auto add_scaled = [&](auto units, int r, const float (&d)[MT][4], float s_g, float s_g8) {
      if (!units) {
        s_g *= kUnitLo;
        s_g8 *= kUnitHi;
      }
#pragma unroll
      for (int mt = 0; mt < MT; ++mt)
#pragma unroll
        for (int c = 0; c < 4; ++c) acc[r][0][mt][c] += (c < 2 ? s_g : s_g8) * d[mt][c];
    };
    auto half_of = [](uint32_t v, int hi) { return __half2float(__ushort_as_half((unsigned short)(hi ? v >> 16 : v & 0xffffu))); };
    const __half* xp = x0 + c0 * (kFrag * 4);
    // activations of either half: fetched half a chunk ahead by int8, and by int4 where that has the
    // registers and gains (scales of a half without zero points: k 4096 x n 57344 35.0 -> 33.9 us; one per
    // row 24.5 -> 25.2), else where they are used
    constexpr bool kXAhead = BITS == 8 || (kFold && SRC == kHalf && !kZ);
    XHalf<kXV, MT> x_here, xb;
    XHalf<kXV, MT>& xa = kXEarly ? x_first : x_here;
    auto load_x = [&](XHalf<kXV, MT>& xv, int half) { load_x_at(xv, xp + half * (2 * kFrag), x_next); };
    Zeros ch_zeros = zeros_const;  // kFoldAll
    if (kFoldAll && has_zeros) {
      uint32_t z2[kRows];
#pragma unroll
      for (int r = 0; r < kRows; ++r) z2[r] = ch_both(ch_z[r]);
      ch_zeros = zeros_of(z2);
    }
    auto in_units = [&](const Zeros& z, auto&& f) {
      if (!kZ || z.codes) f(CodeUnits{});
      else f(PlainUnits{});
    };
    auto half_step = [&](auto set_tag, auto rn_tag, const XHalf<kXV, MT>& xv) {
      constexpr int S = decltype(set_tag)::value, RN = decltype(rn_tag)::value;
      if constexpr (kFoldAll) {
        in_units(ch_zeros, [&](auto units) {
#pragma unroll
          for (int j = 0; j < 2; ++j)
#pragma unroll
            for (int i = 0; i < 2 * kXV; ++i)
#pragma unroll
              for (int r = 0; r < RN; ++r) code_step(units, acc[r][i % kChains], w[S][r][j], ch_zeros.z[r], xv.v[j], i, false);
        });
        return;
      } else if constexpr (kFold) {
        constexpr int kSpan = SRC == kHalf ? 2 : 1;  // tiles of a group (as far as the half goes)
#pragma unroll
        for (int part = 0; part < 2 / kSpan; ++part) {
          Zeros z = zeros_const;
          if (has_zeros) {
            uint32_t z2[kRows];
#pragma unroll
            for (int r = 0; r < kRows; ++r) z2[r] = zg[S][r < RN ? r : 0][part];
            z = zeros_of(z2);
          }
          in_units(z, [&](auto units) {
            float d[RN][MT][4];
#pragma unroll
            for (int j = part * kSpan; j < (part + 1) * kSpan; ++j)
#pragma unroll
              for (int i = 0; i < 2 * kXV; ++i)
#pragma unroll
                for (int r = 0; r < RN; ++r) code_step(units, d[r], w[S][r][j], z.z[r], xv.v[j], i, j == part * kSpan);
#pragma unroll
            for (int r = 0; r < RN; ++r) add_scaled(units, r, d[r], half_of(sg[S][r][part][0], 0), half_of(sg[S][r][part][1], 0));
          });
        }
        return;
      }
#pragma unroll
      for (int j = 0; j < 2; ++j)
#pragma unroll
        for (int r = 0; r < RN; ++r) {
          uint32_t s_g, s_g8, z_g = zconst_h2, z_g8 = zconst_h2;
          if (SRC == kRow32) {
            const uint32_t a = j == 0 ? sv[S][r][0].x : sv[S][r][0].y, b = j == 0 ? sv[S][r][1].x : sv[S][r][1].y;
            s_g = prmt(a, a, half_sel);
            s_g8 = prmt(b, b, half_sel);
            if (has_zeros) {
              const uint32_t za = j == 0 ? zv[S][r][0].x : zv[S][r][0].y, zb = j == 0 ? zv[S][r][1].x : zv[S][r][1].y;
              z_g = prmt(za, za, half_sel);
              z_g8 = prmt(zb, zb, half_sel);
            }
          } else if (SRC == kChannel) {
            s_g = ch_twice(ch_s[r], 0);
            s_g8 = ch_twice(ch_s[r], 1);
            if (has_zeros) {
              z_g = ch_twice(ch_z[r], 0);
              z_g8 = ch_twice(ch_z[r], 1);
            }
          } else {
            const uint32_t a = sg[S][r][SRC == kHalf ? 0 : j][0];
            s_g = prmt(a, a, 0x1010u);
            s_g8 = prmt(a, a, 0x3232u);
            if (has_zeros) {
              const uint32_t b = zg[S][r][SRC == kHalf ? 0 : j];
              z_g = prmt(b, b, 0x1010u);
              z_g8 = prmt(b, b, 0x3232u);
            }
          }
          mma_tile(r, w[S][r][j], s_g, s_g8, z_g, z_g8, xv.v[j]);
        }
    };
    Pass q_next;
    const bool more = pos + (unsigned)q.rn < pos_end;
    const uint8_t* line = nullptr;
    int line_step = stride;
    bool line_on = lane < 16 * q.rn;
    if constexpr (kLead) {
      q_next = get_pass(min(pos + (unsigned)q.rn, pos_end - 1));
      line = line_of(q, c0 + ahead);
    }
    auto all_chunks = [&](auto rn_tag) {
#pragma unroll 1
      for (int c = c0; c < c1; ++c) {
        const bool again = c + 1 < c1;
        if constexpr (kLead) {
          if (c + ahead == c1) {  // on into the next pass
            line = line_of(q_next, c0);
            line_step = min(8, NB - (q_next.nb0 & ~7)) * 2048;
            line_on = more && lane < 16 * q_next.rn;
          }
          if (line_on) prefetch_l2(line);
          line += line_step;
        }
        load_x(kXAhead ? xb : xa, kXAhead ? 1 : 0);
        half_step(I0{}, rn_tag, xa);
        if (again) load_set(I0{}, rn_tag, c + 1);
        if (kXAhead) {
          if (again) xp += kFrag * 4;
          if (!kXEarly || again) load_x(xa, 0);
        } else {
          load_x(xb, 1);
          xp += kFrag * 4;
        }
        half_step(I1{}, rn_tag, xb);
        if (again) load_set(I1{}, rn_tag, c + 1);
      }
    };
    if (c0 < c1) {
      if (kXAhead && !kXEarly) load_x(xa, 0);
      if constexpr (kRows == 2) {
        if (q.rn == 2) all_chunks(I2{});
        else all_chunks(I1{});
      } else {
        all_chunks(I1{});
      }
    }

    if (warp == kWarps - 1) {  // tiles of a short last chunk
      for (int kb = full_chunks * 4; kb < KB; ++kb) {
        uint4 xt[MT][kXV];
#pragma unroll
        for (int mt = 0; mt < MT; ++mt)
#pragma unroll
          for (int i = 0; i < kXV; ++i) xt[mt][i] = ld_x_v4(x0 + mt * x_next + kb * kFrag + i * 8);
        const unsigned k = (unsigned)(kb * kFrag + t * kLaneK);
        const unsigned grp = SRC == kChannel ? 0u : (pp.group_shift >= 0 ? k >> pp.group_shift : k / (unsigned)p.group);
#pragma unroll
        for (int r = 0; r < kRows; ++r) {
          if (r >= q.rn) break;
          const uint4 wt = ld_stream_v4(p.w + (grouped ? q.e * pp.w_expert_bytes : 0) +
                                        frag_tile_offset(q.nb0 + r, kb, NB, KB) + unit16);
          if (kFoldAll) {
            in_units(ch_zeros, [&](auto units) {
#pragma unroll
              for (int i = 0; i < 2 * kXV; ++i) code_step(units, acc[r][i % kChains], wt, ch_zeros.z[r], xt, i, false);
            });
            continue;
          }
          const int64_t o = (grouped ? q.e * pp.s_expert_stride : 0) + ((q.nb0 + r) * 16 + g) * pp.s_n +
                            grp * (unsigned)pp.s_g;
          const uint32_t a = ld_nc_u16(p.s + o), b = ld_nc_u16(p.s + o + row8);
          const uint32_t za = has_zeros ? ld_nc_u16(p.z + o) * 0x10001u : zconst_h2;
          const uint32_t zb = has_zeros ? ld_nc_u16(p.z + o + row8) * 0x10001u : zconst_h2;
          if (kFold) {
            uint32_t z2[kRows];
#pragma unroll
            for (int i = 0; i < kRows; ++i) z2[i] = prmt(za, zb, 0x5410u);
            const Zeros z = zeros_of(z2);
            in_units(z, [&](auto units) {
              float d[MT][4];
#pragma unroll
              for (int i = 0; i < 2 * kXV; ++i) code_step(units, d, wt, z.z[0], xt, i, true);
              add_scaled(units, r, d, half_of(a, 0), half_of(b, 0));
            });
            continue;
          }
          mma_tile(r, wt, a * 0x10001u, b * 0x10001u, za, zb, xt);
        }
      }
    }

    // the next pass's first loads leave before this one's sums are put together
    const Pass done = q;
    float done_s[kRows][2];  // kFoldAll: scales of the sums
#pragma unroll
    for (int r = 0; r < kRows; ++r)
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        done_s[r][i] = !kFoldAll ? 1.0f : (kApart ? half_of(ch_s[r][i], 0) : half_of(ch_s[r][0], i));
        if (kFoldAll && kZ && !ch_zeros.codes) done_s[r][i] *= i ? kUnitHi : kUnitLo;
      }
    pos += (unsigned)q.rn;
    if (more) {
      if constexpr (kLead) q = q_next;
      else q = get_pass(pos);
      start_pass(q);
      if (kXEarly && c0 < c1) load_x_at(x_first, x_of(q) + c0 * (kFrag * 4), x_next_of(q));
    }

    // the k slices meet in warp order
#pragma unroll
    for (int r = 0; r < kRows; ++r)
#pragma unroll
      for (int mt = 0; mt < MT; ++mt) {
        float f[4];
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          f[c] = acc[r][0][mt][c] + (kChains == 2 ? acc[r][kChains - 1][mt][c] : 0.0f);
          if (kFoldAll) f[c] *= done_s[r][c >> 1];
        }
        red[buf][warp][r * MT + mt][lane] = make_float4(f[0], f[1], f[2], f[3]);
      }
    __syncthreads();
    if (warp < done.rn * MT) {
      float v[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll
      for (int i = 0; i < kWarps; ++i) {
        const float4 f = red[buf][i][warp][lane];
        v[0] += f.x;
        v[1] += f.y;
        v[2] += f.z;
        v[3] += f.w;
      }
      if (kFold) {  // the codes' units
        v[0] *= 1.0f / kUnitLo;
        v[1] *= 1.0f / kUnitLo;
        v[2] *= 1.0f / kUnitHi;
        v[3] *= 1.0f / kUnitHi;
      }
      const int nb = done.nb0 + warp / MT, m8 = (warp % MT) * 8 + t * 2;
      if (p.epi.act == kActSwiglu) {
        // rows g / g + 8 of the block are gate_f / up_f of f = 8 nb + g (interleaved repack)
#pragma unroll
        for (int cc = 0; cc < 2; ++cc) {
          const int m = m8 + cc;
          if (m < done.m_n)
            p.out[(int64_t)(done.m_lo + m) * p.ldo + nb * 8 + g] = __float2half_rn(silu_mul(v[cc], v[cc + 2]));
        }
      } else {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const int m = m8 + (i & 1);
          const int64_t n = (int64_t)nb * 16 + g + (i >> 1) * 8;
          if (m < done.m_n)
            p.out[(int64_t)(done.m_lo + m) * p.ldo + n] = __float2half_rn(apply_epilogue(v[i], p.epi, done.m_lo + m, n));
        }
      }
    }
    if (!more) break;
    buf ^= 1;  // the next pass writes the other half, so one barrier per pass is enough
  }
}

template <int BITS, int ZMODE, int SRC>
int launch_inst(const Params& pp, int warps, int grid, cudaStream_t stream) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)grid, 1, 1);
  cfg.blockDim = dim3((unsigned)warps * 32, 1, 1);
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  // always a programmatic dependent: before its wait the kernel only prefetches, unless the host
  // switched launch overlap on
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
#define RB200_RK(GR, W, M) RB200_CUDA(cudaLaunchKernelEx(&cfg, gemv_rk_kernel<BITS, ZMODE, SRC, GR, W, M>, pp))
  // (those experts are all gemv_flat.cuh's)
  constexpr bool kExperts = !(BITS == 4 && ZMODE == kZeroConstInt && (SRC == kRow32 || SRC == kHalf));
  if (pp.indptr) {
    if constexpr (kExperts) {
      if (warps == 8) RB200_RK(true, 8, 1);
      else RB200_RK(true, 4, 1);
    } else {
      RB200_CHECK(false, "no expert kernel for this source of scales");
    }
  } else if (pp.g.m <= 8) {
    if (warps == 8) RB200_RK(false, 8, 1);
    else RB200_RK(false, 4, 1);
  } else {
    if (warps == 8) RB200_RK(false, 8, 2);
    else RB200_RK(false, 4, 2);
  }
#undef RB200_RK
  return 0;
}

template <int BITS, int SRC>
int launch_src(const Params& pp, int zmode, int warps, int grid, cudaStream_t stream) {
  return zmode == kZeroGeneral ? launch_inst<BITS, kZeroGeneral, SRC>(pp, warps, grid, stream)
                               : launch_inst<BITS, kZeroConstInt, SRC>(pp, warps, grid, stream);
}

template <int BITS>
int launch_bits(const Params& pp, int zmode, int src, int warps, int grid, cudaStream_t stream) {
  switch (src) {
    case kChannel:
      return launch_src<BITS, kChannel>(pp, zmode, warps, grid, stream);
    case kHalf:
      return launch_src<BITS, kHalf>(pp, zmode, warps, grid, stream);
    case kTile:
      return launch_src<BITS, kTile>(pp, zmode, warps, grid, stream);
  }
  if constexpr (BITS == 4) {
    if (src == kRow32) return launch_src<BITS, kRow32>(pp, zmode, warps, grid, stream);
  }
  return launch_src<BITS, kGeneral>(pp, zmode, warps, grid, stream);
}

#endif  // __CUDACC__

}  // namespace rk

// Host entry: 1 when offsets of scales or activations need more than 31 bits, 0 on launch, -1 on error.
// Ungrouped: 1 <= p.m <= 16.  Grouped (indptr != nullptr): p.m = total rows, at most 32.
int gemv_rk_run(const GemvParams& p, int bits, int zmode, int sm_count, const int64_t* indptr, int has_prev,
                int num_experts, int64_t w_expert_bytes, int64_t s_expert_stride, cudaStream_t stream);

}  // namespace rb200
