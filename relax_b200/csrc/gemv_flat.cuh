// Decode-path kernel for at most sixteen batch rows of int4: one sequence of units per warp.
//
// The small-batch kernel of gemv_rk.cuh works through row blocks two at a time and starts each pair anew: its
// loads are drained at a pass's end (two chunks of 256 k a warp at k 4096), the two-rounding decode of groups of
// 32 takes 13 instructions a word, and a scale or zero point is a 16-bit load of its own.  Here a warp's work is
// one sequence of units (row block, chunk), always two of them loaded ahead whatever row block they belong to,
// and
//   * sums of up to eight row blocks wait in shared memory, so that the warps of a CTA meet once;
//   * u - z goes into the MMA in the codes' units and the scale is applied to the fp32 sums of a group (see
//     folds() in gemv_rk.cuh), for groups of 32 too: an MMA's k slots reach over a whole tile, two groups, so
//     the MMA's eight columns are up to four batch rows of the tile's first group beside the same rows of its
//     second (a lane's x is zero where its k belong to the other group); five to eight rows have the lanes
//     exchange half of their words, so that an MMA's k are of one group (eight instructions a tile more);
//   * the groups of a chunk are one load of each row where they lie side by side ([N, K/g]);
//   * a column without a batch row is never loaded (zeros stay in its registers): with the absent rows read as
//     row 0 the loads of x took 70 % of what L1 passes on, now 20 %;
//   * k may end within a chunk (k % 256 != 0): the last unit of a row block is shorter.
// Zero points that are not integers do not fit the codes' units.  The loop takes what fits of them, and a warp that met one
// adds the rest to its sums before they are put together (add_fractions, never reached with integers).
//
// Bound: instruction issue and latency, then HBM.  Of 65 instructions a 512-byte tile needs 36 are the codes, 4
// MMAs, 8 the scales; issue slots are half used and a warp mostly waits for its weights, but a third set of loads
// in flight gave nothing, nor did L2 prefetches ahead of them, and with four warps a CTA instead of eight it was
// up to 17 % slower.  Without the codes' arithmetic the loads alone would take 25 % less (k 4096 x n 22016).
// Nine to sixteen rows are two m-tiles with two tiles of x in registers instead of four; their loads of x take 128 of
// L1's clocks a unit, more than the arithmetic.
// Replacing the subtraction of z by z times the sums of x, kept in shared memory, needed 12 % fewer
// instructions and was 5 to 15 % slower: the sums come before the first unit.
//
// Measured against the two-row-block kernel (graphs of launches over 300 MB of weights, launch overlap on; us):
//                                   one row          four rows        eight rows       sixteen rows
//   group 32, k = n = 4096          4.19 / 3.83      4.57 / 3.97      (stays there)
//   group 32, k 4096 x n 22016      14.6 / 12.2      15.4 / 12.3
//   group 32, k 5504 x n 4096       8.2 / 5.1        8.5 / 5.2        8.6 / 6.5        10.6 / 8.9
//   the same with zero points       9.1 / 5.7        9.4 / 6.0        9.6 / 7.3
//   group 32 + z, k 4096 x n 22016  20.1 / 13.2      20.9 / 13.5      21.3 / 16.9
//   group 64 + z, k 4096 x n 22016  23.4 / 13.5      24.3 / 14.0      24.8 / 15.1      (without overlap 31.1 / 22.2)
//   group 128, k 11008 x n 4096     7.7 / 7.2        8.1 / 7.5        (stays there)    11.7 / 10.7
//   group 128 + z [K/g, N], x 11008 11.0 / 8.7       11.6 / 9.1       11.6 / 9.9
#pragma once

#include "gemv_rk.cuh"

namespace rb200 {
namespace fl {

constexpr int kWarps = 8;  // k slices of a row block; two CTAs per SM

// Beside rk::ScaleSrc: [N, K/g] with groups of 64 or 128, the groups of a chunk are one load of each row.
constexpr int kRow64 = 5, kRow128 = 6;
// Groups of 32 as rk::kRow32, for more than four rows.
constexpr int kRow32Wide = 7;

struct Params : rk::Params {
  unsigned s_last;  // offset of the last group's scales
};

// Where this kernel takes its scales from for these operands, or -1: the kernel of gemv_rk.cuh.
int source(const rk::Params& pp, int bits, int zmode, int src, int sm_count);
int launch(const rk::Params& pp, int zmode, int src, int grid, cudaStream_t stream);  // (grouped where pp.indptr is set)

#ifdef __CUDACC__

// Loads that keep the register's value where they are switched off.
__device__ __forceinline__ void ld_w_if(uint4& v, const void* p, bool on) {
  asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.s32 q, %5, 0;\n\t"
               "@q ld.global.nc.L1::no_allocate.v4.u32 {%0, %1, %2, %3}, [%4];\n\t}"
               : "+r"(v.x), "+r"(v.y), "+r"(v.z), "+r"(v.w)
               : "l"(p), "r"((int)on));
}
// (not .nc: see ld_x_v4 in gemv_rk.cuh)
__device__ __forceinline__ void ld_x_if(uint4& v, const void* p, bool on) {
  asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.s32 q, %5, 0;\n\t"
               "@q ld.global.v4.u32 {%0, %1, %2, %3}, [%4];\n\t}"
               : "+r"(v.x), "+r"(v.y), "+r"(v.z), "+r"(v.w)
               : "l"(p), "r"((int)on));
}
__device__ __forceinline__ void ld_nc_if(uint4& v, const void* p, bool on) {
  asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.s32 q, %5, 0;\n\t"
               "@q ld.global.nc.v4.u32 {%0, %1, %2, %3}, [%4];\n\t}"
               : "+r"(v.x), "+r"(v.y), "+r"(v.z), "+r"(v.w)
               : "l"(p), "r"((int)on));
}
__device__ __forceinline__ void ld_nc_if(uint2& v, const void* p, bool on) {
  asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.s32 q, %3, 0;\n\t@q ld.global.nc.v2.u32 {%0, %1}, [%2];\n\t}"
               : "+r"(v.x), "+r"(v.y)
               : "l"(p), "r"((int)on));
}
__device__ __forceinline__ void ld_nc_if(uint32_t& v, const void* p, bool on) {
  asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.s32 q, %2, 0;\n\t@q ld.global.nc.u32 %0, [%1];\n\t}"
               : "+r"(v)
               : "l"(p), "r"((int)on));
}
// (straight into 32 bits: a conversion beside the load is waited for there)
__device__ __forceinline__ void ld_nc16_if(uint32_t& v, const void* p, bool on) {
  asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.s32 q, %2, 0;\n\t@q ld.global.nc.u16 %0, [%1];\n\t}"
               : "+r"(v)
               : "l"(p), "r"((int)on));
}
__device__ __forceinline__ uint32_t word(const uint4& v, int i) { return i == 0 ? v.x : i == 1 ? v.y : i == 2 ? v.z : v.w; }
__device__ __forceinline__ float half_lo(uint32_t v) { return __half2float(__ushort_as_half((unsigned short)v)); }
__device__ __forceinline__ float2 halves(uint32_t v) { return __half22float2(*reinterpret_cast<const __half2*>(&v)); }

constexpr float kUnitLo = 1.0f / (1 << 24), kUnitHi = 16.0f * kUnitLo;  // the codes' units, rows g and g + 8

// What run_blocks works on: the CTA's row blocks of the call's weight, straight from the parameters (as plain fields
// of a run, like an expert's, they cost groups of 128 two to five per cent) ...
struct Call {
  static constexpr bool kWait = true;  // the previous kernel has to be waited for
  const GemvParams& p;
  int pos, blocks;
  __device__ const uint8_t* w() const { return p.w; }
  __device__ const __half* s() const { return p.s; }
  __device__ const __half* z() const { return p.z; }
  __device__ const __half* x() const { return p.x; }
  __device__ __half* out() const { return p.out; }
  __device__ int m() const { return p.m; }
  __device__ int row(int i) const { return i; }
};
// ... or of one entry of an expert layer.
struct Share {
  static constexpr bool kWait = false;
  const uint8_t* w_;
  const __half *s_, *z_, *x_;
  __half* out_;
  int m_, m0, pos, blocks;
  __device__ const uint8_t* w() const { return w_; }
  __device__ const __half* s() const { return s_; }
  __device__ const __half* z() const { return z_; }
  __device__ const __half* x() const { return x_; }
  __device__ __half* out() const { return out_; }
  __device__ int m() const { return m_; }
  __device__ int row(int i) const { return m0 + i; }
};

constexpr int vals(int src) { return src == rk::kRow32 ? 2 : 4; }  // sums of a lane, row block and m-tile

// D(16x8) += A(16x8 tf32) * B(8x8 tf32): row g, columns t, t + 4 of A and rows t, t + 4, column g of B by lane
__device__ __forceinline__ void mma_1688(float (&d)[4], const float (&a)[4], float b0, float b1) {
  asm volatile("mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
               : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
               : "r"(__float_as_uint(a[0])), "r"(__float_as_uint(a[1])), "r"(__float_as_uint(a[2])), "r"(__float_as_uint(a[3])),
                 "r"(__float_as_uint(b0)), "r"(__float_as_uint(b1)));
}
__device__ __forceinline__ float tf32_of(float v) { return __uint_as_float(__float_as_uint(v) & 0xffffe000u); }

// A zero point that is no integer fits the codes' units but for a fraction (of row g + 8, whose units are finer, for what
// is left of sixteenths): z = r + f, sum (u - z) x = sum (u - r) x - f sum x.  The loop has the first part, this adds the
// second to a warp's sums of `count` row blocks, from x, the scales and the zero points and without the weights.  Sums of x
// of a chunk's tiles (groups of 32: of each group) come out of MMAs with a column of ones each in the places of the B of a
// product with -f s (tf32: x in two parts, the fraction, a few per cent of the result, rounded to 11 bits).  k blocks kb0 to
// kb1; x (this lane's sixteen k of a tile), its row eight further and the scales and zero points of the first block's row g.
// Bound: L1, which passes x on once more for each window of row blocks.  Reading and decoding the weights again instead, with
// fractions everywhere (before / now; with integers; gemv_rk.cuh's kernel, which decodes either), us: k 4096 x n 22016, groups
// of 64, one row 43.2 / 17.3; 13.8; 30.3, sixteen rows 76.1 / 33.2; 22.2; 31.2, groups of 32, eight rows 49.1 / 23.1; 18.6;
// 21.9; k = n = 4096, groups of 32, one row 10.2 / 6.3; 4.8; 5.4, eight rows 11.4 / 8.0; 5.9; 6.0, groups of 128 10.1 / 6.9;
// 4.8; 6.0.  One fraction in the whole weight, groups of 128, k 4096 x n 22016, one row: 30.4 / 13.4; 13.0; 16.3.
struct Fractions {
  const __half *x, *x8, *s, *z;
  const uint8_t* w;
  int kb0, kb1, first, count, NB, KB, s_n, s_g, group, group_shift;
};
// Where an activation is not finite its product with u - r is none where the code is r (0 inf) and u - z is not 0: those sums
// anew, from u - z itself.
template <int SRC, int MT>
__device__ __noinline__ void sums_of_infinities(Fractions a, float (*red)[kWarps][32 * vals(SRC)]) {
  constexpr bool kPairs = SRC == rk::kRow32, k32 = kPairs || SRC == kRow32Wide;
  const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const ZeroConsts zc = make_zero_consts(kZeroGeneral, 0.0f);
#pragma unroll 1
  for (int i = 0; i < a.count * MT; ++i) {
    const int b = i / MT;
    const __half* x = MT > 1 && (i & 1) ? a.x8 : a.x;
    float acc[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll 1
    for (int kb = a.kb0; kb < a.kb1; ++kb, x += 64) {
      const uint4 w = rk::ld_stream_v4(a.w + frag_tile_offset(a.first + b, kb, a.NB, a.KB) + frag_unit_pos(lane) * 16);
#pragma unroll 1
      for (int q = 0; q < (SRC == kRow32Wide ? 2 : 1); ++q) {  // groups of 32: one at a time, or in columns of their own
        const bool mine = !k32 || (t >> 1) == (kPairs ? g & 1 : q);
        uint4 xv[2] = {make_uint4(0, 0, 0, 0), make_uint4(0, 0, 0, 0)};
        ld_x_if(xv[0], x, mine);
        ld_x_if(xv[1], x + 8, mine);
        const unsigned grp = (unsigned)(kb * 64) / (unsigned)a.group;
        float d[4], s[2][2];
        uint32_t z[2];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int64_t o = (int64_t)(b * 16 + 8 * h) * a.s_n + (int64_t)grp * a.s_g;
          z[h] = ld_nc_u16(a.z + o + (k32 ? t >> 1 : 0)) * 0x10001u;
          s[h][0] = half_lo(ld_nc_u16(a.s + o + (SRC == kRow32Wide ? q : 0)));
          s[h][1] = kPairs ? half_lo(ld_nc_u16(a.s + o + 1)) : s[h][0];
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          constexpr uint32_t kOne = 0x3c003c00u;
          uint32_t c[4];
          decode_int4_word<kZeroGeneral>(word(w, j), zc, kOne, kOne, z[0], z[1], c);
          if (SRC == kRow32Wide && !mine) c[0] = c[1] = c[2] = c[3] = 0u;  // (an infinite zero point of the other group)
          const uint4& xx = xv[j >> 1];
          if (j == 0) mma_16816_first(d, c, xx.x, xx.y);
          else mma_16816(d, c, (j & 1) ? xx.z : xx.x, (j & 1) ? xx.w : xx.y);
        }
#pragma unroll
        for (int c = 0; c < 4; ++c) acc[c] += (c < 2 ? kUnitLo : kUnitHi) * s[c >> 1][c & 1] * d[c];
      }
    }
    float* sum = &red[i][threadIdx.x >> 5][lane * vals(SRC)];
    if (kPairs) {
      sum[0] = acc[0] + acc[1];
      sum[1] = acc[2] + acc[3];
    } else {
#pragma unroll
      for (int c = 0; c < 4; ++c) sum[c] = acc[c];
    }
  }
}
template <int SRC, bool kTail, int MT>
__device__ __forceinline__ void add_fractions_inline(Fractions a, float (*red)[kWarps][32 * vals(SRC)]) {
  constexpr bool kPairs = SRC == rk::kRow32, k32 = kPairs || SRC == kRow32Wide;
  const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  float* const sums = &red[0][threadIdx.x >> 5][lane * vals(SRC)];
  constexpr int kBlock = MT * kWarps * 32 * vals(SRC);  // from a row block's sums to the next one's
  const uint32_t ones = (k32 ? (g & 1) == t >> 1 : !(g & 1)) ? 0x3c003c00u : 0u;
  const Fractions begin = a;
  bool finite = true;
#pragma unroll 1
  for (; a.kb0 < a.kb1; a.kb0 += 4, a.x += 256, a.x8 += 256) {
    // lane t has the scales and zero points of tile t
    const int kb = a.kb0 + t;
    const bool there = !kTail || kb < a.kb1;
    const unsigned o = k32 ? (unsigned)kb * 2u
                           : (a.group_shift >= 0 ? (unsigned)(kb * 64) >> a.group_shift : (unsigned)(kb * 64) / (unsigned)a.group) * (unsigned)a.s_g;
    const __half *sp = a.s + o, *zp = a.z + o;
    uint32_t s[2], z[2];  // rows g, g + 8
    auto load = [&]() {
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        if (kTail) s[i] = z[i] = 0u;
        if (k32) {
          ld_nc_if(s[i], sp + i * 8 * a.s_n, there);
          ld_nc_if(z[i], zp + i * 8 * a.s_n, there);
        } else {
          ld_nc16_if(s[i], sp + i * 8 * a.s_n, there);
          ld_nc16_if(z[i], zp + i * 8 * a.s_n, there);
        }
      }
      sp += 16 * a.s_n;
      zp += 16 * a.s_n;
    };
    load();
    float xh[MT][2], xl[MT][2];  // of tile t's groups
    {
      uint4 v[MT][4][2];
#pragma unroll
      for (int mt = 0; mt < MT; ++mt)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          if (kTail) v[mt][j][0] = v[mt][j][1] = make_uint4(0, 0, 0, 0);
          if (!kTail || a.kb0 + j < a.kb1) {
            v[mt][j][0] = rk::ld_x_v4((mt ? a.x8 : a.x) + j * 64);
            v[mt][j][1] = rk::ld_x_v4((mt ? a.x8 : a.x) + j * 64 + 8);
          }
        }
      // rows g of A are batch rows g, rows g + 8 batch rows g + 8 - or, in one m-tile, rows g of the next tile, so that
      // tiles of either parity are in rows of their own
      float d[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll
      for (int j = 0; j < 4; j += 3 - MT) {
        const uint32_t one = (MT == 1 ? g >> 2 == j >> 1 : g >> 1 == j) ? ones : 0u;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const uint4 &lo = v[0][j][i >> 1], &hi = v[MT - 1][j + 2 - MT][i >> 1];
          const uint32_t w[4] = {(i & 1) ? lo.z : lo.x, (i & 1) ? hi.z : hi.x, (i & 1) ? lo.w : lo.y, (i & 1) ? hi.w : hi.y};
          mma_16816(d, w, one, one);
        }
      }
#pragma unroll
      for (int mt = 0; mt < MT; ++mt)
#pragma unroll
        for (int q = 0; q < 2; ++q) {
          float sum = MT == 1 ? ((t & 1) ? d[2 + q] : d[q]) : d[2 * mt + q];
          if (kPairs && (g & 1) != q) sum = 0.0f;
          finite = finite && fabsf(sum) <= 3.4e38f;
          xh[mt][q] = tf32_of(sum);
          xl[mt][q] = sum - xh[mt][q];
        }
    }
    float* sum = sums;
#pragma unroll 1
    for (int left = a.count;; sum += kBlock) {
      float f[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll
      for (int q = 0; q < (k32 ? 2 : 1); ++q) {
        const float2 r = halves(zero_rest<4>(prmt(z[0], z[1], q ? 0x7632u : 0x5410u)));
        const float s0 = kUnitLo * half_lo(s[0] >> (16 * q)), s1 = kUnitHi * half_lo(s[1] >> (16 * q));
        if (r.x != 0.0f) f[2 * q] = __uint_as_float(__float_as_uint(-r.x * s0) + 0x1000u);
        if (r.y != 0.0f) f[2 * q + 1] = __uint_as_float(__float_as_uint(-r.y * s1) + 0x1000u);
      }
      const bool more = --left > 0;
      if (more) load();
#pragma unroll
      for (int mt = 0; mt < MT; ++mt) {
        float* at = sum + mt * (kBlock / MT);
        if (kPairs) {
          float2 v = *reinterpret_cast<float2*>(at);
          float d[4] = {v.x, 0.0f, v.y, 0.0f};
          mma_1688(d, f, xl[mt][0], xl[mt][1]);
          mma_1688(d, f, xh[mt][0], xh[mt][1]);
          *reinterpret_cast<float2*>(at) = make_float2(d[0] + d[1], d[2] + d[3]);
        } else {
          const float4 v = *reinterpret_cast<float4*>(at);
          float d[4] = {v.x, v.y, v.z, v.w};
          mma_1688(d, f, xl[mt][0], xl[mt][1]);
          mma_1688(d, f, xh[mt][0], xh[mt][1]);
          *reinterpret_cast<float4*>(at) = make_float4(d[0], d[1], d[2], d[3]);
        }
      }
      if (!more) break;
    }
  }
  if (!__all_sync(0xffffffffu, finite)) sums_of_infinities<SRC, MT>(begin, red);
}
// (Called for kRow32 and by experts: written into those kernels it cost integers 6 %, k 4096 x n 22016, one row, and 2 to 7 %;
// a call costs the others up to 10 % where there are fractions.)
template <int SRC, bool kTail, int MT>
__device__ __noinline__ void add_fractions_call(Fractions a, float (*red)[kWarps][32 * vals(SRC)]) {
  add_fractions_inline<SRC, kTail, MT>(a, red);
}

// kTail: k % 256 != 0; MT: m-tiles of eight batch rows
template <int ZMODE, int SRC, bool kTail, int MT, class Run>
__device__ __forceinline__ void run_blocks(const Params& pp, const Run& run, float (&red)[kWarps][kWarps][32 * vals(SRC)]) {
  using namespace rk;
  constexpr int kFrag = 64, kChunkK = 4 * kFrag;
  constexpr bool kZ = ZMODE == kZeroGeneral;
  constexpr bool kPairs = SRC == kRow32, kWide = SRC == kRow32Wide, k32 = kPairs || kWide, kChan = SRC == kChannel, kRow = SRC == kRow64 || SRC == kRow128;
  constexpr int kSpans = kChan ? 1 : SRC == kHalf || SRC == kRow128 ? 2 : 4, kSpan = 4 / kSpans;  // of a chunk; tiles of one
  constexpr bool kWords = k32 && (kZ || kTail);  // scales by words: lane t has tile t's (registers, alignment)
  constexpr int kVals = vals(SRC);
  constexpr int kSlots = kWarps / MT;  // row blocks whose sums wait in shared memory: [row block, m-tile]
  constexpr int kXTiles = MT == 1 ? 4 : 2;  // tiles of x in registers
  static_assert(MT == 1 || (!kPairs && !kChan), "");
  const GemvParams& p = pp.g;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int g = lane >> 2, t = lane & 3;
  const int NB = p.n / 16, KB = p.k / kFrag;
  const int pos = run.pos, blocks = run.blocks;
  const int chunks = (KB + 3) / 4, nkb_last = KB - (chunks - 1) * 4;
  const int c0 = warp * chunks / kWarps, nc = (warp + 1) * chunks / kWarps - c0;
  const bool ends_short = kTail && warp == kWarps - 1;  // (that warp has at least one chunk)
  const int unit16 = frag_unit_pos(lane) * 16;
  const int row8 = pp.s_n * 8;  // elements from row g's scale to row g + 8's

  // ---- loads: two register sets, each loaded again as it is used up
  uint4 w[2][4];
  uint4 sq[2][2];                               // kRow32: the chunk's groups of rows g, g + 8
  uint32_t sw[2][2], zw[2][2];                  // kRow32 by words: tile t's two groups of them
  uint2 sr[2][2], zr[2][2];                     // kRow64, kRow128: the chunk's groups
  uint32_t sg[2][kSpans][2], zg[2][kSpans][2];  // kHalf, kTile: one by one
  const uint8_t* wp;
  const __half *sp, *zp;
  int stride, left, lnb, to_load;
  unsigned s_at = 0, s_at0 = 0;  // kHalf, kTile: offset of the next group's scales, and what
  int s_left = 0, s_left0 = 0;   // is left of that group
  if (SRC == kHalf || SRC == kTile) {
    const unsigned unit = (unsigned)c0 * (unsigned)kSpans;
    const unsigned grp = pp.group_shift >= 0 ? (unsigned)(c0 * kChunkK) >> pp.group_shift : unit / (unsigned)pp.per;
    s_at0 = grp * (unsigned)pp.s_g;
    s_left0 = pp.per - (int)(unit - grp * (unsigned)pp.per);
  }
  auto aim = [&]() {  // at chunk c0 of row block lnb
    const int nblk = min(8, NB - (lnb & ~7));
    stride = nblk * 2048;
    wp = run.w() + (int64_t)((lnb & ~7) * KB + c0 * 4 * nblk + (lnb & 7) * (kTail && c0 == chunks - 1 ? nkb_last : 4)) * 512 + unit16;
  };
  auto start_at = [&](int block) {  // at the first unit of the CTA's block
    lnb = pos + block;
    to_load = (blocks - block) * nc;
    left = nc;
    aim();
    const int o = (lnb * 16 + g) * pp.s_n + (k32 ? c0 * 8 + (kWords ? 2 * t : 0) : kRow ? c0 * kSpans : 0);
    sp = run.s() + o;
    zp = kZ ? run.z() + o : nullptr;
    s_at = s_at0;
    s_left = s_left0;
  };
  auto advance = [&]() {
    constexpr int kStep = k32 ? 8 : kRow ? kSpans : 0;  // scales of a chunk
    --to_load;
    wp += stride;
    sp += kStep;
    if (kZ) zp += kStep;
    if (--left == 0) {
      left = nc;
      ++lnb;
      aim();  // (as cheap as stepping from one block to the next, which needs a branch at a tile's end)
      const int o = 16 * pp.s_n - nc * kStep;
      sp += o;
      if (kZ) zp += o;
      s_at = s_at0;
      s_left = s_left0;
    } else if (kTail && ends_short && left == 1) {
      wp -= (lnb & 7) * (4 - nkb_last) * 512;
    }
  };
  auto load_w = [&](auto set, int j, bool on) {
    constexpr int S = decltype(set)::value;
    ld_w_if(w[S][j], wp + j * 512, on && (!kTail || !ends_short || left > 1 || j < nkb_last));
  };
  auto load_s = [&](auto set, bool on) {
    constexpr int S = decltype(set)::value;
    if (k32 || kRow) {
      const bool there = on && (!kTail || !ends_short || left > 1 || t < nkb_last);
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        if (kWords) ld_nc_if(sw[S][i], sp + i * row8, there);
        else if (k32) ld_nc_if(sq[S][i], sp + i * row8, on);
        else if (SRC == kRow128) ld_nc_if(sr[S][i].x, sp + i * row8, on);
        else ld_nc_if(sr[S][i], sp + i * row8, on);
        if (!kZ) continue;
        if (kWords) ld_nc_if(zw[S][i], zp + i * row8, there);
        else if (SRC == kRow128) ld_nc_if(zr[S][i].x, zp + i * row8, on);
        else ld_nc_if(zr[S][i], zp + i * row8, on);
      }
    } else if (!kChan) {
#pragma unroll
      for (int q = 0; q < kSpans; ++q) {
        const unsigned o = kTail ? min(s_at, pp.s_last) : s_at;  // (behind the end of k the last group's once more)
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          ld_nc16_if(sg[S][q][i], sp + o + i * row8, on);
          if (kZ) ld_nc16_if(zg[S][q][i], zp + o + i * row8, on);
        }
        if (--s_left == 0) {
          s_left = pp.per;
          s_at += (unsigned)pp.s_g;
        }
      }
    }
  };
  using I0 = std::integral_constant<int, 0>;
  using I1 = std::integral_constant<int, 1>;
  auto load = [&](auto set) {
    const bool on = to_load > 0;
#pragma unroll
    for (int j = 0; j < 4; ++j) load_w(set, j, on);
    load_s(set, on);
    advance();
  };
  auto clear = [&]() {
#pragma unroll
    for (int S = 0; S < 2; ++S) {
#pragma unroll
      for (int j = 0; j < 4; ++j) w[S][j] = make_uint4(0, 0, 0, 0);
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        sq[S][i] = make_uint4(0, 0, 0, 0);
        sw[S][i] = zw[S][i] = 0;
        sr[S][i] = zr[S][i] = make_uint2(0, 0);
#pragma unroll
        for (int q = 0; q < kSpans; ++q) sg[S][q][i] = zg[S][q][i] = 0;
      }
    }
  };
  // What a sequence begins with.  With zero points it may have to begin again (below), so that these loads are the head of a
  // loop there; otherwise they leave as early as they can (1 to 2 % of a small matmul).
  auto first_weights = [&](int block) {
    start_at(block);
    clear();
    if (!Run::kWait || pp.early) {
      load(I0{});
      load(I1{});
    } else if (lane < 16) {
      // before the wait: a prefetch returns nothing to this kernel, so it is safe whatever the previous
      // kernel still writes
      const uint8_t* line = wp - unit16 + lane * 128;
      for (int c = 0; c < min(2, min(nc, KB / 4 - c0)); ++c, line += stride) prefetch_l2(line);
    }
    if (Run::kWait) griddep_wait();
    if (Run::kWait && !pp.early) {
      load(I0{});
      load(I1{});
    }
  };
  if (!kZ) first_weights(0);
  // kChannel: the scales of the row block whose sums this warp puts together
  uint32_t ch_s[2] = {0x3c00u, 0x3c00u};
  auto load_channel = [&](int first, int count) {
    if (kChan && warp < count) {
      const __half* s = run.s() + ((pos + first + warp) * 16 + g) * pp.s_n;
#pragma unroll
      for (int i = 0; i < 2; ++i) ld_nc16_if(ch_s[i], s + i * row8, true);
    }
  };
  int count = min(kSlots, blocks);
  load_channel(0, count);

  // ---- activations: each tile's are loaded for the next unit as it is used.  (No branch around the first
  // loads, that costs 5 % of a small matmul: a warp without chunks has no column.)
  const int m = kPairs ? g >> 1 : g;
  bool mine[MT];
#pragma unroll
  for (int mt = 0; mt < MT; ++mt) mine[mt] = m + 8 * mt < run.m() && nc > 0 && (!kPairs || (t >> 1) == (g & 1));
  const __half* const x0 = run.x() + (m < run.m() ? m : 0) * (unsigned)p.ldx + (kWide ? (t & 1) * 16 + (t >> 1) * 8 : t * 16) + c0 * kChunkK;
  const __half* xp;
  uint4 x[kXTiles][MT][2];
  auto clear_x = [&](int j) {
#pragma unroll
    for (int mt = 0; mt < MT; ++mt) x[j][mt][0] = x[j][mt][1] = make_uint4(0, 0, 0, 0);
  };
  auto load_x = [&](int j, bool last) {
    const bool there = !kTail || !ends_short || !last || j < nkb_last;
    if (kTail && MT > 1) clear_x(j % kXTiles);  // (one m-tile: before the short unit)
#pragma unroll
    for (int mt = 0; mt < MT; ++mt)
#pragma unroll
      for (int i = 0; i < 2; ++i)
        ld_x_if(x[j % kXTiles][mt][i], xp + mt * 8u * (unsigned)p.ldx + j * kFrag + i * (kWide ? 32 : 8), mine[mt] && there);
  };
  auto first_x = [&]() {
    xp = x0;
#pragma unroll
    for (int j = 0; j < kXTiles; ++j) {
      clear_x(j);
      load_x(j, nc == 1);
    }
  };
  if (!kZ) first_x();

  float acc[MT][4], acc2[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll
  for (int mt = 0; mt < MT; ++mt) acc[mt][0] = acc[mt][1] = acc[mt][2] = acc[mt][3] = 0.0f;
  int done_left = nc;  // chunks of the row block that are to be done
  uint32_t misfit = 0;  // not zero: a zero point was no integer
  uint32_t z_g, z_g8;
  auto set_zero = [&](uint32_t z2) {
    const uint32_t z = zero_in_codes<4>(z2, misfit);
    z_g = prmt(z, z, 0x1010u);
    z_g8 = prmt(z, z, 0x3232u);
  };
  if (!kZ) set_zero(h2_bcast(__float2half_rn(p.zero_const)));
  auto step = [&](auto set) {
    constexpr int S = decltype(set)::value;
    const bool on = to_load > 0;
    const bool this_last = done_left == 1, next_last = done_left == 2 || nc == 1;
    if constexpr (kTail && MT == 1) {
      if (ends_short && this_last) {
#pragma unroll
        for (int j = 1; j < 4; ++j)
          if (j >= nkb_last) clear_x(j);
      }
    }
    auto next_x = [&](int j) {  // after tile j: what takes its place
      if (j == 4 - kXTiles) xp = this_last ? x0 : xp + kChunkK;
      load_x((j + kXTiles) & 3, j + kXTiles < 4 ? this_last : next_last);
    };
    if constexpr (kWide) {
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        // Lanes t < 2 hold words of the tile's first group, the others of its second: they exchange two each, and every
        // MMA then sums over one group: lane t has the k from 16 (t & 1) + 8 (t >> 1) on of either.
        const bool hi = t >> 1;
        const uint4 v = w[S][j];
        const uint32_t r0 = __shfl_xor_sync(0xffffffffu, hi ? v.x : v.z, 2), r1 = __shfl_xor_sync(0xffffffffu, hi ? v.y : v.w, 2);
        const uint32_t ww[2][2] = {{hi ? r0 : v.x, hi ? r1 : v.y}, {hi ? v.z : r0, hi ? v.w : r1}};
        uint32_t za = 0, zb = 0, s2[2];
        if (kZ) {
          za = __shfl_sync(0xffffffffu, zw[S][0], j, 4);
          zb = __shfl_sync(0xffffffffu, zw[S][1], j, 4);
        }
#pragma unroll
        for (int i = 0; i < 2; ++i) s2[i] = kWords ? __shfl_sync(0xffffffffu, sw[S][i], j, 4) : word(sq[S][i], j);
#pragma unroll
        for (int q = 0; q < 2; ++q) {
          if (kZ) set_zero(prmt(za, zb, q ? 0x7632u : 0x5410u));
          float d[MT][4];
          uint32_t a[4];
          const uint4(&xx)[MT][2] = x[j % kXTiles];
          codes_int4_word(ww[q][0], z_g, z_g8, a);
#pragma unroll
          for (int mt = 0; mt < MT; ++mt) mma_16816_first(d[mt], a, xx[mt][q].x, xx[mt][q].y);
          codes_int4_word(ww[q][1], z_g, z_g8, a);
#pragma unroll
          for (int mt = 0; mt < MT; ++mt) mma_16816(d[mt], a, xx[mt][q].z, xx[mt][q].w);
          const float s_g = half_lo(s2[0] >> (q ? 16 : 0)), s_g8 = half_lo(s2[1] >> (q ? 16 : 0));
#pragma unroll
          for (int mt = 0; mt < MT; ++mt)
#pragma unroll
            for (int c = 0; c < 4; ++c) acc[mt][c] += (c < 2 ? s_g : s_g8) * d[mt][c];
        }
        load_w(set, j, on);
        next_x(j);
      }
      load_s(set, on);
      advance();
      return;
    }
#pragma unroll
    for (int q = 0; q < kSpans; ++q) {
      if (kZ) {
        if (kPairs) {
          const uint32_t a = __shfl_sync(0xffffffffu, zw[S][0], q, 4), b = __shfl_sync(0xffffffffu, zw[S][1], q, 4);
          set_zero(prmt(a, b, t >> 1 ? 0x7632u : 0x5410u));
        } else if (kRow) {
          const uint32_t a = q < 2 ? zr[S][0].x : zr[S][0].y, b = q < 2 ? zr[S][1].x : zr[S][1].y;
          set_zero(prmt(a, b, q & 1 ? 0x7632u : 0x5410u));
        } else {
          set_zero(zg[S][q][0] | (zg[S][q][1] << 16));
        }
      }
      float d[MT][4];
#pragma unroll
      for (int j = q * kSpan; j < (q + 1) * kSpan; ++j) {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          uint32_t a[4];
          codes_int4_word(word(w[S][j], i), z_g, z_g8, a);
#pragma unroll
          for (int mt = 0; mt < MT; ++mt) {
            const uint4& xx = x[j % kXTiles][mt][i >> 1];
            const uint32_t b0 = (i & 1) ? xx.z : xx.x, b1 = (i & 1) ? xx.w : xx.y;
            if (kChan) mma_16816(j & 1 ? acc2 : acc[mt], a, b0, b1);
            else if (i == 0 && j == q * kSpan) mma_16816_first(d[mt], a, b0, b1);
            else mma_16816(d[mt], a, b0, b1);
          }
        }
        load_w(set, j, on);
        next_x(j);
      }
      if (!kChan) {
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          const uint32_t one = kRow ? (q < 2 ? sr[S][i].x : sr[S][i].y) >> (q & 1 ? 16 : 0) : sg[S][q][i];
          const float2 s = !kPairs ? make_float2(half_lo(one), half_lo(one))
                                   : halves(kWords ? __shfl_sync(0xffffffffu, sw[S][i], q, 4) : word(sq[S][i], q));
#pragma unroll
          for (int mt = 0; mt < MT; ++mt) {
            acc[mt][2 * i] += s.x * d[mt][2 * i];
            acc[mt][2 * i + 1] += s.y * d[mt][2 * i + 1];
          }
        }
      }
    }
    load_s(set, on);
    advance();
  };

  // the sums of a row block are kept until kSlots blocks are done, or all
  int slot = 0, window = 0;
  auto window_done = [&]() {
    if (--done_left != 0) return false;
    if (kChan) {
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        acc[0][c] += acc2[c];
        acc2[c] = 0.0f;
      }
    }
#pragma unroll
    for (int mt = 0; mt < MT; ++mt) {
      float(&f)[4] = acc[mt];
      if (kPairs) *reinterpret_cast<float2*>(&red[slot][warp][lane * 2]) = make_float2(f[0] + f[1], f[2] + f[3]);
      else *reinterpret_cast<float4*>(&red[slot * MT + mt][warp][lane * 4]) = make_float4(f[0], f[1], f[2], f[3]);
      f[0] = f[1] = f[2] = f[3] = 0.0f;
    }
    done_left = nc;
    return ++slot == count;
  };
  // the k slices meet in warp order
  auto put_together = [&]() {
    if (warp >= count * MT) return;
    float v[kVals];
#pragma unroll
    for (int c = 0; c < kVals; ++c) v[c] = 0.0f;
#pragma unroll
    for (int i = 0; i < kWarps; ++i)
#pragma unroll
      for (int c = 0; c < kVals; ++c) v[c] += red[warp][i][lane * kVals + c];
#pragma unroll
    for (int c = 0; c < kVals; ++c) v[c] *= (c < kVals / 2 ? 1.0f / kUnitLo : 1.0f / kUnitHi) * half_lo(ch_s[c / (kVals / 2)]);
    const int nb = pos + window + warp / MT;
#pragma unroll
    for (int c = 0; c < kVals / 2; ++c) {
      const int mm = (warp % MT) * 8 + t * (kVals / 2) + c;
      if (mm >= run.m()) continue;
      const float lo = v[c], hi = v[c + kVals / 2];
      if (p.epi.act == kActSwiglu) {
        // rows g / g + 8 of the block are gate_f / up_f of f = 8 nb + g (interleaved repack)
        run.out()[(int64_t)mm * p.ldo + nb * 8 + g] = __float2half_rn(silu_mul(lo, hi));
      } else {
        const int64_t n = (int64_t)nb * 16 + g;
        run.out()[(int64_t)mm * p.ldo + n] = __float2half_rn(apply_epilogue(lo, p.epi, run.row(mm), n));
        run.out()[(int64_t)mm * p.ldo + n + 8] = __float2half_rn(apply_epilogue(hi, p.epi, run.row(mm), n + 8));
      }
    }
  };
  auto window_stored = [&]() {  // true: that was the last
    __syncthreads();
    put_together();
    window += count;
    if (window >= blocks) return true;
    count = min(kSlots, blocks - window);
    load_channel(window, count);
    slot = 0;
    __syncthreads();
    return false;
  };
  for (;;) {
    if (kZ) {
      first_weights(window);
      first_x();
    }
    bool odd = false;  // which set is next
    for (;;) {
      if (nc == 0) {
        for (int i = 0; i < count * MT; ++i)
#pragma unroll
          for (int v = 0; v < kVals; ++v) red[i][warp][lane * kVals + v] = 0.0f;
      } else {
#pragma unroll 1
        for (;;) {
          if (!odd) {
            step(I0{});
            odd = true;
            if (window_done()) break;
          }
          step(I1{});
          odd = false;
          if (window_done()) break;
        }
      }
      if (kZ && __any_sync(0xffffffffu, misfit != 0)) break;
      if (window_stored()) return;
    }
    // A zero point was no integer.  What is loaded ahead is loaded again: kept over this it would spill.
    const unsigned at = (unsigned)((pos + window) * 16 + g) * (unsigned)pp.s_n;
    const __half* xa = x0 + (kWide ? t * 16 - ((t & 1) * 16 + (t >> 1) * 8) : 0);
    const Fractions a = {xa, MT > 1 && mine[MT - 1] ? xa + 8u * (unsigned)p.ldx : xa, run.s() + at, run.z() + at, run.w(), c0 * 4,
                         min(KB, (c0 + nc) * 4), pos + window, count, NB, KB, pp.s_n, pp.s_g, p.group, pp.group_shift};
    if (kPairs || !Run::kWait) add_fractions_call<SRC, kTail, MT>(a, red);
    else add_fractions_inline<SRC, kTail, MT>(a, red);
    misfit = 0;
    if (window_stored()) return;
  }
}

template <int ZMODE, int SRC, bool kTail, int MT>
__global__ void __launch_bounds__(kWarps * 32, 2) gemv_flat_kernel(const Params pp) {
  __shared__ __align__(16) float red[kWarps][kWarps][32 * vals(SRC)];
  griddep_launch_dependents();
  const Call call = {pp.g, (int)(blockIdx.x * pp.per_cta + min(blockIdx.x, pp.extra)), (int)(pp.per_cta + (blockIdx.x < pp.extra ? 1u : 0u))};
  run_blocks<ZMODE, SRC, kTail, MT>(pp, call, red);
}

// Expert form: the row blocks of all entries (expert, up to eight of its rows) in one line, shared out evenly.
template <int ZMODE, int SRC, bool kTail>
__global__ void __launch_bounds__(kWarps * 32, 2) gemv_flat_experts_kernel(const Params pp) {
  __shared__ __align__(16) float red[kWarps][kWarps][32 * vals(SRC)];
  __shared__ rk::Entries tab;
  griddep_launch_dependents();
  griddep_wait();  // the row table is the routing kernel's output
  rk::list_entries(pp, tab);
  const unsigned NB = (unsigned)pp.g.n / 16u, total = (unsigned)tab.count * NB;  // total * grid fits 32 bits (checked by the host)
  unsigned at = blockIdx.x * total / gridDim.x;
  const unsigned end = (blockIdx.x + 1) * total / gridDim.x;
#pragma unroll 1
  while (at < end) {
    const unsigned i = at / NB, first = at - i * NB, count = min(end - at, NB - first);
    const int64_t so = tab.expert[i] * pp.s_expert_stride;
    const Share share = {pp.g.w + tab.expert[i] * pp.w_expert_bytes, pp.g.s + so, pp.g.z + so, pp.g.x + (int64_t)tab.m_lo[i] * pp.g.ldx,
                         pp.g.out + (int64_t)tab.m_lo[i] * pp.g.ldo, tab.m_n[i], tab.m_lo[i], (int)first, (int)count};
    run_blocks<ZMODE, SRC, kTail, 1>(pp, share, red);
    at += count;
    __syncthreads();
  }
}

#endif  // __CUDACC__

}  // namespace fl
}  // namespace rb200
