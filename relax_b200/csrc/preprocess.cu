// Weight repack into the fragment layout (see dequant.cuh), one 16 KB stage run per CTA pass.
// Stands in for fastertransformer::preprocess_weights as called by
// cutlass.ft_preprocess_weight (src/runtime/contrib/cutlass/weight_preprocess.cc:38-58): same
// byte size in and out, signed codes biased to unsigned, layout private to the matmul kernels.
#include "dequant.cuh"
#include "preprocess.h"

namespace rb200 {
namespace {

// Unsigned code of logical element (n, k) of one expert in the given source layout.
template <int BITS, int LAYOUT>
__device__ __forceinline__ uint32_t load_code(const uint8_t* src, int64_t n, int64_t k, int64_t K,
                                              int64_t N) {
  if (LAYOUT == 0) {  // FT: int8 container [K, N/2] (int4) or [K, N] (int8), signed
    if (BITS == 4) {
      uint32_t b = src[k * (N / 2) + (n >> 1)];
      return ((b >> ((n & 1) * 4)) & 15u) ^ 8u;  // two's-complement nibble + 8
    }
    return (uint32_t)src[k * N + n] ^ 0x80u;  // signed byte + 128
  }
  if (LAYOUT == 2) {  // AutoGPTQ: uint32 [K/8, N], nibble j of word (k/8, n) = element k = 8*(k/8) + j
    const uint32_t w = reinterpret_cast<const uint32_t*>(src)[(k >> 3) * N + n];
    return (w >> ((k & 7) * 4)) & 15u;
  }
  return 0;
}

// AutoGPTQ zero points: zq uint32 [G, N/8] (nibble j of word (g, n/8) = column 8*(n/8) + j) ->
// fp16 [G, N] holding f16(zq) + f16(1), the value the decode subtracts
// (tests/python/dlight/test_gpu_gemv.py:648).
// A thread per word: its eight columns are neighbours, 16 bytes where the output allows (with the
// repack, k 4096 x n 11008: 16.2 -> 11.0 us; a thread per column with two 64-bit divisions before).
__global__ void __launch_bounds__(256) unpack_zeros_autogptq_kernel(const uint32_t* zq, __half* out, int64_t words, bool vec) {
  griddep_wait();  // zero points are read like weights: no dependent may start before they are written
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < words; i += (int64_t)gridDim.x * blockDim.x) {
    const uint32_t q = zq[i];
    __align__(16) __half v[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) v[j] = __hadd(__int2half_rn((int)((q >> (4 * j)) & 15u)), __float2half_rn(1.0f));
    if (vec) {
      *reinterpret_cast<uint4*>(out + i * 8) = *reinterpret_cast<const uint4*>(v);
    } else {
#pragma unroll
      for (int j = 0; j < 8; ++j) out[i * 8 + j] = v[j];
    }
  }
}

// Gate/up interleave: the source holds gate rows [0, N/2) and up rows [N/2, N); fragment row block
// nb then takes gate rows 8nb..8nb+7 as its rows 0..7 and up rows 8nb..8nb+7 as its rows 8..15, so
// that one lane of the warp-MMA kernels (rows g and g+8) owns gate_f and up_f of the same f.
__host__ __device__ __forceinline__ int64_t gate_up_source_row(int64_t j, int64_t N) {
  const int64_t nb = j >> 4, r = j & 15;
  return r < 8 ? 8 * nb + r : N / 2 + 8 * nb + (r - 8);
}

template <int BITS, int LAYOUT>
__global__ void repack_kernel(const uint8_t* __restrict__ src, uint8_t* __restrict__ dst,
                              int64_t K, int64_t N, int64_t units_per_expert, int64_t total_units, int interleave,
                              const int32_t* __restrict__ k_perm) {
  constexpr int kFrag = BITS == 4 ? 64 : 32;
  const int64_t expert_bytes = K * N * BITS / 8;
  for (int64_t u = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; u < total_units;
       u += (int64_t)gridDim.x * blockDim.x) {
    // unit index -> (expert, row block, k block, lane): 32-bit divisions whenever the unit count
    // fits (64-bit ones are routines of a hundred instructions, three per 16 bytes moved)
    int64_t e, nb, kb;
    int lane;
    const int64_t KB = K / kFrag;
    if (total_units < (1ll << 31)) {
      const uint32_t u32 = (uint32_t)u, upe = (uint32_t)units_per_expert, kb32 = (uint32_t)KB;
      const uint32_t e32 = u32 / upe, r32 = u32 - e32 * upe;
      const uint32_t tile = r32 >> 5, nb32 = tile / kb32;
      e = e32;
      lane = (int)(r32 & 31u);
      nb = nb32;
      kb = tile - nb32 * kb32;
    } else {
      e = u / units_per_expert;
      const int64_t r = u % units_per_expert;
      lane = (int)(r & 31);
      const int64_t tile = r >> 5;
      nb = tile / KB;
      kb = tile % KB;
    }
    const int g = lane >> 2, t = lane & 3;
    const uint8_t* s = src + e * expert_bytes;
    uint32_t words[4];
    if (BITS == 4) {
      const int64_t k0 = kb * 64 + t * 16;
      // nibble slot p of a word <- (row offset, k offset inside the word's 4 k)
      const int row_of[8] = {0, 8, 0, 8, 0, 8, 0, 8};
      const int k_of[8] = {0, 0, 2, 2, 1, 1, 3, 3};
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        uint32_t w = 0;
#pragma unroll
        for (int p = 0; p < 8; ++p) {
          int64_t srow = nb * 16 + g + row_of[p];
          if (interleave) srow = gate_up_source_row(srow, N);
          int64_t ks = k0 + 4 * j + k_of[p];
          if (LAYOUT == 2 && k_perm) ks = k_perm[ks];  // act-order: k position -> source row
          uint32_t c = load_code<BITS, LAYOUT>(s, srow, ks, K, N);
          w |= c << (4 * p);
        }
        words[j] = w;
      }
    } else {
      const int64_t k0 = kb * 32 + t * 8;
#pragma unroll
      for (int j = 0; j < 2; ++j)
#pragma unroll
        for (int r8 = 0; r8 < 2; ++r8) {
          uint32_t w = 0;
#pragma unroll
          for (int c4 = 0; c4 < 4; ++c4) {
            int64_t srow = nb * 16 + g + 8 * r8;
            if (interleave) srow = gate_up_source_row(srow, N);
            w |= load_code<BITS, LAYOUT>(s, srow, k0 + 4 * j + c4, K, N) << (8 * c4);
          }
          words[2 * j + r8] = w;
        }
    }
    reinterpret_cast<uint4*>(dst + e * expert_bytes + frag_tile_offset(nb, kb, N / 16, KB))[frag_unit_pos(lane)] = make_uint4(words[0], words[1], words[2], words[3]);
  }
}

// 4x4 byte transpose: out[m] = bytes m of in[0..3]
__device__ __forceinline__ void transpose_bytes4(uint32_t a, uint32_t b, uint32_t c, uint32_t d, uint32_t (&out)[4]) {
  const uint32_t ab0 = prmt(a, b, 0x5140u), cd0 = prmt(c, d, 0x5140u);
  const uint32_t ab1 = prmt(a, b, 0x7362u), cd1 = prmt(c, d, 0x7362u);
  out[0] = prmt(ab0, cd0, 0x5410u);
  out[1] = prmt(ab0, cd0, 0x7632u);
  out[2] = prmt(ab1, cd1, 0x5410u);
  out[3] = prmt(ab1, cd1, 0x7632u);
}

// The repack proper.  Bound: HBM, every byte read once and written once.  One CTA pass makes one
// stage run of the destination (128 output rows x 4 k-blocks, 16 KB contiguous): a thread owns
// the 16 rows x (16 | 8) k of one (row block, k-block, lane group t), fetches them with 8 or 16
// independent vector loads that fill whole 32-byte sectors in every source layout, transposes
// in registers (nibbles: one masked swap and two byte permutes; bytes: two permutes), stages its
// eight 16-byte units in shared memory and the CTA streams the run out with full lines.  The
// earlier forms gathered code by code (150 instructions per 16 bytes) and were bound by
// instruction issue.
// Measured, k 8192 x n 28672, source + destination bytes: q4f16_1 45 us (5.2 TB/s), AutoGPTQ 54 us,
// FT int4 46 us (5.1 TB/s; 3.6 before), FT int8 90 us (5.2 TB/s).
template <int BITS, int LAYOUT, bool GATE_UP>
__global__ void __launch_bounds__(128) repack_stage_kernel(const uint8_t* src, uint8_t* dst,
                                                           int64_t K, int64_t N, uint32_t tiles, uint32_t chunks,
                                                           uint32_t total) {
  constexpr int kFrag = BITS == 4 ? 64 : 32;
  constexpr uint32_t kLow = 0x0f0f0f0fu;
  __shared__ __align__(16) uint4 run[1024];
  const int tid = threadIdx.x;
  const int t = tid & 3, b = (tid >> 2) & 7, kbl = tid >> 5;
  const int64_t KB = K / kFrag, NB = N / 16;
  const int64_t expert_bytes = K * N * BITS / 8;
  griddep_wait();  // a programmatic dependent (of the quantiser, when a model is loaded) that lets none start early
  for (uint32_t st = blockIdx.x; st < total; st += gridDim.x) {
    // neighbours in flight share the source's contiguous axis: n for [K, N] layouts, k for [N, K]
    uint32_t e, tile, chunk;
    if (LAYOUT == 1) {
      const uint32_t q = st / chunks;
      chunk = st - q * chunks;
      e = q / tiles;
      tile = q - e * tiles;
    } else {
      const uint32_t q = st / tiles;
      tile = st - q * tiles;
      e = q / chunks;
      chunk = q - e * chunks;
    }
    const int nblk = (int)min((int64_t)8, NB - (int64_t)tile * 8);
    const int nkb = (int)min((int64_t)4, KB - (int64_t)chunk * 4);
    const bool active = b < nblk && kbl < nkb;
    uint4 unit[8];
    if (active) {
      const uint8_t* s = src + e * expert_bytes;
      const int64_t nb = (int64_t)tile * 8 + b, kb = (int64_t)chunk * 4 + kbl;
      const int64_t n_lo = GATE_UP ? 8 * nb : 16 * nb;           // source rows of fragment rows 0..7
      const int64_t n_hi = GATE_UP ? N / 2 + 8 * nb : 16 * nb + 8;  // and 8..15
      if (LAYOUT == 0 && BITS == 4) {
        // [K, N/2] bytes: k rows of 16 nibbles, eight each from the lo and hi rows
        const int64_t pitch = N / 2;
        const uint8_t* q = s + (kb * 64 + t * 16) * pitch;
        uint2 v[16];
#pragma unroll
        for (int i = 0; i < 16; ++i) {
          if (GATE_UP) {
            v[i].x = *(reinterpret_cast<const uint32_t*>(q + i * pitch + n_lo / 2));
            v[i].y = *(reinterpret_cast<const uint32_t*>(q + i * pitch + n_hi / 2));
          } else {
            v[i] = *(reinterpret_cast<const uint2*>(q + i * pitch + n_lo / 2));
          }
        }
        uint32_t w[4][8];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          // byte pairs of the word in slot order k, k + 2, k + 1, k + 3; row g low, row g + 8 high
          uint32_t ev[4], od[4];
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const uint2 r = v[4 * j + (i == 1 ? 2 : (i == 2 ? 1 : i))];
            ev[i] = ((r.x & kLow) | ((r.y << 4) & ~kLow)) ^ 0x88888888u;
            od[i] = (((r.x >> 4) & kLow) | (r.y & ~kLow)) ^ 0x88888888u;
          }
          uint32_t oe[4], oo[4];
          transpose_bytes4(ev[0], ev[1], ev[2], ev[3], oe);
          transpose_bytes4(od[0], od[1], od[2], od[3], oo);
#pragma unroll
          for (int m = 0; m < 4; ++m) {
            w[j][2 * m] = oe[m];
            w[j][2 * m + 1] = oo[m];
          }
        }
#pragma unroll
        for (int g = 0; g < 8; ++g) unit[g] = make_uint4(w[0][g], w[1][g], w[2][g], w[3][g]);
      } else if (LAYOUT == 0) {
        // [K, N] bytes
        const uint8_t* q = s + (kb * 32 + t * 8) * N;
        uint4 v[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          if (GATE_UP) {
            const uint2 lo = *(reinterpret_cast<const uint2*>(q + i * N + n_lo));
            const uint2 hi = *(reinterpret_cast<const uint2*>(q + i * N + n_hi));
            v[i] = make_uint4(lo.x, lo.y, hi.x, hi.y);
          } else {
            v[i] = *(reinterpret_cast<const uint4*>(q + i * N + n_lo));
          }
        }
        uint32_t w[4][8];  // word 2j + r8 of the unit of row g
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          uint32_t o[4];
#define RB200_T4(C, R8, G0)                                                                                       \
  transpose_bytes4(v[4 * j].C ^ 0x80808080u, v[4 * j + 1].C ^ 0x80808080u, v[4 * j + 2].C ^ 0x80808080u,          \
                   v[4 * j + 3].C ^ 0x80808080u, o);                                                              \
  w[2 * j + R8][G0] = o[0], w[2 * j + R8][G0 + 1] = o[1], w[2 * j + R8][G0 + 2] = o[2], w[2 * j + R8][G0 + 3] = o[3]
          RB200_T4(x, 0, 0);
          RB200_T4(y, 0, 4);
          RB200_T4(z, 1, 0);
          RB200_T4(w, 1, 4);
#undef RB200_T4
        }
#pragma unroll
        for (int g = 0; g < 8; ++g) unit[g] = make_uint4(w[0][g], w[1][g], w[2][g], w[3][g]);
      } else {
        // words of eight consecutive k: two per row of the unit
        uint32_t lo[2][8], hi[2][8];
        if (LAYOUT == 1) {  // [N, K/8]
          const uint8_t* q = s + (kb * 8 + t * 2) * 4;
          const int64_t pitch = K / 2;
#pragma unroll
          for (int g = 0; g < 8; ++g) {
            const uint2 a = *(reinterpret_cast<const uint2*>(q + (n_lo + g) * pitch));
            const uint2 c = *(reinterpret_cast<const uint2*>(q + (n_hi + g) * pitch));
            lo[0][g] = a.x, lo[1][g] = a.y, hi[0][g] = c.x, hi[1][g] = c.y;
          }
        } else {  // [K/8, N]
          const uint8_t* q = s + (kb * 8 + t * 2) * N * 4;
#pragma unroll
          for (int h = 0; h < 2; ++h)
#pragma unroll
            for (int g4 = 0; g4 < 8; g4 += 4) {
              const uint4 a = *(reinterpret_cast<const uint4*>(q + (h * N + n_lo + g4) * 4));
              const uint4 c = *(reinterpret_cast<const uint4*>(q + (h * N + n_hi + g4) * 4));
              lo[h][g4] = a.x, lo[h][g4 + 1] = a.y, lo[h][g4 + 2] = a.z, lo[h][g4 + 3] = a.w;
              hi[h][g4] = c.x, hi[h][g4 + 1] = c.y, hi[h][g4 + 2] = c.z, hi[h][g4 + 3] = c.w;
            }
        }
#pragma unroll
        for (int g = 0; g < 8; ++g) {
          uint32_t w[4];
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            const uint32_t ev = (lo[h][g] & kLow) | ((hi[h][g] << 4) & ~kLow);  // k, k + 2, k + 4, k + 6
            const uint32_t od = ((lo[h][g] >> 4) & kLow) | (hi[h][g] & ~kLow);
            w[2 * h] = prmt(ev, od, 0x5410u);
            w[2 * h + 1] = prmt(ev, od, 0x7632u);
          }
          unit[g] = make_uint4(w[0], w[1], w[2], w[3]);
        }
      }
    }
    __syncthreads();  // the previous run has left shared memory
    if (active) {
#pragma unroll
      for (int g = 0; g < 8; ++g) run[(b * nkb + kbl) * 32 + frag_unit_pos(4 * g + t)] = unit[g];
    }
    __syncthreads();
    uint4* d = reinterpret_cast<uint4*>(dst + e * expert_bytes + frag_stage_offset(tile, chunk, NB, KB));
    for (int i = tid; i < nblk * nkb * 32; i += 128) d[i] = run[i];
  }
}

// Act-order AutoGPTQ weights (tests/python/dlight/test_gpu_gemv.py:639-649 reads scale and zero
// of element k through g_idx[k]): perm lists the k rows group by group, in their original order
// inside a group, so that the weight repacked through perm has its groups contiguous along k and
// the matmul of x gathered through the same perm equals the reference's.  One CTA; every thread
// owns groups g = tid, tid + blockDim, ... and scans g_idx twice (count, then place).
// status: 0 = fine, 1 = some group does not have exactly K / G members or an index is out of range.
__global__ void gptq_act_order_kernel(const int32_t* __restrict__ g_idx, int K, int G, int32_t* __restrict__ perm,
                                      int* __restrict__ status) {
  extern __shared__ int s_start[];  // [G + 1]
  const int per = K / G;
  __shared__ int bad;
  if (threadIdx.x == 0) bad = 0;
  __syncthreads();
  for (int g = threadIdx.x; g < G; g += blockDim.x) {
    int c = 0;
    for (int k = 0; k < K; ++k) c += g_idx[k] == g;
    if (c != per) bad = 1;
    s_start[g] = g * per;  // groups of equal size, or the result is rejected
  }
  __syncthreads();
  if (threadIdx.x == 0) *status = bad;
  if (bad) return;
  for (int g = threadIdx.x; g < G; g += blockDim.x) {
    int pos = s_start[g];
    for (int k = 0; k < K; ++k)
      if (g_idx[k] == g) perm[pos++] = k;
  }
}

// out[m, j] = x[m, perm[j]] over fp16.  A thread takes VEC neighbouring j of every gridDim.y-th row; eight where
// the rows of `out` and perm are 16-byte aligned.
template <int VEC>
__global__ void __launch_bounds__(128) gather_columns_kernel(const __half* x, const int32_t* perm, __half* out, int64_t M, int64_t K,
                                                             int64_t ldx, int64_t ldo) {
  griddep_chain();
  const int64_t j = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) * VEC;
  if (j >= K) return;
  __align__(16) int32_t from[VEC];
  if (VEC == 8) {
    *reinterpret_cast<int4*>(from) = *reinterpret_cast<const int4*>(perm + j);
    *reinterpret_cast<int4*>(from + 4) = *reinterpret_cast<const int4*>(perm + j + 4);
  } else {
    from[0] = perm[j];
  }
  for (int64_t m = blockIdx.y; m < M; m += gridDim.y) {
    __align__(16) __half v[VEC];
#pragma unroll
    for (int i = 0; i < VEC; ++i) v[i] = x[m * ldx + from[i]];
    if (VEC == 8) *reinterpret_cast<uint4*>(out + m * ldo + j) = *reinterpret_cast<const uint4*>(v);
    else out[m * ldo + j] = v[0];
  }
}

// The same with `rows` rows at a time in shared memory: whole lines in and out, and the indices read once for them.
__global__ void __launch_bounds__(256) gather_columns_staged_kernel(const __half* x, const int32_t* perm, __half* out, int64_t M,
                                                                    int K, int64_t ldx, int64_t ldo, int rows) {
  extern __shared__ __align__(16) uint4 staged[];  // [rows][K / 8]
  const __half* h = reinterpret_cast<const __half*>(staged);
  const int vecs = K / 8;
  griddep_chain();
  for (int64_t m0 = (int64_t)blockIdx.x * rows; m0 < M; m0 += (int64_t)gridDim.x * rows) {
    const int n = (int)min((int64_t)rows, M - m0);
    for (int r = 0; r < n; ++r)
      for (int c = threadIdx.x; c < vecs; c += 256) staged[r * vecs + c] = reinterpret_cast<const uint4*>(x + (m0 + r) * ldx)[c];
    __syncthreads();
    for (int c = threadIdx.x; c < vecs; c += 256) {
      const int4 a = reinterpret_cast<const int4*>(perm)[2 * c], b = reinterpret_cast<const int4*>(perm)[2 * c + 1];
      const int from[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
      for (int r = 0; r < n; ++r) {
        __align__(16) __half v[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) v[i] = h[r * K + from[i]];
        reinterpret_cast<uint4*>(out + (m0 + r) * ldo)[c] = *reinterpret_cast<const uint4*>(v);
      }
    }
    __syncthreads();
  }
}

}  // namespace

// dst[o][j][i] = src[o][gate_up_source_row(j)][i] over fp16 elements: the row permutation of the
// interleaved repack applied to a scale / zero-point tensor viewed as [outer][n][inner]
__global__ void interleave_rows_kernel(const __half* __restrict__ src, __half* __restrict__ dst, int64_t outer,
                                       int64_t N, int64_t inner) {
  const int64_t total = outer * N * inner;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < total; i += (int64_t)gridDim.x * blockDim.x) {
    const int64_t in = i % inner, j = (i / inner) % N, o = i / (inner * N);
    dst[i] = src[(o * N + gate_up_source_row(j, N)) * inner + in];
  }
}

int preprocess_launch(const void* src, void* dst, int64_t experts, int64_t k, int64_t n, int bits,
                      int layout_flags, const int32_t* k_perm, cudaStream_t stream) {
  const int interleave = (layout_flags & 0x100) ? 1 : 0;
  const int layout = layout_flags & 0xff;
  RB200_CHECK(!k_perm || layout == 2, "a k permutation goes with the AutoGPTQ source layout only");
  const int64_t units = k * n * bits / 8 / 16;
  const int64_t total = units * experts;
  const int threads = 256;
  int64_t blocks = (total + threads - 1) / threads;
  if (blocks > (int64_t)sm_count_current() * 32) blocks = (int64_t)sm_count_current() * 32;
  if (blocks == 0) return 0;
  const uint8_t* s = static_cast<const uint8_t*>(src);
  uint8_t* d = static_cast<uint8_t*>(dst);
  // widest load each layout makes: the interleaved forms split every row group in two
  const uintptr_t need = layout == 0 ? (bits == 8 ? (interleave ? 8 : 16) : (interleave ? 4 : 8)) : (layout == 1 ? 8 : 16);
  const int64_t tiles = (n + 127) / 128, chunks = (k / (bits == 4 ? 64 : 32) + 3) / 4;
  if (!k_perm && (reinterpret_cast<uintptr_t>(src) & (need - 1)) == 0 && experts * tiles * chunks < (1ll << 31)) {
    const uint32_t stages = (uint32_t)(experts * tiles * chunks);
    uint32_t grid = (uint32_t)sm_count_current() * 12;
    if (grid > stages) grid = stages;
#define RB200_RS(B, L)                                                                                           \
  RB200_CUDA(launch_dependent(interleave ? repack_stage_kernel<B, L, true> : repack_stage_kernel<B, L, false>, dim3(grid), 128, 0, \
                              stream, s, d, k, n, (uint32_t)tiles, (uint32_t)chunks, stages))
    if (bits == 8) RB200_RS(8, 0);
    else if (layout == 0) RB200_RS(4, 0);
    else if (layout == 1) RB200_RS(4, 1);
    else RB200_RS(4, 2);
#undef RB200_RS
    return 0;
  }
  // a k permutation (act-order) or an unaligned source: code by code
  if (bits == 4 && layout == 0)
    repack_kernel<4, 0><<<(int)blocks, threads, 0, stream>>>(s, d, k, n, units, total, interleave, k_perm);
  else if (bits == 4 && layout == 2)
    repack_kernel<4, 2><<<(int)blocks, threads, 0, stream>>>(s, d, k, n, units, total, interleave, k_perm);
  else if (bits == 8 && layout == 0)
    repack_kernel<8, 0><<<(int)blocks, threads, 0, stream>>>(s, d, k, n, units, total, interleave, k_perm);
  else
    RB200_CHECK(false, "unsupported preprocess combination bits=%d layout=%d", bits, layout);

  RB200_CUDA(cudaGetLastError());
  return 0;
}

int interleave_rows_launch(const void* src, void* dst, int64_t outer, int64_t n, int64_t inner, cudaStream_t stream) {
  const int64_t total = outer * n * inner;
  if (total == 0) return 0;
  int64_t blocks = (total + 255) / 256;
  if (blocks > (int64_t)sm_count_current() * 16) blocks = (int64_t)sm_count_current() * 16;
  interleave_rows_kernel<<<(int)blocks, 256, 0, stream>>>(static_cast<const __half*>(src), static_cast<__half*>(dst),
                                                         outer, n, inner);
  RB200_CUDA(cudaGetLastError());
  return 0;
}

int gptq_act_order_launch(const int32_t* g_idx, int64_t k, int64_t groups, int32_t* perm, int* status,
                          cudaStream_t stream) {
  gptq_act_order_kernel<<<1, 1024, (size_t)(groups + 1) * sizeof(int), stream>>>(g_idx, (int)k, (int)groups, perm, status);
  RB200_CUDA(cudaGetLastError());
  return 0;
}

int gather_columns_launch(const void* x, const int32_t* perm, void* out, int64_t m, int64_t k, int64_t ldx,
                          int64_t ldo, cudaStream_t stream) {
  if (m * k == 0) return 0;
  const bool vec = k % 8 == 0 && ldo % 8 == 0 && ((reinterpret_cast<uintptr_t>(out) | reinterpret_cast<uintptr_t>(perm)) & 15u) == 0;
  // From 65 rows on through shared memory, where the rows can be read 16 bytes at a time; below, the direct form's
  // single trip to memory is shorter, as long as its CTAs run at once.  The line suits k 4096 (64 rows direct 1.8 us,
  // 65 staged 2.0); longer rows would cross earlier: k 11008, 48 rows 2.6 direct, 64 rows 4.2, 65 staged 3.5; k 14336,
  // 32 rows 2.7 direct, 48 rows 4.6, 65 staged 3.9.  Measured (graph of launches; element by element with 64-bit
  // divisions before): k 4096, 16 rows 1.5 us (2.0), 512 rows 3.8 (7.9), 2048 rows 11.1 (25.4); k 14336, 512 rows
  // 10.5 (26.9), 2048 rows 41 (105).
  constexpr int64_t kStaged = 96 * 1024;
  if (vec && m > 64 && ldx % 8 == 0 && (reinterpret_cast<uintptr_t>(x) & 15u) == 0 && k * 2 <= kStaged) {
    static thread_local int configured_device = -1;
    int dev = 0;
    RB200_CUDA(cudaGetDevice(&dev));
    if (configured_device != dev) {
      RB200_CUDA(cudaFuncSetAttribute(gather_columns_staged_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kStaged));
      configured_device = dev;
    }
    int64_t rows = kStaged / (k * 2);
    if (rows > 4) rows = 4;
    while (rows > 1 && (m + rows - 1) / rows < sm_count_current() * 2) --rows;
    const int64_t need = (m + rows - 1) / rows, most = (int64_t)sm_count_current() * 8;
    RB200_CUDA(launch_dependent(gather_columns_staged_kernel, dim3((unsigned)(need < most ? need : most)), 256, (size_t)(rows * k * 2),
                                stream, static_cast<const __half*>(x), perm, static_cast<__half*>(out), m, (int)k, ldx, ldo, (int)rows));
    return 0;
  }
  const int64_t columns = (k / (vec ? 8 : 1) + 127) / 128;
  RB200_CHECK(columns < (1ll << 31), "k=%lld is too large", (long long)k);
  // rows that a thread does one after the other share its indices: no more CTAs than fill the device a few times
  int64_t rows = (int64_t)sm_count_current() * 16 / columns + 1;
  if (rows > m) rows = m;
  if (rows > 65535) rows = 65535;
  RB200_CUDA(launch_dependent(vec ? gather_columns_kernel<8> : gather_columns_kernel<1>, dim3((unsigned)columns, (unsigned)rows), 128, 0,
                              stream, static_cast<const __half*>(x), perm, static_cast<__half*>(out), m, k, ldx, ldo));
  return 0;
}

int unpack_zeros_autogptq_launch(const void* zq, void* out, int64_t groups, int64_t n, cudaStream_t stream) {
  const int64_t words = groups * (n / 8);
  if (words == 0) return 0;
  int64_t blocks = (words + 255) / 256;
  if (blocks > (int64_t)sm_count_current() * 16) blocks = (int64_t)sm_count_current() * 16;
  RB200_CUDA(launch_dependent(unpack_zeros_autogptq_kernel, dim3((unsigned)blocks), 256, 0, stream, static_cast<const uint32_t*>(zq),
                              static_cast<__half*>(out), words, (reinterpret_cast<uintptr_t>(out) & 15u) == 0));
  return 0;
}

}  // namespace rb200
