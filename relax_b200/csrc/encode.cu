// Quantiser on the GPU: the reference tests' encode TIR
// (tests/python/relax/test_codegen_cutlass.py:1391-1457 int4 per-row, :1630-1676 int8 per-row,
// :2043-2109 int8 in groups of 64) - the transform_params stage that the reference runs on the
// CPU before ft_preprocess_weight.
//   absmax over the row (or the row's group) in fp16;
//   scale = max(f32(absmax), 1e-4) * (1/8 | 1/128) in fp32;
//   code  = clamp(round_half_away(f32(a) / scale), -8..7 | -128..127);
//   packed int8 [K, N/2] (low nibble = even n) or [K, N]; scales fp16 [N] or [K/g, N].
//
// Bound: HBM, the fp16 weight read once.  A CTA keeps 32 rows x a slice of k in shared memory
// between the two passes over it (absmax, quantise); with one scale per row the slices of a row
// are the CTAs of one cluster, which exchange their maxima through distributed shared memory.
// Quantising multiplies by the reciprocal scale and rounds by an addition, seven instructions
// per value; a value whose product lies within the error bound of a rounding boundary is divided
// instead, so that every code is the one the division gives.  Measured, fp16 11008 x 4096: int4 55 us
// (2.1 TB/s), int8 in groups of 64 50 us; 230 us with a division and two global reads per value.
// The source is read from memory once; what bounds the rest has not been profiled (the instructions above are
// some 12 us of issue at that size, the bytes 17).
#include <cooperative_groups.h>

#include "../../include/relax_b200.h"
#include "common.cuh"

namespace rb200 {
namespace {

constexpr int kRows = 32;     // n per CTA
constexpr int kMaxSpan = 512;  // k per pass through shared memory

// code of one value by the definition: round_half_away(a / scale), clamped
template <int BITS>
__device__ __noinline__ int encode_exact(float a, float scale) {
  constexpr float qlo = BITS == 4 ? -8.0f : -128.0f, qhi = BITS == 4 ? 7.0f : 127.0f;
  return (int)fminf(fmaxf(roundf(__fdiv_rn(a, scale)), qlo), qhi);
}

// Rows in tiles of 32, k in slices that fit shared memory; needs n % 32 == 0, 16-byte rows and
// groups of whole 16-byte vectors (the kernel below covers the rest).
// PER_ROW: gridDim.y slices of a row form one cluster.  Otherwise a slice holds whole groups.
template <int BITS, bool PER_ROW>
__global__ void __launch_bounds__(256, 4) encode_slices_kernel(const __half* __restrict__ A, int8_t* __restrict__ packed,
                                                            __half* __restrict__ scales, int64_t N, int64_t K, int slice,
                                                            int group) {
  namespace cg = cooperative_groups;
  extern __shared__ __align__(16) uint8_t enc_smem[];
  __half* tile = reinterpret_cast<__half*>(enc_smem);                             // [32][slice]
  unsigned* amax = reinterpret_cast<unsigned*>(enc_smem + (size_t)kRows * slice * 2);  // [32][groups] fp16 bits
  const int groups = PER_ROW ? 1 : slice / group;
  float* s_scale = reinterpret_cast<float*>(amax + kRows * groups);               // [groups][32]
  float* s_inv = s_scale + kRows * groups;                                        // [groups][32]
  const int64_t n0 = (int64_t)blockIdx.x * kRows, k0 = (int64_t)blockIdx.y * slice;
  const int span = (int)min((int64_t)slice, K - k0);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const float mul = BITS == 4 ? 0.125f : 0.0078125f;

  for (int i = tid; i < kRows * groups; i += 256) amax[i] = 0u;
  __syncthreads();
  // pass 1: rows warp, warp + 8, ... of the slice into shared memory, absolute maxima on the way
  const __half* src = A + (n0 + warp) * K + k0;
  __half2 mx[kRows / 8];
#pragma unroll
  for (int i = 0; i < kRows / 8; ++i) mx[i] = __half2half2(__ushort_as_half(0));
#pragma unroll 2
  for (int c = lane * 8; c < span; c += 256) {
    uint4 v[kRows / 8];
#pragma unroll
    for (int i = 0; i < kRows / 8; ++i) v[i] = __ldg(reinterpret_cast<const uint4*>(src + (int64_t)i * 8 * K + c));
#pragma unroll
    for (int i = 0; i < kRows / 8; ++i) {
      const int r = warp + 8 * i;
      *reinterpret_cast<uint4*>(tile + (size_t)r * slice + c) = v[i];
      const __half2* h = reinterpret_cast<const __half2*>(&v[i]);
      // __hmax2 drops a NaN operand, as fmaxf does
      const __half2 m = __hmax2(__hmax2(__habs2(h[0]), __habs2(h[1])), __hmax2(__habs2(h[2]), __habs2(h[3])));
      if (PER_ROW) {
        mx[i] = __hmax2(mx[i], m);
      } else {
        const __half hm = __hmax(__hmax(__low2half(m), __high2half(m)), __ushort_as_half(0));
        atomicMax(&amax[r * groups + c / group], (unsigned)__half_as_ushort(hm));  // non-negative: bits order as values
      }
    }
  }
  if (PER_ROW) {
#pragma unroll
    for (int i = 0; i < kRows / 8; ++i) {
      unsigned m = max((unsigned)__half_as_ushort(__low2half(mx[i])), (unsigned)__half_as_ushort(__high2half(mx[i])));
      m = __reduce_max_sync(0xffffffffu, m);
      if (lane == 0) amax[warp + 8 * i] = m;
    }
    cg::cluster_group cl = cg::this_cluster();
    cl.sync();
    if (tid < kRows) {
      unsigned m = 0u;
      for (unsigned c = 0; c < cl.num_blocks(); ++c) m = max(m, *cl.map_shared_rank(amax + tid, c));
      const float sc = fmaxf(__half2float(__ushort_as_half((unsigned short)m)), 1e-4f) * mul;
      s_scale[tid] = sc;
      s_inv[tid] = __fdiv_rn(1.0f, sc);
      if (blockIdx.y == 0) scales[n0 + tid] = __float2half_rn(sc);
    }
    cl.sync();  // no CTA leaves while its maxima are being read
  } else {
    __syncthreads();
    for (int i = tid; i < kRows * (span / group); i += 256) {
      const int r = i % kRows, g = i / kRows;
      const float sc = fmaxf(__half2float(__ushort_as_half((unsigned short)amax[r * groups + g])), 1e-4f) * mul;
      s_scale[g * kRows + r] = sc;
      s_inv[g * kRows + r] = __fdiv_rn(1.0f, sc);
      scales[(k0 / group + g) * N + n0 + r] = __float2half_rn(sc);
    }
    __syncthreads();
  }

  // pass 2: a thread takes two neighbouring k of all 32 rows and writes their packed bytes
  constexpr float kMagic = 12582912.0f;  // 1.5 * 2^23: adding it rounds to an integer in the low mantissa bits
  constexpr float kTop = kMagic + (BITS == 4 ? 7.0f : 127.0f);
  // |a * rn(1/s) - a/s| and the division's own rounding are 2^-24 relative each: at most 2^-20 (int4)
  // or 2^-16 (int8) in total; a product closer than that to k + 1/2 is settled by the division
  constexpr float kSafe = 0.5f - (BITS == 4 ? 2e-6f : 2e-5f);
  for (int c = tid * 2; c < span; c += 512) {
    const int g = PER_ROW ? 0 : c / group;
    const float* sc = s_scale + g * kRows;
    const float* inv = s_inv + g * kRows;
    uint32_t lo[BITS], hi[BITS];  // 32 codes of k and of k + 1: BITS words each
    constexpr int kPer = 32 / BITS;
    constexpr uint32_t mask = BITS == 4 ? 15u : 255u;
    unsigned doubtful = 0u;       // words with a value near a rounding boundary
#pragma unroll
    for (int w = 0; w < BITS; ++w) {
      uint32_t x = 0u, y = 0u;
      bool near = false;
#pragma unroll
      for (int i = kPer - 1; i >= 0; --i) {
        const int r = w * kPer + i;
        const float2 a = __half22float2(*reinterpret_cast<const __half2*>(tile + (size_t)r * slice + c));
        const float iv = inv[r];
        const float t0 = fmaf(a.x, iv, kMagic), t1 = fmaf(a.y, iv, kMagic);
        near |= !(fabsf(fmaf(a.x, iv, kMagic - t0)) < kSafe) | !(fabsf(fmaf(a.y, iv, kMagic - t1)) < kSafe);
        x = (x << BITS) | (__float_as_uint(fminf(t0, kTop)) & mask);
        y = (y << BITS) | (__float_as_uint(fminf(t1, kTop)) & mask);
      }
      lo[w] = x;
      hi[w] = y;
      doubtful |= (near ? 1u : 0u) << w;
    }
    const int64_t pitch = N * BITS / 8;
    int8_t* d = packed + (k0 + c) * pitch + n0 * BITS / 8;
#pragma unroll
    for (int q = 0; q < BITS / 4; ++q) {
      *reinterpret_cast<uint4*>(d + q * 16) = make_uint4(lo[4 * q], lo[4 * q + 1], lo[4 * q + 2], lo[4 * q + 3]);
      *reinterpret_cast<uint4*>(d + pitch + q * 16) = make_uint4(hi[4 * q], hi[4 * q + 1], hi[4 * q + 2], hi[4 * q + 3]);
    }
    while (doubtful) {  // rare: those words again, by division
      const int w = __ffs(doubtful) - 1;
      doubtful &= doubtful - 1u;
      uint32_t x = 0u, y = 0u;
#pragma unroll 1
      for (int i = kPer - 1; i >= 0; --i) {
        const int r = w * kPer + i;
        const float2 a = __half22float2(*reinterpret_cast<const __half2*>(tile + (size_t)r * slice + c));
        x = (x << BITS) | ((uint32_t)encode_exact<BITS>(a.x, sc[r]) & mask);
        y = (y << BITS) | ((uint32_t)encode_exact<BITS>(a.y, sc[r]) & mask);
      }
      reinterpret_cast<uint32_t*>(d)[w] = x;
      reinterpret_cast<uint32_t*>(d + pitch)[w] = y;
    }
  }
}

// Any shape: one CTA per 32 rows x one group, two reads of the weight.
template <int BITS>
__global__ void __launch_bounds__(256) encode_ft_kernel(const __half* __restrict__ A, int8_t* __restrict__ packed,
                                                        __half* __restrict__ scales, int64_t N, int64_t K,
                                                        int64_t group, int per_row) {
  __shared__ __half tile[kRows][kMaxSpan + 8];
  __shared__ float s_scale[kRows];
  const int64_t n0 = (int64_t)blockIdx.x * kRows;
  const int64_t g = blockIdx.y;  // group index (0 when one scale per row)
  const int64_t k_begin = g * group, k_end = k_begin + group;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const float mul = BITS == 4 ? 0.125f : 0.0078125f;
  const float qlo = BITS == 4 ? -8.0f : -128.0f, qhi = BITS == 4 ? 7.0f : 127.0f;

  // pass 1: absmax of every row over [k_begin, k_end)
  float amax[kRows / 8];
#pragma unroll
  for (int i = 0; i < kRows / 8; ++i) amax[i] = 0.0f;
  for (int64_t k = k_begin + lane; k < k_end; k += 32) {
#pragma unroll
    for (int i = 0; i < kRows / 8; ++i) {
      const int64_t n = n0 + warp + 8 * i;
      if (n < N) amax[i] = fmaxf(amax[i], fabsf(__half2float(A[n * K + k])));
    }
  }
#pragma unroll
  for (int i = 0; i < kRows / 8; ++i) {
    float v = amax[i];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
    if (lane == 0) s_scale[warp + 8 * i] = fmaxf(v, 1e-4f) * mul;  // |a| is exact in fp16, so is its max
  }
  __syncthreads();
  if (tid < kRows && n0 + tid < N)
    scales[(per_row ? 0 : g * N) + n0 + tid] = __float2half_rn(s_scale[tid]);

  // pass 2: quantise spans of k, transposing through shared memory
  for (int64_t ks = k_begin; ks < k_end; ks += kMaxSpan) {
    const int span = (int)min((int64_t)kMaxSpan, k_end - ks);
    __syncthreads();
    for (int i = tid; i < kRows * span; i += 256) {
      const int r = i / span, c = i % span;
      tile[r][c] = (n0 + r < N) ? A[(n0 + r) * K + ks + c] : __float2half_rn(0.0f);
    }
    __syncthreads();
    if (BITS == 4) {
      // thread -> (k, pair of rows): 16 byte columns per k
      for (int i = tid; i < span * (kRows / 2); i += 256) {
        const int c = i / (kRows / 2), pr = i % (kRows / 2);
        const int r0 = 2 * pr, r1 = r0 + 1;
        if (n0 + r0 >= N) continue;
        const float q0 = fminf(fmaxf(roundf(__fdiv_rn(__half2float(tile[r0][c]), s_scale[r0])), qlo), qhi);
        const float q1 = (n0 + r1 < N)
                             ? fminf(fmaxf(roundf(__fdiv_rn(__half2float(tile[r1][c]), s_scale[r1])), qlo), qhi)
                             : 0.0f;
        const int b = ((int)q0 & 15) | (((int)q1 & 15) << 4);
        packed[(ks + c) * (N / 2) + (n0 >> 1) + pr] = (int8_t)b;
      }
    } else {
      for (int i = tid; i < span * kRows; i += 256) {
        const int c = i / kRows, r = i % kRows;
        if (n0 + r >= N) continue;
        const float q = fminf(fmaxf(roundf(__fdiv_rn(__half2float(tile[r][c]), s_scale[r])), qlo), qhi);
        packed[(ks + c) * N + n0 + r] = (int8_t)(int)q;
      }
    }
  }
}

template <int BITS, bool PER_ROW>
int launch_slices(const void* a, void* packed, void* scales, int64_t n, int64_t k, int slice, int group, int slices,
                  size_t smem, cudaStream_t stream) {
  auto kern = encode_slices_kernel<BITS, PER_ROW>;
  static thread_local int configured_device = -1;
  int dev = 0;
  RB200_CUDA(cudaGetDevice(&dev));
  if (configured_device != dev) {
    RB200_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024));
    configured_device = dev;
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(n / kRows), (unsigned)slices, 1);
  cfg.blockDim = dim3(256, 1, 1);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 1;
  attr[0].val.clusterDim.y = PER_ROW ? (unsigned)slices : 1u;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  RB200_CUDA(cudaLaunchKernelEx(&cfg, kern, static_cast<const __half*>(a), static_cast<int8_t*>(packed),
                                static_cast<__half*>(scales), n, k, slice, group));
  return 0;
}

}  // namespace
}  // namespace rb200

using namespace rb200;

extern "C" int rb200_encode_ft(const void* a, void* packed, void* scales, int64_t n, int64_t k, int weight_bits,
                               int64_t group_size, void* stream) {
  RB200_CHECK(a && packed && scales, "a, packed and scales must be non-NULL");
  RB200_CHECK(weight_bits == 4 || weight_bits == 8, "weight_bits must be 4 or 8");
  RB200_CHECK(n > 0 && k > 0 && (weight_bits == 8 || n % 2 == 0), "bad shape n=%lld k=%lld", (long long)n, (long long)k);
  const bool per_row = group_size <= 0 || group_size >= k;
  const int64_t group = per_row ? k : group_size;
  RB200_CHECK(k % group == 0, "group_size=%lld must divide k=%lld", (long long)group, (long long)k);
  RB200_CHECK(k / group <= 65535, "too many groups");
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const bool aligned = ((reinterpret_cast<uintptr_t>(a) | reinterpret_cast<uintptr_t>(packed)) & 15u) == 0;
  if (aligned && n % kRows == 0 && k % 8 == 0 && n / kRows < (1ll << 31)) {
    // slice of k per CTA: 32 rows x 1024 k are 64 KB, two or three CTAs per SM.  One scale per row:
    // the slices of a row are a cluster of at most eight CTAs, so long rows take longer slices.
    if (per_row) {
      int64_t c = 1;
      while (c < 8 && k > c * 512) c *= 2;
      const int64_t slice = ((k + c - 1) / c + 7) / 8 * 8;
      const size_t smem = (size_t)kRows * slice * 2 + kRows * 12;
      if (smem <= 200 * 1024 && (c - 1) * slice < k)
        return weight_bits == 4 ? launch_slices<4, true>(a, packed, scales, n, k, (int)slice, 0, (int)c, smem, s)
                                : launch_slices<8, true>(a, packed, scales, n, k, (int)slice, 0, (int)c, smem, s);
    } else if (group % 8 == 0 && group <= 1024) {
      const int64_t slice = (group > 512 ? 1024 : 512) / group * group;
      const size_t smem = (size_t)kRows * slice * 2 + kRows * (slice / group) * 12;
      const int64_t c = (k + slice - 1) / slice;
      if (c <= 65535)
        return weight_bits == 4 ? launch_slices<4, false>(a, packed, scales, n, k, (int)slice, (int)group, (int)c, smem, s)
                                : launch_slices<8, false>(a, packed, scales, n, k, (int)slice, (int)group, (int)c, smem, s);
    }
  }
  dim3 grid((unsigned)((n + kRows - 1) / kRows), (unsigned)(k / group), 1);
  if (weight_bits == 4)
    encode_ft_kernel<4><<<grid, 256, 0, s>>>(static_cast<const __half*>(a), static_cast<int8_t*>(packed),
                                             static_cast<__half*>(scales), n, k, group, per_row ? 1 : 0);
  else
    encode_ft_kernel<8><<<grid, 256, 0, s>>>(static_cast<const __half*>(a), static_cast<int8_t*>(packed),
                                             static_cast<__half*>(scales), n, k, group, per_row ? 1 : 0);
  RB200_CUDA(cudaGetLastError());
  return 0;
}
