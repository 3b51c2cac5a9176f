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
// are the CTAs of one cluster, which push their maxima into one another's shared memory: one cluster
// barrier between the passes, and none that a CTA has to leave behind.
// Quantising is four instructions per value (widen, multiply into the rounding constant, shift-add into
// the packed word; half of a clamp).  The division of the definition is not needed: with a scale made
// from an fp16 absmax, a / scale is either a tie exactly or more than 1.2e-4 away from one, so a
// reciprocal that is four units too large rounds every tie away from zero and nothing else differently.
// That was checked for all (absmax, value) pairs of fp16 and both widths, 2e9 of them, against the
// division; the test repeats it for a sample.  Infinite maxima and NaN take the division.
// The CTAs are persistent: three slices in shared memory, one being quantised, one whose maxima travel, one on
// its way from memory; rows of more than 16384 k have room for two, of more than 24576 for one (encode_plan.h).
// Measured, fp16 11008 x 4096 (90 MB): one scale per row 31 us, int8 in groups of 64
// 35 us; 45 / 55 us with a CTA per slice and a cluster barrier (its loads, its exchange and its arithmetic
// one after the other, 37 us of it before the first code), and 53 / 50 us with a test for ties per value as well.
// Loading and exchanging alone take 21 us, the codes 6, their stores (16 bytes of a k at a time) 6.
// 8192 x 16384 int4 99 us (2.7 TB/s of source), x 18944 134, x 24576 149, x 28672 218 (one buffer).
#include <atomic>

#include "../../include/relax_b200.h"
#include "common.cuh"
#include "encode_plan.h"

namespace rb200 {
namespace {

constexpr int kRows = kEncodeRows;  // n per CTA
constexpr int kMaxSpan = 512;       // k per pass through shared memory
constexpr int kMaxCluster = kEncodeMaxCluster;
constexpr int kPlaces = 3;  // for maxima

// code of one value by the definition: round_half_away(a / scale), clamped
template <int BITS>
__device__ __noinline__ int encode_exact(float a, float scale) {
  constexpr float qlo = BITS == 4 ? -8.0f : -128.0f, qhi = BITS == 4 ? 7.0f : 127.0f;
  return (int)fminf(fmaxf(roundf(__fdiv_rn(a, scale)), qlo), qhi);
}

constexpr float kMagic = 12582912.0f;  // 1.5 * 2^23: adding it rounds to an integer in the low mantissa bits

// Reciprocal of a scale, four units too large (ties go away from zero, see above), and the largest value
// that is worth looking at: fp16(7 | 127 scales), as two halves, so that no code leaves its range upwards.
template <int BITS>
__device__ __forceinline__ float2 quantiser(float scale) {
  const float inv = __uint_as_float(__float_as_uint(__fdiv_rn(1.0f, scale)) + 4u);
  const unsigned cap = __half_as_ushort(__float2half_rn((BITS == 4 ? 7.0f : 127.0f) * scale));
  return make_float2(inv, __uint_as_float(cap * 0x10001u));
}
// what the packed sums of a word hold beside the codes: the bits of kMagic less the codes' bias, at every position
template <int BITS>
constexpr uint32_t rounding_sum() {
  uint32_t sum = 0u;
  for (int i = 0; i < 32 / BITS; ++i) sum = (sum << BITS) + 0x4b400000u - (1u << (BITS - 1));
  return sum;
}

// without the NaNs: __hmax2 drops one NaN operand and gives NaN for two, hence the maximum with zero
__device__ __forceinline__ __half2 abs_max(uint4 v) {
  const __half2* h = reinterpret_cast<const __half2*>(&v);
  return __hmax2(__hmax2(__hmax2(__habs2(h[0]), __habs2(h[1])), __hmax2(__habs2(h[2]), __habs2(h[3]))),
                 __half2half2(__ushort_as_half(0)));
}
__device__ __forceinline__ __half2 abs_max_nan(uint4 v) {  // 0x7fff for a NaN
  const __half2* h = reinterpret_cast<const __half2*>(&v);
  return __hmax2_nan(__hmax2_nan(__habs2(h[0]), __habs2(h[1])), __hmax2_nan(__habs2(h[2]), __habs2(h[3])));
}
__device__ __forceinline__ unsigned larger_bits(__half2 m) {  // non-negative: bits order as values
  const unsigned u = *reinterpret_cast<const unsigned*>(&m);
  return max(u & 0xffffu, u >> 16);
}

// 16-byte unit `u` of row r in shared memory: the rows of different packed words lie on different banks, since
// the lanes of a quarter-warp read one word's rows each, at the same few k.
template <int BITS>
__device__ __forceinline__ int unit_at(int r, int u) {
  return u ^ (BITS == 4 ? ((r >> 3) & 3) << 1 : (r >> 2) & 7);
}

// Status word of the kernel's waits, read and cleared by encode_read_status.  A word of its own: quantising is what a
// process does first, before any call has made the library's scratch.
__device__ int g_status;

// Bounded wait (about two seconds) for the maxima other CTAs of the cluster push; false when it ran out.  (The lanes
// of a warp wait each for itself: bringing them together first takes 3 % of the whole kernel.)
__device__ __forceinline__ bool wait_pushed(uint64_t* bar, uint32_t phase) {
#pragma unroll 1
  for (int i = 0; i < 200000; ++i) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2, 10000;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(phase)
        : "memory");
    if (ok) return true;
  }
  return false;
}

// Rows in tiles of 32, k in slices that fit shared memory; needs n % 32 == 0, 16-byte rows and
// groups of whole 16-byte vectors (the kernel below covers the rest).
// PER_ROW: the slices of a row form one cluster (rank = slice), the clusters share out the row tiles.
// Otherwise a slice holds whole groups and the CTAs share out the (row tile, slice) pairs.
// kBufs: slices of a CTA in shared memory.  Three: quantised, maxima being exchanged, on its way.  Long rows have room
// for two, and a slice's maxima then leave after the one before has been quantised, or for one.
template <int BITS, bool PER_ROW, int kThreads, int kBufs>
__global__ void __launch_bounds__(kThreads, kThreads == 256 ? 2 : 1)
    encode_slices_kernel(const __half* __restrict__ A, int8_t* __restrict__ packed, __half* __restrict__ scales, int64_t N, int64_t K,
                         int slice, int slices, int group) {
  constexpr int kWarps = kThreads / 32, kOwnRows = kRows / kWarps;
  constexpr unsigned kInf = 0x7c00u;
  extern __shared__ __align__(128) uint8_t enc_smem[];
  __shared__ unsigned row_max[kPlaces][PER_ROW ? kMaxCluster : 1][kRows];  // PER_ROW: bits of a slice's maximum | NaN << 15
  __shared__ __align__(8) uint64_t max_bar[kPlaces];                    // counts the bytes of the maxima
  const int units = (slice + 63) / 64 * 8;                           // 16-byte units of a row
  const int groups = PER_ROW ? 1 : slice / group;
  uint4* ring = reinterpret_cast<uint4*>(enc_smem);                                          // [kBufs][32][units]
  float2* quant = reinterpret_cast<float2*>(enc_smem + (size_t)kBufs * kRows * units * 16);  // [groups][33]: reciprocal, clamp
  float* s_scale = reinterpret_cast<float*>(quant + (kRows + 1) * groups);                   // [groups][32]
  unsigned* amax = reinterpret_cast<unsigned*>(s_scale + kRows * groups);                    // [32][amax_pitch] fp16 bits
  const int amax_pitch = encode_amax_pitch(groups);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const float mul = BITS == 4 ? 0.125f : 0.0078125f;
  const unsigned n_tiles = (unsigned)(N / kRows);
  unsigned rank = 0u, ranks = 1u;
  if (PER_ROW) {
    asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
    asm("mov.u32 %0, %%cluster_nctarank;" : "=r"(ranks));
    if (tid == 0) {
      for (int i = 0; i < kPlaces; ++i) {
        mbar_init(&max_bar[i], 1);
        mbar_arrive_expect_tx(&max_bar[i], ranks * kRows * 4);
      }
      mbar_fence_init();
    }
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");  // every CTA's barriers exist
  } else {
    for (int i = tid; i < kRows * amax_pitch; i += kThreads) amax[i] = 0u;
    __syncthreads();
  }
  // this CTA's items
  const unsigned first = blockIdx.x / ranks, step = gridDim.x / ranks, items = PER_ROW ? n_tiles : n_tiles * (unsigned)slices;
  auto tile_of = [&](unsigned item) { return PER_ROW ? item : item % n_tiles; };
  auto slice_of = [&](unsigned item) { return PER_ROW ? rank : item / n_tiles; };
  auto span_of = [&](unsigned item) { return (int)min((int64_t)slice, K - (int64_t)slice_of(item) * slice); };
  auto row_of = [&](int i) { return warp + kWarps * i; };  // rows this warp loads and takes the maxima of
  auto load = [&](unsigned item, int buf) {                // a lane's vectors of them; the lane reads them back itself
    const __half* src = A + ((int64_t)tile_of(item) * kRows + warp) * K + (int64_t)slice_of(item) * slice;
    const int span = span_of(item);
    uint4* dst = ring + (size_t)buf * kRows * units;
    for (int u = lane; u * 8 < span; u += 32)
#pragma unroll
      for (int i = 0; i < kOwnRows; ++i)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(dst + row_of(i) * units + unit_at<BITS>(row_of(i), u))),
                     "l"(src + (int64_t)i * kWarps * K + u * 8)
                     : "memory");
  };
  auto commit = [] { asm volatile("cp.async.commit_group;" ::: "memory"); };

  // maxima of a slice's rows, pushed to every CTA of the cluster: asynchronous stores that count on the
  // receiver's barrier, since a release of cluster scope would wait for the packed bytes on their way to memory.
  // A CTA may be two items ahead of another (only one warp waits for the maxima of an item before it pushes
  // the next), so there are three places for them.
  auto push_maxima = [&](unsigned item, int buf, int place) {
    const int span = span_of(item);
    const uint4* t = ring + (size_t)buf * kRows * units;
    unsigned own[kOwnRows], any = 0u;
    __half2 mx[kOwnRows];
#pragma unroll
    for (int i = 0; i < kOwnRows; ++i) mx[i] = __half2half2(__ushort_as_half(0));
    for (int u = lane; u * 8 < span; u += 32)
#pragma unroll
      for (int i = 0; i < kOwnRows; ++i) mx[i] = __hmax2_nan(mx[i], abs_max_nan(t[row_of(i) * units + unit_at<BITS>(row_of(i), u)]));
#pragma unroll
    for (int i = 0; i < kOwnRows; ++i) {
      own[i] = __reduce_max_sync(0xffffffffu, larger_bits(mx[i]));
      any = max(any, own[i]);
    }
    if (any > kInf) {  // without the NaNs
#pragma unroll 1
      for (int i = 0; i < kOwnRows; ++i) {
        unsigned m = 0u;
        for (int u = lane; u * 8 < span; u += 32) m = max(m, larger_bits(abs_max(t[row_of(i) * units + unit_at<BITS>(row_of(i), u)])));
        m = __reduce_max_sync(0xffffffffu, m) | 0x8000u;
#pragma unroll
        for (int j = 0; j < kOwnRows; ++j)
          if (j == i) own[j] = m;
      }
    }
    for (unsigned at = (unsigned)lane; at < kOwnRows * ranks; at += 32) {  // (row, receiver) pairs
      const unsigned i = at / ranks, to = at - i * ranks;
      unsigned v = own[0];
#pragma unroll
      for (int j = 1; j < kOwnRows; ++j)
        if (i == (unsigned)j) v = own[j];
      uint32_t dst, bar;
      asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(dst) : "r"(smem_u32(&row_max[place][rank][warp + kWarps * i])), "r"(to));
      asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(bar) : "r"(smem_u32(&max_bar[place])), "r"(to));
      asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.u32 [%0], %1, [%2];" ::"r"(dst), "r"(v), "r"(bar) : "memory");
    }
  };
  // maxima of the slice's groups
  const int seg = PER_ROW ? 1 : group / 8;  // vectors of a group
  const bool fold_seg = seg <= 32 && (seg & (seg - 1)) == 0;
  const int seg_shift = 31 - __clz(seg);
  auto group_of = [&](int u) { return fold_seg ? u >> seg_shift : u / seg; };
  auto group_maxima = [&](unsigned item, int buf) -> bool {
    const int span = span_of(item);
    const uint4* t = ring + (size_t)buf * kRows * units;
    bool special = false;
    for (int u0 = 0; u0 * 8 < span; u0 += 32) {
      const int u = u0 + lane;
      const bool in = u * 8 < span;
      const int g = in ? group_of(u) : 0;
      uint4 v[kOwnRows];
      __half2 m[kOwnRows / 2];  // of two rows
#pragma unroll
      for (int i = 0; i < kOwnRows; ++i) v[i] = in ? t[row_of(i) * units + unit_at<BITS>(row_of(i), u)] : make_uint4(0u, 0u, 0u, 0u);
      bool nan = false;
#pragma unroll
      for (int i = 0; i < kOwnRows / 2; ++i) {
        const __half2 a = abs_max_nan(v[2 * i]), b = abs_max_nan(v[2 * i + 1]);
        m[i] = __hmax2_nan(__lows2half2(a, b), __highs2half2(a, b));
        nan |= __hisnan(__low2half(m[i])) | __hisnan(__high2half(m[i]));
      }
      if (nan) {
        special = true;
#pragma unroll
        for (int i = 0; i < kOwnRows / 2; ++i) {
          const __half2 a = abs_max(v[2 * i]), b = abs_max(v[2 * i + 1]);
          m[i] = __hmax2(__lows2half2(a, b), __highs2half2(a, b));
        }
      }
      __syncwarp();
      if (fold_seg)  // the lanes of a group are neighbours
        for (int o = seg >> 1; o > 0; o >>= 1)
#pragma unroll
          for (int i = 0; i < kOwnRows / 2; ++i) m[i] = __hmax2(m[i], __shfl_xor_sync(0xffffffffu, m[i], o));
      if (in && (!fold_seg || (lane & (seg - 1)) == 0)) {
#pragma unroll
        for (int i = 0; i < kOwnRows; ++i) {
          const unsigned b = __half_as_ushort(i & 1 ? __high2half(m[i / 2]) : __low2half(m[i / 2]));
          if (fold_seg) amax[row_of(i) * amax_pitch + g] = b;
          else atomicMax(&amax[row_of(i) * amax_pitch + g], b);
        }
      }
    }
    return special;
  };
  // scale of (group g, row r) of an item from the bits of its maximum; true where the division has to do it
  auto set_scale = [&](unsigned item, int g, int r, unsigned m) -> bool {
    const float sc = fmaxf(__half2float(__ushort_as_half((unsigned short)m)), 1e-4f) * mul;
    s_scale[g * kRows + r] = sc;
    quant[g * (kRows + 1) + r + (r >> 4)] = quantiser<BITS>(sc);
    const int64_t n = (int64_t)tile_of(item) * kRows + r;
    if (!PER_ROW) scales[((int64_t)slice_of(item) * groups + g) * N + n] = __float2half_rn(sc);
    else if (rank == 0) scales[n] = __float2half_rn(sc);
    return m >= kInf;
  };

  // a thread makes one packed word each of eight neighbouring k; the words of a k are made by neighbouring lanes
  const int word = tid % BITS, r0 = word * (32 / BITS);
  auto quantise = [&](unsigned item, int buf, bool special) {
    constexpr int kPer = 32 / BITS;             // codes of a word
    constexpr uint32_t kSum = rounding_sum<BITS>(), kSigns = BITS == 4 ? 0x88888888u : 0x80808080u;
    const int64_t pitch = N * BITS / 8;
    const int span = span_of(item);
    const uint4* t = ring + ((size_t)buf * kRows + r0) * units;
    int8_t* d = packed + (int64_t)tile_of(item) * (kRows * BITS / 8) + word * 4 +
                ((int64_t)slice_of(item) * slice + tid / BITS * 8) * pitch;
    for (int u = tid / BITS; u * 8 < span; u += kThreads / BITS, d += (kThreads / BITS * 8) * pitch) {
      const int g = PER_ROW ? 0 : group_of(u);
      const uint4* col = t + unit_at<BITS>(r0, u);
      uint32_t x[8];
#pragma unroll
      for (int j = 0; j < 8; ++j) x[j] = 0u;
      if (special) {
#pragma unroll 1
        for (int j = 0; j < 8; ++j) {
          uint32_t y = 0u;
#pragma unroll 1
          for (int i = kPer - 1; i >= 0; --i)
            y = (y << BITS) | ((uint32_t)encode_exact<BITS>(__half2float(reinterpret_cast<const __half*>(col + (size_t)i * units)[j]),
                                                            s_scale[g * kRows + r0 + i]) & ((1u << BITS) - 1u));
#pragma unroll
          for (int k = 0; k < 8; ++k)
            if (k == j) x[k] = y;
        }
      } else {
        // sums of (rounding constant + code) << position; the constants come off at the end
        const float2* qz = quant + g * (kRows + 1) + r0 + (r0 >> 4);
#pragma unroll
        for (int i = kPer - 1; i >= 0; --i) {
          const uint4 raw = col[(size_t)i * units];
          const float2 q = qz[i];
          const __half2 cap = *reinterpret_cast<const __half2*>(&q.y);
          const __half2* h = reinterpret_cast<const __half2*>(&raw);
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const float2 a = __half22float2(__hmin2(h[j], cap));
            x[2 * j] = (x[2 * j] << BITS) + __float_as_uint(fmaf(a.x, q.x, kMagic));
            x[2 * j + 1] = (x[2 * j + 1] << BITS) + __float_as_uint(fmaf(a.y, q.x, kMagic));
          }
        }
#pragma unroll
        for (int j = 0; j < 8; ++j) x[j] = (x[j] - kSum) ^ kSigns;
      }
#pragma unroll
      for (int j = 0; j < 8; ++j) *reinterpret_cast<uint32_t*>(d + j * pitch) = x[j];
    }
  };

  griddep_wait();  // a programmatic dependent that lets none start early: its outputs are weights
  for (int i = 0; i < kBufs; ++i) {
    if (first + i * step < items) load(first + i * step, i);
    commit();
  }
  if (PER_ROW) asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
  int buf = 0, place = 0;
  bool gave_up = false;  // a wait for maxima ran out
  uint32_t phase = 0u;
  if (PER_ROW && first < items) {
    asm volatile("cp.async.wait_group %0;" ::"n"(kBufs - 1) : "memory");
    push_maxima(first, 0, 0);
  }
  for (unsigned item = first; item < items; item += step) {
    bool special = false;  // the division has to make the codes
    bool lost = false;     // the wait for the item's maxima ran out
    const int next = buf + 1 == kBufs ? 0 : buf + 1, next_place = place + 1 == kPlaces ? 0 : place + 1;
    if (PER_ROW) {
      // the next item's maxima are on their way through the cluster while this one is quantised
      if (kBufs == 3) asm volatile("cp.async.wait_group 1;" ::: "memory");
      if (warp == 0) {
        const bool fine = wait_pushed(&max_bar[place], phase);
        if (fine) {
          unsigned m = 0u;
          for (unsigned c = 0; c < ranks; ++c) {
            const unsigned b = row_max[place][c][lane];
            m = max(m, b & 0x7fffu);
            special |= b >= 0x8000u;
          }
          special |= set_scale(item, 0, lane, m);
        } else {
          special = lost = true;
        }
        __syncwarp();
        // for the item kPlaces further on: no CTA pushes that one before this warp has pushed the next
        if (lane == 0 && fine) mbar_arrive_expect_tx(&max_bar[place], ranks * kRows * 4);
      }
      if (kBufs == 3 && item + step < items) push_maxima(item + step, next, next_place);
    } else {
      asm volatile("cp.async.wait_group %0;" ::"n"(kBufs - 1) : "memory");
      special = group_maxima(item, buf);
      __syncthreads();
      for (int i = tid; i < kRows * (span_of(item) / group); i += kThreads) {
        const int r = i % kRows, g = i / kRows;
        special |= set_scale(item, g, r, amax[r * amax_pitch + g]);
        amax[r * amax_pitch + g] = 0u;
      }
    }
    special = __syncthreads_or(special);
    if (PER_ROW && special && (gave_up = __syncthreads_or(lost))) break;  // nothing more is written
    quantise(item, buf, special);
    __syncthreads();  // the buffer is free
    if (item + kBufs * step < items) load(item + kBufs * step, buf);
    commit();
    if (PER_ROW && kBufs < 3) {
      asm volatile("cp.async.wait_group %0;" ::"n"(kBufs - 1) : "memory");
      if (item + step < items) push_maxima(item + step, next, next_place);
    }
    buf = next;
    place = next_place;
    if (place == 0) phase ^= 1u;
  }
  if (PER_ROW && gave_up) {
    // The other CTAs of the cluster have left, or meet here when their own waits run out (they miss what this one has
    // not pushed), so that none is gone while another still stores into its shared memory.
    if (tid == 0) atomicExch(&g_status, kStatusWaitTimeout);
    asm volatile("cp.async.wait_all;" ::: "memory");
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
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

constexpr int kMaxDevices = 64;
std::atomic<bool> g_launched[kMaxDevices];  // devices whose status word a wait may have set

template <int BITS, bool PER_ROW, int kThreads, int kBufs>
int launch_slices(const void* a, void* packed, void* scales, int64_t n, int64_t k, int group, const EncodePlan& plan,
                  cudaStream_t stream) {
  auto kern = encode_slices_kernel<BITS, PER_ROW, kThreads, kBufs>;
  static thread_local FitCache cache;
  int dev = 0;
  RB200_CUDA(cudaGetDevice(&dev));
  cudaLaunchConfig_t cfg = {};
  cfg.blockDim = dim3(kThreads, 1, 1);
  cfg.dynamicSmemBytes = plan.smem;
  cfg.stream = stream;
  const unsigned ranks = PER_ROW ? (unsigned)plan.slices : 1u;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = ranks;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  const int fit = cache.get(dev, (int)ranks, plan.smem, [&] {  // clusters that run at the same time
    int clusters = 0;
    cfg.gridDim = dim3(ranks * (unsigned)sm_count_current(), 1, 1);
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kEncodeSmem) != cudaSuccess ||
        cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess ||
        cudaOccupancyMaxActiveClusters(&clusters, kern, &cfg) != cudaSuccess) {
      cudaGetLastError();  // the kernel for any shape takes it
      return 0;
    }
    return clusters;
  });
  if (fit < 1) return 1;
  const int64_t items = n / kRows * (PER_ROW ? 1 : plan.slices);
  cfg.gridDim = dim3((unsigned)(items < fit ? items : fit) * ranks, 1, 1);
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.numAttrs = 2;
  RB200_CUDA(cudaLaunchKernelEx(&cfg, kern, static_cast<const __half*>(a), static_cast<int8_t*>(packed),
                                static_cast<__half*>(scales), n, k, plan.slice, plan.slices, group));
  if (dev >= 0 && dev < kMaxDevices) g_launched[dev].store(true, std::memory_order_relaxed);
  return 0;
}

template <int BITS>
int launch_rows(const void* a, void* packed, void* scales, int64_t n, int64_t k, const EncodePlan& plan, cudaStream_t stream) {
  if (plan.bufs == 2) return launch_slices<BITS, true, 512, 2>(a, packed, scales, n, k, 0, plan, stream);
  if (plan.bufs == 1) return launch_slices<BITS, true, 512, 1>(a, packed, scales, n, k, 0, plan, stream);
  return plan.threads == 256 ? launch_slices<BITS, true, 256, 3>(a, packed, scales, n, k, 0, plan, stream)
                             : launch_slices<BITS, true, 512, 3>(a, packed, scales, n, k, 0, plan, stream);
}
template <int BITS>
int launch_groups(const void* a, void* packed, void* scales, int64_t n, int64_t k, int group, const EncodePlan& plan,
                  cudaStream_t stream) {
  return plan.threads == 256 ? launch_slices<BITS, false, 256, 3>(a, packed, scales, n, k, group, plan, stream)
                             : launch_slices<BITS, false, 512, 3>(a, packed, scales, n, k, group, plan, stream);
}

}  // namespace

// Status of the quantiser's waits on the current device, cleared when set; 0 where nothing was launched.
int encode_read_status(int* status_out) {
  *status_out = 0;
  int dev = -1;
  RB200_CUDA(cudaGetDevice(&dev));
  if (dev < 0 || dev >= kMaxDevices || !g_launched[dev].load(std::memory_order_relaxed)) return 0;
  int v = 0;
  RB200_CUDA(cudaMemcpyFromSymbol(&v, g_status, sizeof(int)));
  if (v != 0) {
    const int zero = 0;
    RB200_CUDA(cudaMemcpyToSymbol(g_status, &zero, sizeof(int)));
  }
  *status_out = v;
  return 0;
}

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
    int rc = 1;
    EncodePlan plan;
    if (per_row) {
      if (plan_encode_rows(k, &plan))
        rc = weight_bits == 4 ? launch_rows<4>(a, packed, scales, n, k, plan, s) : launch_rows<8>(a, packed, scales, n, k, plan, s);
    } else if (group % 8 == 0 && plan_encode_groups(k, group, &plan) && n / kRows * plan.slices < (1ll << 31)) {
      rc = weight_bits == 4 ? launch_groups<4>(a, packed, scales, n, k, (int)group, plan, s)
                            : launch_groups<8>(a, packed, scales, n, k, (int)group, plan, s);
    }
    if (rc <= 0) return rc;
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
