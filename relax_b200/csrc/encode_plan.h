// Host side of the quantiser that needs no device.
#pragma once

#include <cstddef>
#include <cstdint>

namespace rb200 {

// How the kernel that reads the weight once is run: 32 rows x `slice` of k per item, `bufs` items of a CTA in shared
// memory.
struct EncodePlan {
  int slice, slices;  // slices of a row; one scale per row: a cluster of so many CTAs
  int bufs, threads;
  size_t smem;
};
constexpr int kEncodeRows = 32;
constexpr int kEncodeMaxCluster = 16;
constexpr size_t kEncodeSmem = 200 * 1024;

// Words from a row's group maxima to the next row's: odd, since a warp reads one group of all rows (fp16 11008 x 4096,
// groups of 8, an even pitch: 84 us instead of 55; groups of 16 53 instead of 41).
constexpr int encode_amax_pitch(int groups) { return groups | 1; }

inline size_t encode_smem(int64_t slice, int64_t groups, int bufs) {
  return (size_t)bufs * kEncodeRows * ((slice + 63) / 64 * 128) + (size_t)groups * ((kEncodeRows + 1) * 8 + kEncodeRows * 4) +
         (size_t)kEncodeRows * encode_amax_pitch((int)groups) * 4;
}

// Sixteen warps an SM: two CTAs of eight where two fit, else one of sixteen.  Two fit with slices of up to 512 k, but not
// with groups of 8, whose scales bring the shared memory to 129 KB (fp16 11008 x 4096, groups of 8: int4 55 us, with one
// CTA of eight warps 59; int8 55 / 64).  `places`: words for maxima; 1 KB of a CTA is the system's.
inline int encode_threads(size_t smem, size_t places) { return 2 * (smem + places * 4 + 64 + 1024) <= 228 * 1024 ? 256 : 512; }

// One scale per row (k % 8 == 0).  The slices of a row are a cluster, of eight CTAs up to 8192 k and sixteen above.
// Three buffers hold slices of up to 1024 k; above, two (up to 24576 k) and then one are still several times faster
// than the kernel for any shape.  False where not even one fits, above 50176 k.
inline bool plan_encode_rows(int64_t k, EncodePlan* p) {
  int64_t c = 1;
  while (c < 8 && k > c * 512) c *= 2;
  if (k > 8192) c = kEncodeMaxCluster;
  const int64_t slice = ((k + c - 1) / c + 7) / 8 * 8;
  int bufs = 3;
  while (bufs > 1 && encode_smem(slice, 1, bufs) > kEncodeSmem) --bufs;
  const size_t smem = encode_smem(slice, 1, bufs);
  if (smem > kEncodeSmem || (c - 1) * slice >= k) return false;
  *p = EncodePlan{(int)slice, (int)c, bufs, bufs == 3 ? encode_threads(smem, 3 * kEncodeMaxCluster * kEncodeRows) : 512, smem};
  return true;
}

// Groups (group % 8 == 0, k % group == 0): slices of whole groups.
inline bool plan_encode_groups(int64_t k, int64_t group, EncodePlan* p) {
  if (group > 1024) return false;
  const int64_t slice = (group > 512 ? 1024 : 512) / group * group, c = (k + slice - 1) / slice;
  if (c >= (1ll << 31)) return false;
  const size_t smem = encode_smem(slice, slice / group, 3);
  *p = EncodePlan{(int)slice, (int)c, 3, encode_threads(smem, 3 * kEncodeRows), smem};
  return true;
}

// How many clusters of a launch run at the same time, asked of the driver once per device and launch shape; 0 for a
// shape that does not fit is an answer like any other, kept with its shape.
struct FitCache {
  int device = -1, ranks = 0, fit = 0;
  size_t smem = 0;
  template <class Query>
  int get(int dev, int cluster_ranks, size_t smem_bytes, Query query) {
    if (device != dev || ranks != cluster_ranks || smem != smem_bytes) {
      fit = query();
      device = dev;
      ranks = cluster_ranks;
      smem = smem_bytes;
    }
    return fit;
  }
};

}  // namespace rb200
