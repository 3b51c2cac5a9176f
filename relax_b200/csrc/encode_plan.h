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

inline size_t encode_smem(int64_t slice, int64_t groups, int bufs) {
  return (size_t)bufs * kEncodeRows * ((slice + 63) / 64 * 128) + (size_t)groups * ((kEncodeRows + 1) * 8 + kEncodeRows * 8);
}

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
  // two CTAs per SM where a slice is at most 512 k (100 KB of shared memory), else one: sixteen warps either way
  *p = EncodePlan{(int)slice, (int)c, bufs, slice <= 512 ? 256 : 512, smem};
  return true;
}

// Groups (group % 8 == 0, k % group == 0): slices of whole groups.
inline bool plan_encode_groups(int64_t k, int64_t group, EncodePlan* p) {
  if (group > 1024) return false;
  const int64_t slice = (group > 512 ? 1024 : 512) / group * group, c = (k + slice - 1) / slice;
  if (c >= (1ll << 31)) return false;
  *p = EncodePlan{(int)slice, (int)c, 3, slice <= 512 ? 256 : 512, encode_smem(slice, slice / group, 3)};
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
