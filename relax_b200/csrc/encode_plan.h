// Host side of the quantiser that needs no device.
#pragma once

#include <cstddef>

namespace rb200 {

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
