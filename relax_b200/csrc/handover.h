// Hand-over words: fp32 parts of a tile that several CTAs of one launch computed together (umma_sk.cuh,
// umma_pair.cuh), vacant - all bits set - between launches.
//
// Launches that may overlap must not share them, so an area belongs to one order of launches: a stream, or,
// under capture, what one stream contributes to one capture (the graph's launches run in that order whenever
// and wherever it is replayed; the graph gives the area back when it and its instances are gone).  At most
// kMaxAreas per device, 19 MB each; a launch without one computes whole tiles only, which needs none.
#pragma once

#include <cuda_runtime.h>
#include <stddef.h>
#include <stdint.h>

namespace rb200 {

// The area for a launch on `stream` of the current device, nullptr when there is none (never an error).
// Made on the first call, also inside a capture; `bytes`: what the launch needs.
uint32_t* handover_words(cudaStream_t stream, int sm_count, size_t bytes);

// Every area of the current device back to rest; nothing that uses one may be running.
int handover_reset();

}  // namespace rb200
