#include "handover.h"

#include <atomic>
#include <mutex>

#include "common.cuh"

namespace rb200 {
namespace {

constexpr int kMaxDevices = 64;
constexpr int kMaxAreas = 32;

struct Area {
  uint32_t* words = nullptr;
  size_t bytes = 0;
  unsigned long long capture = 0, stream = 0;  // owner; capture 0: launches outside any capture
  bool owned = false;
  std::atomic<bool> given_back{false};         // by the destruction of the capture's graph
};
// Never destroyed: a graph may outlive every other static object.
struct Pool {
  std::mutex mutex;
  Area areas[kMaxAreas];
  int made = 0;
};
std::atomic<Pool*> g_pools[kMaxDevices];

Pool* pool_of_current_device() {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) return nullptr;
  Pool* p = g_pools[dev].load(std::memory_order_acquire);
  if (p) return p;
  Pool* fresh = new Pool();
  if (g_pools[dev].compare_exchange_strong(p, fresh)) return fresh;
  delete fresh;
  return p;
}

// runs on a thread of the driver, where no CUDA call is allowed
void CUDART_CB give_back(void* area) { static_cast<Area*>(area)->given_back.store(true, std::memory_order_release); }

// Allocation and fill that are legal whatever this thread or another one is capturing.
int make_area(Area& a, size_t bytes) {
  cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
  if (cudaThreadExchangeStreamCaptureMode(&mode) != cudaSuccess) return -1;
  int rc = cudaMalloc(reinterpret_cast<void**>(&a.words), bytes) == cudaSuccess ? 0 : -1;
  if (rc == 0 && fill_now(a.words, 0xff, bytes) != 0) {
    cudaFree(a.words);
    rc = -1;
  }
  if (rc == 0) a.bytes = bytes;
  else a.words = nullptr;
  cudaThreadExchangeStreamCaptureMode(&mode);
  return rc;
}

}  // namespace

uint32_t* handover_words(cudaStream_t stream, int sm_count, size_t bytes) {
  const size_t area_bytes = (size_t)sm_count * 128 * 256 * sizeof(float);  // a 128 x 256 tile per SM
  if (bytes > area_bytes) return nullptr;
  cudaStreamCaptureStatus status = cudaStreamCaptureStatusNone;
  unsigned long long capture = 0, id = 0;
  cudaGraph_t graph = nullptr;
  if (cudaStreamGetCaptureInfo(stream, &status, &capture, &graph) != cudaSuccess) {
    cudaGetLastError();
    return nullptr;
  }
  // A stream is known by its id, which no later stream takes over; asking for it while the stream captures
  // would invalidate the capture, but through a capture the handle itself stays with its stream.
  if (status == cudaStreamCaptureStatusActive) {
    id = (unsigned long long)reinterpret_cast<uintptr_t>(stream);
  } else {
    capture = 0;
    if (status != cudaStreamCaptureStatusNone || cudaStreamGetId(stream, &id) != cudaSuccess) {
      cudaGetLastError();
      return nullptr;
    }
  }
  Pool* p = pool_of_current_device();
  if (!p) return nullptr;
  std::lock_guard<std::mutex> lock(p->mutex);
  Area* a = nullptr;
  for (int i = 0; i < p->made; ++i) {
    Area& c = p->areas[i];
    if (c.given_back.exchange(false, std::memory_order_acquire)) c.owned = false;
    if (c.owned && c.capture == capture && c.stream == id) return c.words;
    if (!c.owned && !a) a = &c;
  }
  if (!a) {
    if (p->made == kMaxAreas || make_area(p->areas[p->made], area_bytes) != 0) {
      cudaGetLastError();
      return nullptr;
    }
    a = &p->areas[p->made++];
  }
  if (capture != 0) {
    cudaUserObject_t obj = nullptr;
    if (cudaUserObjectCreate(&obj, a, give_back, 1, cudaUserObjectNoDestructorSync) != cudaSuccess) {
      cudaGetLastError();
      return nullptr;
    }
    if (cudaGraphRetainUserObject(graph, obj, 1, cudaGraphUserObjectMove) != cudaSuccess) {
      cudaGetLastError();
      a->owned = true;  // until the object's destruction gives it back
      a->capture = a->stream = ~0ull;
      cudaUserObjectRelease(obj, 1);
      return nullptr;
    }
  }
  a->capture = capture;
  a->stream = id;
  a->owned = true;
  return a->words;
}

int handover_reset() {
  Pool* p = pool_of_current_device();
  if (!p) return 0;
  std::lock_guard<std::mutex> lock(p->mutex);
  for (int i = 0; i < p->made; ++i)
    if (fill_now(p->areas[i].words, 0xff, p->areas[i].bytes) != 0) return -1;
  return 0;
}

}  // namespace rb200
