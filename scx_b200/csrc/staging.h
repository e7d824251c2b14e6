// Host staging of small results.
#pragma once

#include <cuda_runtime_api.h>

#include <cstdlib>
#include <mutex>
#include <new>
#include <utility>
#include <vector>

namespace scx {

// Page-locked staging of small results: device-to-host copies into it run
// without the driver's own staging and its wait per copy, and one
// synchronisation serves them all.  Buffers go back to a list that keeps at most
// kStageHeld bytes; a buffer whose copies may still run is waited for first.
// Where page-locked memory is refused a buffer is ordinary memory, freed after
// its use: the same copies, each with the driver's wait.
constexpr size_t kStageMost = size_t(16) << 20;  // larger results are copied directly
constexpr size_t kStageHeld = size_t(64) << 20;
struct StageList {
  std::mutex mu;
  std::vector<std::pair<void*, size_t>> idle;
  size_t held = 0;
};
inline StageList& stage_list() {
  static StageList* l = new StageList;  // never destroyed: plans may outlive static objects
  return *l;
}
struct Staging {
  char* p = nullptr;
  size_t bytes = 0;
  cudaStream_t busy = nullptr;  // stream whose copies into the buffer have not been waited for
  bool pending = false;
  bool locked = true;
  explicit Staging(size_t need, cudaStream_t st) : busy(st) {
    StageList& l = stage_list();
    {
      std::lock_guard<std::mutex> lock(l.mu);
      size_t best = l.idle.size();
      for (size_t i = 0; i < l.idle.size(); ++i)
        if (l.idle[i].second >= need && (best == l.idle.size() || l.idle[i].second < l.idle[best].second)) best = i;
      if (best < l.idle.size()) {
        p = static_cast<char*>(l.idle[best].first);
        bytes = l.idle[best].second;
        l.held -= bytes;
        l.idle.erase(l.idle.begin() + best);
        return;
      }
    }
    bytes = size_t(1) << 16;
    while (bytes < need) bytes *= 2;
    void* q = nullptr;
    if (cudaHostAlloc(&q, bytes, cudaHostAllocPortable) != cudaSuccess) {
      cudaGetLastError();  // not the error of a later call
      locked = false;
      q = malloc(bytes);
      if (!q) throw std::bad_alloc();
    }
    p = static_cast<char*>(q);
  }
  Staging(const Staging&) = delete;
  Staging& operator=(const Staging&) = delete;
  cudaError_t fetch(size_t at, const void* src, size_t n) {
    pending = true;
    return cudaMemcpyAsync(p + at, src, n, cudaMemcpyDeviceToHost, busy);
  }
  cudaError_t wait() {
    const cudaError_t e = cudaStreamSynchronize(busy);
    if (e == cudaSuccess) pending = false;
    return e;
  }
  template <typename T> const T* at(size_t o) const { return reinterpret_cast<const T*>(p + o); }
  ~Staging() {
    if (pending) cudaStreamSynchronize(busy);
    if (!locked) {
      free(p);
      return;
    }
    StageList& l = stage_list();
    try {
      std::lock_guard<std::mutex> lock(l.mu);
      if (l.held + bytes <= kStageHeld) {
        l.idle.emplace_back(p, bytes);
        l.held += bytes;
        return;
      }
    } catch (...) {  // no room for the list to grow: the buffer goes back instead
    }
    cudaFreeHost(p);
  }
};

}  // namespace scx
