// Device scratch of one build (a plan's, a mesh's edge table's): blocks handed out in
// stack order from a few large allocations, all of them freed with the object.  A
// build makes some forty temporary arrays; as an allocation each they cost 10 us
// to make and, because freeing one waits for the device, 10 to 300 us to give back
// (measured, 64^3 P1 plan: 0.5 ms of allocations and 2 ms of frees; the plan's build
// as a whole 10.2 -> 7.4 ms with packed sort keys and the box from the mesh check).  Every user of one scratch works on one stream, so a block that is
// given back may be handed out again at once: the next use is ordered after the last.
#pragma once

#include <algorithm>
#include <cstddef>
#include <vector>

#include "mg_internal.h"

namespace mg {

class DeviceScratch {
 public:
  struct Mark {
    size_t chunk, used;
  };
  DeviceScratch() = default;
  DeviceScratch(const DeviceScratch&) = delete;
  DeviceScratch& operator=(const DeviceScratch&) = delete;
  ~DeviceScratch()
  {
    for (const Chunk& c : chunks_) cudaFree(c.base);
  }
  template <typename T>
  mg_status take(T** p, int64_t n)
  {
    const size_t bytes = (sizeof(T) * (size_t)std::max<int64_t>(n, 1) + 255) & ~(size_t)255;
    while (at_.chunk < chunks_.size() && chunks_[at_.chunk].size - at_.used < bytes) at_ = Mark{at_.chunk + 1, 0};
    if (at_.chunk == chunks_.size()) MG_TRY(grow(bytes));
    *p = reinterpret_cast<T*>(chunks_[at_.chunk].base + at_.used);
    at_.used += bytes;
    return MG_OK;
  }
  // room for `bytes` more in one allocation, so that the takes that follow need no other
  mg_status reserve(size_t bytes)
  {
    for (size_t c = at_.chunk; c < chunks_.size(); ++c)
      if (chunks_[c].size - (c == at_.chunk ? at_.used : 0) >= bytes) return MG_OK;
    return grow(bytes);
  }
  // frees everything (nothing may be in use) if it is more than `limit`
  void trim(size_t limit)
  {
    size_t all = 0;
    for (const Chunk& c : chunks_) all += c.size;
    if (all <= limit) return;
    for (const Chunk& c : chunks_) cudaFree(c.base);
    chunks_.clear();
    at_ = Mark{0, 0};
  }
  Mark mark() const { return at_; }
  void release(Mark m) { at_ = m; }

 private:
  struct Chunk {
    char* base;
    size_t size;
  };
  // at least 2 MiB (the driver's granularity) and a quarter of what there is
  mg_status grow(size_t bytes)
  {
    size_t all = 0;
    for (const Chunk& c : chunks_) all += c.size;
    const size_t round = (size_t)2 << 20;
    size_t size = (std::max(bytes, all / 4) + round - 1) / round * round;
    void* q = nullptr;
    cudaError_t e = cudaMalloc(&q, size);
    if (e != cudaSuccess && size > bytes) {  // little memory left: what is asked for, no more
      cudaGetLastError();
      size = bytes;
      e = cudaMalloc(&q, size);
    }
    if (e != cudaSuccess) return cuda_error(e, "device build scratch");
    chunks_.push_back(Chunk{static_cast<char*>(q), size});
    return MG_OK;
  }
  std::vector<Chunk> chunks_;
  Mark at_{0, 0};
};

// One scope's buffers: scratch, given back when the scope ends, and arrays for the
// plan, freed at the scope's end unless kept.
class BuildBuffers {
 public:
  explicit BuildBuffers(DeviceScratch& s) : scratch_(s), mark_(s.mark()) {}
  BuildBuffers(const BuildBuffers&) = delete;
  BuildBuffers& operator=(const BuildBuffers&) = delete;
  ~BuildBuffers()
  {
    for (void* q : ptrs_) cudaFree(q);
    scratch_.release(mark_);
  }
  template <typename T>
  mg_status temp(T** p, int64_t n)
  {
    return scratch_.take(p, n);
  }
  template <typename T>
  mg_status alloc(T** p, int64_t n)
  {
    void* q = nullptr;
    const cudaError_t e = cudaMalloc(&q, sizeof(T) * (size_t)std::max<int64_t>(n, 1));
    if (e != cudaSuccess) return cuda_error(e, "device plan buffer");
    ptrs_.push_back(q);
    *p = static_cast<T*>(q);
    return MG_OK;
  }
  void keep(void* q) { ptrs_.erase(std::remove(ptrs_.begin(), ptrs_.end(), q), ptrs_.end()); }

 private:
  DeviceScratch& scratch_;
  DeviceScratch::Mark mark_;
  std::vector<void*> ptrs_;
};

}  // namespace mg
