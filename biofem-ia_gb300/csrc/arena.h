/*
 * Device memory of one owner (a mesh handle, its solver, its multigrid
 * hierarchy): many arrays carved out of few allocations of the stream-ordered
 * pool.  The pool's cost per allocation grows with the number of streams that
 * have used it (0.8 us with one, 13 us with 16, 40 us with 48, and an order of
 * magnitude more when 16 threads allocate at once: measured), and a handle has
 * some 140 arrays; allocated one by one they were most of a served batch's
 * time.
 *
 * Slabs grow with what the owner already holds, a quarter of it between 2 and
 * 32 MB, so that little is left unused; an array larger than half a slab gets
 * an allocation of its own, and where a slab can't be had the array alone is
 * tried.
 */
#ifndef BIOFEM_ARENA_H
#define BIOFEM_ARENA_H

#include <cuda_runtime.h>

#include <algorithm>
#include <vector>

namespace biofem {

class Arena {
 public:
  cudaError_t get(void **p, size_t bytes, cudaStream_t st)
  {
    bytes = (std::max<size_t>(bytes, 1) + kAlign - 1) / kAlign * kAlign;
    if (bytes > left_) {
      const size_t slab = std::min(std::max(held_ / 4, kMinSlab), kMaxSlab);
      if (bytes > slab / 2) return take(p, bytes, st);
      void *q = nullptr;
      if (take(&q, slab, st) != cudaSuccess) {
        cudaGetLastError();
        return take(p, bytes, st);
      }
      cur_ = static_cast<char *>(q);
      left_ = slab;
    }
    *p = cur_;
    cur_ += bytes;
    left_ -= bytes;
    return cudaSuccess;
  }

  /* device memory taken from the pool, the unused ends of slabs included */
  size_t held() const { return held_; }

  void release(cudaStream_t st)
  {
    for (void *p : slabs_) cudaFreeAsync(p, st);
    slabs_.clear();
    cur_ = nullptr;
    left_ = held_ = 0;
  }

 private:
  static constexpr size_t kAlign = 256, kMinSlab = 2 << 20, kMaxSlab = 32 << 20;

  cudaError_t take(void **p, size_t bytes, cudaStream_t st)
  {
    const cudaError_t e = cudaMallocAsync(p, bytes, st);
    if (e == cudaSuccess) {
      slabs_.push_back(*p);
      held_ += bytes;
    }
    return e;
  }

  std::vector<void *> slabs_;
  char *cur_ = nullptr;
  size_t left_ = 0, held_ = 0;
};

}  /* namespace biofem */

#endif
