// Errors and grow-only device buffers (host code; no kernels).
#pragma once

#include <cuda_runtime.h>

#include <algorithm>
#include <cstddef>
#include <stdexcept>
#include <string>
#include <vector>

#include "../../include/ftlm_gpu.h"

namespace ftlm {

struct Error : std::runtime_error {
  int code;
  Error(int c, const std::string& m) : std::runtime_error(m), code(c) {}
};

#define FTLM_CUDA(call)                                                                  \
  do {                                                                                   \
    cudaError_t e_ = (call);                                                             \
    if (e_ != cudaSuccess)                                                               \
      throw ::ftlm::Error(FTLM_ERR_CUDA, std::string(#call) + ": " + cudaGetErrorString(e_)); \
  } while (0)

// Small device buffers of one context, cut from slabs that live as long as the
// context. A curve on a small lattice creates about 70 buffers and grows them, and
// a cudaMalloc and a cudaFree of each (which also wait for the device) took 0.1 to
// 1 ms apiece, by host: 15-30% of a curve. A region that a growing buffer leaves
// is not used again, so nothing waits for the kernels that still read it. A buffer
// at least doubles while it is on a slab (ensure_keep: grows by half), up to kMax,
// so what it leaves behind stays below 2 (3) kMax; a larger one is an allocation of
// its own, freed when it grows.
//
// Slabs grow from 256 KB to 64 MB: what is held doubles up to 1 MB (small calls stay
// with allocations the driver has at hand; a larger one takes it 0.4 ms), then each
// is four times the last.
struct Arena {
  static constexpr size_t kLast = size_t(64) << 20;
  static constexpr size_t kMax = size_t(32) << 20;  // largest buffer taken from a slab
  size_t first = size_t(256) << 10;  // the first slab's size
  std::vector<void*> slabs;
  size_t used = 0, size = 0;  // of the last slab
  size_t held = 0;            // all slabs
  void* take(size_t bytes) {
    bytes = (bytes + 255) / 256 * 256;
    if (used + bytes > size) {
      size_t next = std::max(bytes, std::min(kLast, std::max(first, held < (size_t(1) << 20) ? held : 4 * size)));
      void* p = nullptr;
      if (next > bytes && cudaMalloc(&p, next) != cudaSuccess) {  // near full memory: what is asked, no more
        cudaGetLastError();
        p = nullptr;
        next = bytes;
      }
      if (!p) FTLM_CUDA(cudaMalloc(&p, next));
      slabs.push_back(p);
      size = next;
      held += next;
      used = 0;
    }
    void* q = static_cast<char*>(slabs.back()) + used;
    used += bytes;
    return q;
  }
  void release() {
    for (void* p : slabs) cudaFree(p);
    slabs.clear();
    used = size = held = 0;
  }
};

// Grow-only device buffer owned by a context.
struct DBuf {
  void* p = nullptr;
  size_t cap = 0;
  Arena* arena = nullptr;  // where it is taken from up to Arena::kMax bytes
  bool own = false;        // p is an allocation of its own
  void ensure(size_t bytes) {
    if (bytes <= cap) return;
    // small buffers grow by doubling, from 4 KB in a slab and 64 KB alone: a curve
    // over many small sectors otherwise spends its time growing them
    const size_t first = arena ? kFirstBytes / 16 : kFirstBytes, small = arena ? Arena::kMax : kSmallBytes;
    if (bytes <= small) bytes = std::max(bytes, std::max(first, std::min(2 * cap, small)));
    release();
    get(bytes);
  }
  static constexpr size_t kFirstBytes = size_t(64) << 10, kSmallBytes = size_t(16) << 20;
  // Grows (by at least half) keeping the first `cap` bytes; stream-ordered copy.
  void ensure_keep(size_t bytes, cudaStream_t stream) {
    if (bytes <= cap) return;
    DBuf old = *this;
    p = nullptr;
    cap = 0;
    try {
      get(std::max(bytes, std::max(old.cap + old.cap / 2, arena ? size_t(64) << 10 : size_t(1) << 20)));
    } catch (...) {
      *this = old;
      throw;
    }
    if (!old.p) return;
    FTLM_CUDA(cudaMemcpyAsync(p, old.p, old.cap, cudaMemcpyDeviceToDevice, stream));
    if (old.own) FTLM_CUDA(cudaStreamSynchronize(stream));
    old.release();
  }
  template <typename T>
  T* as() const { return static_cast<T*>(p); }
  void release() {
    if (p && own) cudaFree(p);
    p = nullptr;
    cap = 0;
  }

 private:
  void get(size_t bytes) {
    if (arena && bytes <= Arena::kMax) {
      p = arena->take(bytes);
      own = false;
    } else {
      FTLM_CUDA(cudaMalloc(&p, bytes));
      own = true;
    }
    cap = bytes;
  }
};

}  // namespace ftlm
