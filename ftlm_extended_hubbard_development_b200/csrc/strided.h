// Strided device values to the host (host code; no kernels).
#pragma once

#include <cuda_runtime.h>

#include <cstddef>
#include <cstdint>

#include "dbuf.h"

namespace ftlm {

// Largest pitch of a 2D copy: cudaDevAttrMaxPitch on sm_100a.
constexpr int64_t kMaxCopyPitch = 0x7fffffff;

// dst[i] = src[i * stride] for i < count, complete on return: one 2D copy where the
// stride in bytes is a pitch that CUDA takes, else a copy per value (8x4 (0, 16):
// 6.0e8 words a class, 4.8 GB).
inline void copy_strided(int64_t* dst, const int64_t* src, int64_t stride, int64_t count, cudaStream_t st) {
  const int64_t pitch = stride * static_cast<int64_t>(sizeof(int64_t));
  if (pitch <= kMaxCopyPitch) {
    FTLM_CUDA(cudaMemcpy2DAsync(dst, sizeof(int64_t), src, static_cast<size_t>(pitch), sizeof(int64_t),
                                static_cast<size_t>(count), cudaMemcpyDeviceToHost, st));
  } else {
    for (int64_t i = 0; i < count; ++i)
      FTLM_CUDA(cudaMemcpyAsync(dst + i, src + i * stride, sizeof(int64_t), cudaMemcpyDeviceToHost, st));
  }
  FTLM_CUDA(cudaStreamSynchronize(st));
}

}  // namespace ftlm
