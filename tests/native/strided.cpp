// copy_strided against a driver that refuses pitches above its limit, as CUDA does,
// and gives every address's index as its value. Prints the number of wrong values, or
// -1 for a refused copy.
#include <cstdio>
#include <cstdlib>
#include <vector>

#include "strided.h"

namespace {
constexpr uintptr_t kBase = 4096;
int64_t value(const void* p) { return static_cast<int64_t>((reinterpret_cast<uintptr_t>(p) - kBase) / 8); }
}  // namespace

extern "C" {
cudaError_t cudaMemcpy2DAsync(void* dst, size_t dpitch, const void* src, size_t spitch, size_t width, size_t height,
                              cudaMemcpyKind, cudaStream_t) {
  if (dpitch > 0x7fffffff || spitch > 0x7fffffff || width > spitch || width != 8) return cudaErrorInvalidPitchValue;
  for (size_t i = 0; i < height; ++i)
    *reinterpret_cast<int64_t*>(static_cast<char*>(dst) + i * dpitch) =
        value(reinterpret_cast<const void*>(reinterpret_cast<uintptr_t>(src) + i * spitch));
  return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void* dst, const void* src, size_t n, cudaMemcpyKind, cudaStream_t) {
  if (n != 8) return cudaErrorInvalidValue;
  *static_cast<int64_t*>(dst) = value(src);
  return cudaSuccess;
}
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaMalloc(void**, size_t) { return cudaErrorMemoryAllocation; }
cudaError_t cudaFree(void*) { return cudaSuccess; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
const char* cudaGetErrorString(cudaError_t) { return "error"; }
}

int main(int, char** argv) {
  const int64_t stride = std::atoll(argv[1]), count = std::atoll(argv[2]);
  std::vector<int64_t> out(static_cast<size_t>(count) + 1, -7);
  try {
    ftlm::copy_strided(out.data(), reinterpret_cast<const int64_t*>(kBase), stride, count, nullptr);
  } catch (const ftlm::Error&) {
    std::printf("-1\n");
    return 0;
  }
  int bad = out[static_cast<size_t>(count)] != -7;
  for (int64_t i = 0; i < count; ++i) bad += out[static_cast<size_t>(i)] != i * stride;
  std::printf("%d\n", bad);
  return 0;
}
