// Device buffers on slabs, against a driver that only counts: `grow` prints the most
// bytes held while one buffer grows from 16 to 40 MB in small steps, `full` whether a
// 1 KB request succeeds where less than a slab is left.
#include <cstdio>
#include <cstring>
#include <map>

#include "dbuf.h"

namespace {
std::map<void*, size_t> g_live;
size_t g_held = 0, g_total = size_t(1) << 40, g_next = 4096, g_most = 0;
cudaError_t g_last = cudaSuccess;
cudaError_t note(cudaError_t e) {
  if (e != cudaSuccess) g_last = e;
  return e;
}
}  // namespace

extern "C" {
cudaError_t cudaMalloc(void** p, size_t n) {
  if (g_held + n > g_total) return note(cudaErrorMemoryAllocation);
  *p = reinterpret_cast<void*>(g_next);
  g_next += (n + 4095) / 4096 * 4096;
  g_live[*p] = n;
  g_held += n;
  g_most = g_held > g_most ? g_held : g_most;
  return cudaSuccess;
}
cudaError_t cudaFree(void* p) {
  g_held -= g_live[p];
  g_live.erase(p);
  return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void*, const void*, size_t, cudaMemcpyKind, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaGetLastError() {
  const cudaError_t e = g_last;
  g_last = cudaSuccess;
  return e;
}
const char* cudaGetErrorString(cudaError_t) { return "error"; }
}

int main(int argc, char** argv) {
  ftlm::Arena arena;
  ftlm::DBuf b;
  b.arena = &arena;
  if (argc > 1 && !std::strcmp(argv[1], "grow")) {
    const bool keep = argc > 2;
    for (size_t n = size_t(16) << 20; n <= size_t(40) << 20; n += size_t(200) << 10) {
      if (keep) b.ensure_keep(n, nullptr);
      else b.ensure(n);
      if (b.cap < n) return 1;
    }
    std::printf("%zu\n", g_most);
  } else {
    arena.held = size_t(21) << 20;  // slabs of 256 KB ... 16 MB are in use
    arena.size = arena.used = size_t(16) << 20;
    g_total = size_t(1) << 20;
    try {
      b.ensure(1024);
      std::printf("%d\n", b.p && b.cap >= 1024 && cudaGetLastError() == cudaSuccess);
    } catch (const ftlm::Error&) {
      std::printf("0\n");
    }
  }
  b.release();
  arena.release();
  return 0;
}
