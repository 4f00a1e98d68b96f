// Test harness: the pinned staging buffer (HBuf) on a fake of the pinning call
// that refuses more than a limit.  Not part of the library.
#include <cstdio>
#include <cstdlib>

#include "../../rabbitbin_b200/csrc/engine_internal.h"

static size_t g_limit = 0;

static cudaError_t pin(void **p, size_t bytes) {
  *p = bytes <= g_limit ? std::malloc(bytes) : nullptr;
  return *p ? cudaSuccess : cudaErrorMemoryAllocation;
}
extern "C" {
cudaError_t cudaMallocHost(void **p, size_t bytes) { return pin(p, bytes); }
cudaError_t cudaHostAlloc(void **p, size_t bytes, unsigned) { return pin(p, bytes); }
cudaError_t cudaFreeHost(void *p) {
  std::free(p);
  return cudaSuccess;
}
cudaError_t cudaGetLastError() { return cudaSuccess; }
const char *cudaGetErrorString(cudaError_t) { return "fake"; }
}

// Limit of the pinning call, then sizes asked for in turn; prints the capacity
// after each, -1 where the size is refused.
int main(int argc, char **argv) {
  g_limit = std::strtoull(argv[1], nullptr, 10);
  rbg::HBuf b;
  for (int i = 2; i < argc; ++i) {
    try {
      b.ensure(std::strtoull(argv[i], nullptr, 10));
      std::printf("%zu\n", b.cap);
    } catch (const rbg::Error &) {
      std::printf("-1\n");
    }
  }
  b.release();
  return 0;
}
