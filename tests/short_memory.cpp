// Device allocations that fail on demand, in the place of the runtime's (linked
// with --wrap): the next `fail_next` of them, and all above `limit` bytes.
#include <cuda_runtime_api.h>

#include <cstddef>

static size_t g_limit = ~(size_t)0;
static int g_fail_next = 0, g_failed = 0, g_trims = 0;

extern "C" {
cudaError_t __real_cudaMalloc(void** p, size_t n);
cudaError_t __real_cudaMallocFromPoolAsync(void** p, size_t n, cudaMemPool_t pool, cudaStream_t s);
cudaError_t __real_cudaMemPoolTrimTo(cudaMemPool_t pool, size_t keep);

static bool fails(size_t n) {
  if (n <= g_limit && g_fail_next == 0) return false;
  if (g_fail_next) g_fail_next--;
  g_failed++;
  return true;
}
// (a size that no device has: the runtime's own error, with what it leaves behind)
cudaError_t __wrap_cudaMalloc(void** p, size_t n) { return __real_cudaMalloc(p, fails(n) ? (size_t)1 << 60 : n); }
cudaError_t __wrap_cudaMallocFromPoolAsync(void** p, size_t n, cudaMemPool_t pool, cudaStream_t s) {
  return __real_cudaMallocFromPoolAsync(p, fails(n) ? (size_t)1 << 60 : n, pool, s);
}
cudaError_t __wrap_cudaMemPoolTrimTo(cudaMemPool_t pool, size_t keep) {
  g_trims++;
  return __real_cudaMemPoolTrimTo(pool, keep);
}

void pk_test_memory(size_t limit, int fail_next) {
  g_limit = limit;
  g_fail_next = fail_next;
  g_failed = g_trims = 0;
}
int pk_test_memory_failed(void) { return g_failed; }
int pk_test_memory_trims(void) { return g_trims; }
}
