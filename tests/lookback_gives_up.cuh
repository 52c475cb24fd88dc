// Included before pk_util.cu in a test's build: look-backs over `from` <= n < `to`
// elements give up at once, as one whose wait ran out does.
#include <cuda_runtime.h>
static __device__ unsigned g_gives_up[2][2];  // [scan, sort][from, to]
#define PK_SCAN_GIVES_UP(n) ((n) >= g_gives_up[0][0] && (n) < g_gives_up[0][1])
#define PK_SORT_GIVES_UP(n) ((n) >= g_gives_up[1][0] && (n) < g_gives_up[1][1])
extern "C" int pk_test_gives_up(int kind, unsigned from, unsigned to) {
  const unsigned range[2] = {from, to};
  return (int)cudaMemcpyToSymbol(g_gives_up, range, sizeof range, kind * sizeof range);
}
