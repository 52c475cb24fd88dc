// pk_util.cu -- device-wide exclusive scan (single pass, decoupled look-back),
// a stable LSD radix sort of 64-bit keys and the level lists of a binary tree,
// used by the BVH and env builders.
#include <cuda_runtime.h>
#include <unistd.h>

#include <algorithm>
#include <mutex>
#include <string>
#include <utility>
#include <utility>
#include <vector>

#include "pk_internal.cuh"
#include "pk_util.h"

namespace pk {

void touch_pages(void* p, size_t bytes) {
  cudaPointerAttributes a;
  if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
    cudaGetLastError();
    return;
  }
  if (a.type != cudaMemoryTypeUnregistered) return;  // pinned, or not the host's to touch
  static const size_t page = (size_t)std::max(4096l, sysconf(_SC_PAGESIZE));
  volatile char* b = static_cast<volatile char*>(p);
  for (size_t i = 0; i < bytes; i += page) b[i] = b[i];
  if (bytes) b[bytes - 1] = b[bytes - 1];
}

// The pools that exist, for device_malloc; contexts come and go on several threads.
// (Never destroyed: a context may be closed after this library's statics.)
static std::mutex& g_pools_lock = *new std::mutex;
static std::vector<std::pair<int, cudaMemPool_t>>& g_pools = *new std::vector<std::pair<int, cudaMemPool_t>>;

static void give_pools_back() {
  int device = 0;
  cudaGetDevice(&device);
  std::lock_guard<std::mutex> hold(g_pools_lock);
  for (const auto& p : g_pools)
    if (p.first == device) cudaMemPoolTrimTo(p.second, 0);
}

template <class F>
static void* malloc_or_throw(const char* what, F attempt) {
  void* p = nullptr;
  cudaError_t e = attempt(&p);
  if (e == cudaErrorMemoryAllocation) {
    cudaGetLastError();
    give_pools_back();
    e = attempt(&p);
  }
  if (e != cudaSuccess) {
    cudaGetLastError();
    check(e, what);
  }
  return p;
}
void* device_malloc(size_t bytes) {
  return malloc_or_throw("cudaMalloc", [&](void** p) { return cudaMalloc(p, bytes); });
}
void* scratch_malloc(const Scratch& w, size_t bytes) {
  return malloc_or_throw("cudaMallocFromPoolAsync",
                         [&](void** p) { return cudaMallocFromPoolAsync(p, bytes, w.pool, w.s); });
}

void destroy_scratch_pool(cudaMemPool_t pool) {
  if (!pool) return;
  std::lock_guard<std::mutex> hold(g_pools_lock);
  for (size_t i = 0; i < g_pools.size(); i++)
    if (g_pools[i].second == pool) {
      g_pools.erase(g_pools.begin() + i);
      break;
    }
  cudaMemPoolDestroy(pool);
}

cudaMemPool_t create_scratch_pool(int device) {
  cudaMemPoolProps props = {};
  props.allocType = cudaMemAllocationTypePinned;
  props.location.type = cudaMemLocationTypeDevice;
  props.location.id = device;
  cudaMemPool_t pool = nullptr;
  check(cudaMemPoolCreate(&pool, &props), "cudaMemPoolCreate");
  uint64_t keep = SCRATCH_KEEP;
  const cudaError_t e = cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep);
  if (e != cudaSuccess) {
    cudaMemPoolDestroy(pool);
    check(e, "cudaMemPoolSetAttribute");
  }
  std::lock_guard<std::mutex> hold(g_pools_lock);
  g_pools.emplace_back(device, pool);
  return pool;
}

void check_lookback(uint32_t err, const char* what) {
  if (err & ERR_LOOKBACK) throw CudaError(std::string(what) + ": a look-back timed out");
}

// A test's build says which look-backs (of n elements) give up at once, so that
// what follows a wait that ran out can be watched.
#ifndef PK_SCAN_GIVES_UP
#define PK_SCAN_GIVES_UP(n) false
#endif
#ifndef PK_SORT_GIVES_UP
#define PK_SORT_GIVES_UP(n) false
#endif

constexpr int SCAN_THREADS = 256;
constexpr int SCAN_ITEMS = 8;
constexpr int SCAN_TILE = SCAN_THREADS * SCAN_ITEMS;

__global__ void __launch_bounds__(SCAN_THREADS) k_scan_u32(const uint32_t* in, uint32_t* out,
                                                          uint32_t n, uint32_t* __restrict__ total,
                                                          unsigned long long* __restrict__ tiles,
                                                          uint32_t* __restrict__ ticket, uint32_t* __restrict__ err) {
  __shared__ uint32_t s_tile;
  __shared__ uint32_t s_warp[SCAN_THREADS / 32 + 1][2];
  __shared__ unsigned long long s_excl;
  const uint32_t ntiles = (n + SCAN_TILE - 1) / SCAN_TILE;
  for (;;) {
    if (threadIdx.x == 0) s_tile = atomicAdd(ticket, 1u);
    __syncthreads();
    const uint32_t tile = s_tile;
    if (tile >= ntiles) break;
    const size_t base = (size_t)tile * SCAN_TILE + (size_t)threadIdx.x * SCAN_ITEMS;
    uint32_t v[SCAN_ITEMS];
    uint32_t sum = 0;
#pragma unroll
    for (int k = 0; k < SCAN_ITEMS; k++) {
      v[k] = (base + k < n) ? in[base + k] : 0u;
      sum += v[k];
    }
    uint32_t ea, eb, ta, tb;
    block_scan2<SCAN_THREADS / 32>(sum, 0u, ea, eb, ta, tb, s_warp);
    if (threadIdx.x < 32) {
      unsigned long long e = 0;
      if (!PK_SCAN_GIVES_UP(n)) e = lookback2_warp(tiles, tile, pack2(ta, 0u), err);
      else if (tile) atomicOr(err, ERR_LOOKBACK);
      if (threadIdx.x == 0) s_excl = e;
    }
    __syncthreads();
    uint32_t run = unpack_a(s_excl) + ea;
#pragma unroll
    for (int k = 0; k < SCAN_ITEMS; k++) {
      if (base + k < n) out[base + k] = run;
      run += v[k];
    }
    if (tile == ntiles - 1 && threadIdx.x == 0 && total) *total = unpack_a(s_excl) + ta;
    __syncthreads();
  }
}

static int multiprocessors() {
  int dev = 0, sms = 1;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  return sms;
}

void scan_exclusive_u32(const Scratch& w, const uint32_t* in, uint32_t* out, uint32_t n, uint32_t* total,
                        uint32_t* err) {
  if (n == 0) {
    if (total) check(cudaMemsetAsync(total, 0, 4, w.s), "memset");
    return;
  }
  const uint32_t ntiles = (n + SCAN_TILE - 1) / SCAN_TILE;
  TmpBuf<unsigned long long> state(w, (size_t)ntiles + 1);  // tile states, then the ticket
  check(cudaMemsetAsync(state.p, 0, state.bytes(), w.s), "memset");
  const unsigned grid = (unsigned)std::min<uint32_t>(ntiles, (uint32_t)multiprocessors() * 4u);
  k_scan_u32<<<grid, SCAN_THREADS, 0, w.s>>>(in, out, n, total, state.p, reinterpret_cast<uint32_t*>(state.p + ntiles),
                                             err);
  check(cudaGetLastError(), "k_scan_u32");
}

// ---------------- exclusive scan of 64-bit values (three phases) -------------
// Tiles of SCAN_TILE values: each block scans its tile and writes the tile's
// sum; the tile sums are scanned recursively; a last pass adds each tile's
// offset.  Integer sums do not depend on the grouping.  A tile's sum is the result
// of at most 8 (thread) + 5 (warp) + 8 (warps) additions, a prefix within a tile
// of 8 more and one, and every further level adds a tile's sum and the offset:
// at most 30 + 2 * 22 for three levels.
template <class T>
__device__ __forceinline__ T warp_scan_incl(T v) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const T x = __shfl_up_sync(0xffffffffu, v, o);
    if (lane >= o) v += x;
  }
  return v;
}

template <class T>
__global__ void __launch_bounds__(SCAN_THREADS) k_scan64_tiles(const T* in, T* out, size_t n,
                                                               T* __restrict__ tile_sums) {
  __shared__ T s_warp[SCAN_THREADS / 32];
  const size_t base = (size_t)blockIdx.x * SCAN_TILE + (size_t)threadIdx.x * SCAN_ITEMS;
  T v[SCAN_ITEMS], sum = 0;
#pragma unroll
  for (int k = 0; k < SCAN_ITEMS; k++) {
    v[k] = base + k < n ? in[base + k] : (T)0;
    sum += v[k];
  }
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const T incl = warp_scan_incl(sum);
  T excl = __shfl_up_sync(0xffffffffu, incl, 1);  // no subtraction: a double prefix stays a sum of what it covers
  if (lane == 0) excl = 0;
  if (lane == 31) s_warp[warp] = incl;
  __syncthreads();
  T woff = 0, tot = 0;
  for (int k = 0; k < SCAN_THREADS / 32; k++) {
    if (k < warp) woff += s_warp[k];
    tot += s_warp[k];
  }
  T run = woff + excl;
#pragma unroll
  for (int k = 0; k < SCAN_ITEMS; k++) {
    if (base + k < n) out[base + k] = run;
    run += v[k];
  }
  if (threadIdx.x == 0) tile_sums[blockIdx.x] = tot;
}

template <class T>
__global__ void k_scan64_add(T* out, size_t n, const T* __restrict__ tile_offs) {
  const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) out[i] += tile_offs[i / SCAN_TILE];
}

template <class T>
static void scan64(const Scratch& w, const T* in, T* out, size_t n) {
  if (n == 0) return;
  const size_t ntiles = (n + SCAN_TILE - 1) / SCAN_TILE;
  TmpBuf<T> sums(w, ntiles);
  k_scan64_tiles<T><<<(unsigned)ntiles, SCAN_THREADS, 0, w.s>>>(in, out, n, sums.p);
  check(cudaGetLastError(), "k_scan64_tiles");
  if (ntiles > 1) {
    scan64<T>(w, sums.p, sums.p, ntiles);
    k_scan64_add<T><<<(unsigned)((n + 255) / 256), 256, 0, w.s>>>(out, n, sums.p);
    check(cudaGetLastError(), "k_scan64_add");
  }
}
void scan_exclusive_u64(const Scratch& w, const unsigned long long* in, unsigned long long* out, size_t n) {
  scan64<unsigned long long>(w, in, out, n);
}
void scan_exclusive_f64(const Scratch& w, const double* in, double* out, size_t n) { scan64<double>(w, in, out, n); }

// ---------------- stable LSD radix sort -------------------------------------
// One kernel per 8-bit digit (after Adinets & Merrill, "Onesweep: A Faster
// Least Significant Digit Radix Sort for GPUs", 2022): one pass over the keys
// counts all eight digits; then each pass ranks a tile of keys in shared
// memory, finds the tile's offset per digit by decoupled look-back (256
// independent chains, one per thread) and writes the tile out in digit order,
// so every key is read and written once per pass.  Bound by the 24 bytes per
// pair and pass; several equal-length arrays sort in the same launches
// (blockIdx.y).
constexpr int SORT_THREADS = 256;
constexpr int SORT_WARPS = SORT_THREADS / 32;
// rounds of 32 keys per warp (2048x1024 map's tables: 6 929 us, 8 915, 10 925, 12 948)
constexpr int SORT_ROUNDS = 8;
constexpr int SORT_TILE = SORT_THREADS * SORT_ROUNDS;  // 2048 keys per block: 24 KB of pairs in shared memory
constexpr int RADIX = 256;
constexpr int SORT_PASSES = 8;
constexpr uint32_t SORT_BACK = 4;  // tiles a look-back reads at once (2048x1024 map: 1 958 us, 4 948, 8 953, 16 965)
static_assert(SORT_THREADS == RADIX, "one thread per digit");

__global__ void __launch_bounds__(SORT_THREADS) k_sort_hist(const uint64_t* __restrict__ keys, uint32_t n,
                                                            uint32_t* __restrict__ hist) {
  __shared__ uint32_t h[SORT_PASSES][RADIX];
  for (int i = threadIdx.x; i < SORT_PASSES * RADIX; i += SORT_THREADS) (&h[0][0])[i] = 0;
  __syncthreads();
  const uint64_t* in = keys + (size_t)blockIdx.y * n;
  const int lane = threadIdx.x & 31;
  const size_t stride = (size_t)gridDim.x * SORT_THREADS;
  for (size_t base = (size_t)blockIdx.x * SORT_THREADS + (threadIdx.x - lane); base < n; base += stride) {
    const size_t i = base + lane;
    const bool on = i < n;
    const uint64_t k = on ? in[i] : 0;
    const uint32_t act = __ballot_sync(0xffffffffu, on);
    if (on) {
#pragma unroll
      for (int p = 0; p < SORT_PASSES; p++) {
        const uint32_t d = (uint32_t)(k >> (8 * p)) & 0xffu;
        int same;  // digits that the whole warp shares (the high ones mostly) cost one atomic
        __match_all_sync(act, d, &same);
        if (!same) atomicAdd(&h[p][d], 1u);
        else if (lane == __ffs(act) - 1) atomicAdd(&h[p][d], (uint32_t)__popc(act));
      }
    }
  }
  __syncthreads();
  uint32_t* out = hist + (size_t)blockIdx.y * SORT_PASSES * RADIX;
  for (int i = threadIdx.x; i < SORT_PASSES * RADIX; i += SORT_THREADS) {
    const uint32_t c = (&h[0][0])[i];
    if (c) atomicAdd(out + i, c);
  }
}

// Look-back words: the top two bits say what the rest holds (1: this tile's
// count, 2: the inclusive prefix).  32 bits for fewer than 2^30 keys, else 64.
template <class W>
struct SortWord;
template <>
struct SortWord<uint32_t> {
  static constexpr uint32_t AGG = 1u << 30, PRE = 2u << 30, VAL = (1u << 30) - 1u;
  static __device__ __forceinline__ uint32_t load(const uint32_t* p) {
    uint32_t v;
    asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
  }
  static __device__ __forceinline__ void store(uint32_t* p, uint32_t v) {
    asm volatile("st.relaxed.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
  }
};
template <>
struct SortWord<unsigned long long> {
  static constexpr unsigned long long AGG = TILE_AGG, PRE = TILE_PRE, VAL = TILE_VAL;
  static __device__ __forceinline__ unsigned long long load(const unsigned long long* p) { return ld_word(p); }
  static __device__ __forceinline__ void store(unsigned long long* p, unsigned long long v) { st_word(p, v); }
};

// Exclusive prefix over the block's threads (one digit each).
__device__ __forceinline__ uint32_t digit_scan(uint32_t v, uint32_t* s_warp) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint32_t inc = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t x = __shfl_up_sync(0xffffffffu, inc, o);
    if (lane >= o) inc += x;
  }
  if (lane == 31) s_warp[warp] = inc;
  __syncthreads();
  uint32_t before = 0;
#pragma unroll
  for (int k = 0; k < SORT_WARPS; k++)
    if (k < warp) before += s_warp[k];
  __syncthreads();
  return before + inc - v;
}

template <class W>
__global__ void __launch_bounds__(SORT_THREADS) k_sort_pass(const uint64_t* __restrict__ keys,
                                                            const uint32_t* __restrict__ vals, uint32_t n, int pass,
                                                            uint32_t ntiles, const uint32_t* __restrict__ hist,
                                                            W* __restrict__ state, uint32_t* __restrict__ tickets,
                                                            uint64_t* __restrict__ keys_out,
                                                            uint32_t* __restrict__ vals_out, uint32_t* err) {
  __shared__ uint64_t s_key[SORT_TILE];
  __shared__ uint32_t s_val[SORT_TILE];
  __shared__ uint32_t wh[SORT_WARPS][RADIX];
  __shared__ uint32_t s_out[RADIX];  // where the tile's first key of a digit goes, less its place in the tile
  __shared__ uint32_t s_warp[SORT_WARPS];
  __shared__ uint32_t s_tile;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const uint32_t seg = blockIdx.y;
  if (threadIdx.x == 0) s_tile = atomicAdd(tickets + seg, 1u);  // tiles in the order blocks start
  for (int i = threadIdx.x; i < SORT_WARPS * RADIX; i += SORT_THREADS) (&wh[0][0])[i] = 0;
  __syncthreads();
  const uint32_t tile = s_tile;
  const int shift = 8 * pass;
  const uint64_t* kin = keys + (size_t)seg * n;
  const uint32_t* vin = vals + (size_t)seg * n;
  const size_t wbase = (size_t)tile * SORT_TILE + (size_t)warp * (SORT_ROUNDS * 32);
  const uint32_t lt = (1u << lane) - 1u;
  uint64_t key[SORT_ROUNDS];
  uint32_t val[SORT_ROUNDS], rank[SORT_ROUNDS];
#pragma unroll
  for (int r = 0; r < SORT_ROUNDS; r++) {
    const size_t i = wbase + (size_t)r * 32 + lane;
    key[r] = i < n ? kin[i] : 0;
    val[r] = i < n ? vin[i] : 0;
  }
#pragma unroll
  for (int r = 0; r < SORT_ROUNDS; r++) {
    const size_t i = wbase + (size_t)r * 32 + lane;
    const uint32_t d = i < n ? (uint32_t)(key[r] >> shift) & 0xffu : RADIX;
    const uint32_t peers = __match_any_sync(0xffffffffu, d);
    uint32_t pre = 0;
    if (d < RADIX) pre = wh[warp][d];
    __syncwarp();
    rank[r] = pre + (uint32_t)__popc(peers & lt);
    if (d < RADIX && (peers & lt) == 0) wh[warp][d] = pre + (uint32_t)__popc(peers);
    __syncwarp();
  }
  __syncthreads();
  const int d = threadIdx.x;
  uint32_t count = 0;
  for (int k = 0; k < SORT_WARPS; k++) {  // exclusive prefix over warps, in place
    const uint32_t c = wh[k][d];
    wh[k][d] = count;
    count += c;
  }
  using L = SortWord<W>;
  W* mine = state + ((size_t)seg * ntiles + tile) * RADIX + d;
  L::store(mine, (tile == 0 ? L::PRE : L::AGG) | (W)count);
  const uint32_t local = digit_scan(count, s_warp);
  const uint32_t global = digit_scan(hist[((size_t)seg * SORT_PASSES + pass) * RADIX + d], s_warp);
  for (int k = 0; k < SORT_WARPS; k++) wh[k][d] += local;
  W before = 0;
  if (tile) {  // SORT_BACK earlier tiles at a time, back to the nearest inclusive prefix
    const W* p = mine;
    bool found = PK_SORT_GIVES_UP(n);
    if (found) atomicOr(err, ERR_LOOKBACK);
    for (uint32_t t = tile; t && !found; p -= SORT_BACK * RADIX, t = t > SORT_BACK ? t - SORT_BACK : 0u) {
      W v[SORT_BACK];
#pragma unroll
      for (uint32_t k = 0; k < SORT_BACK; k++) v[k] = k < t ? L::load(p - (size_t)(k + 1) * RADIX) : L::PRE;
#pragma unroll
      for (uint32_t k = 0; k < SORT_BACK; k++) {
        if (found) continue;
        int spins = 0;
        while ((v[k] & ~L::VAL) == 0) {
          if (++spins > LOOKBACK_SPIN_LIMIT) {
            atomicOr(err, ERR_LOOKBACK);
            v[k] = L::PRE;
            break;
          }
          __nanosleep(32);
          v[k] = L::load(p - (size_t)(k + 1) * RADIX);
        }
        before += v[k] & L::VAL;
        found = (v[k] & ~L::VAL) == L::PRE;
      }
    }
    L::store(mine, L::PRE | (before + (W)count));
  }
  s_out[d] = global + (uint32_t)before - local;
  __syncthreads();
#pragma unroll
  for (int r = 0; r < SORT_ROUNDS; r++) {
    const size_t i = wbase + (size_t)r * 32 + lane;
    if (i >= n) continue;
    const uint32_t pos = wh[warp][(uint32_t)(key[r] >> shift) & 0xffu] + rank[r];
    s_key[pos] = key[r];
    s_val[pos] = val[r];
  }
  __syncthreads();
  const size_t first = (size_t)tile * SORT_TILE;
  const uint32_t here = (uint32_t)(n - first < (size_t)SORT_TILE ? n - first : (size_t)SORT_TILE);
  for (uint32_t i = threadIdx.x; i < here; i += SORT_THREADS) {
    const uint64_t k = s_key[i];
    const uint32_t to = s_out[(uint32_t)(k >> shift) & 0xffu] + i;
    if (to < n) {  // always, unless a look-back gave up
      keys_out[(size_t)seg * n + to] = k;
      vals_out[(size_t)seg * n + to] = s_val[i];
    }
  }
}

void radix_sort_pairs_u64(const Scratch& w, uint64_t* keys, uint32_t* vals, uint64_t* keys_tmp, uint32_t* vals_tmp,
                          uint32_t n, uint32_t segs, uint32_t* err) {
  if (n <= 1 || segs == 0) return;
  const uint32_t ntiles = (n + SORT_TILE - 1) / SORT_TILE;
  const bool wide = n >= (1u << 30);
  const size_t words = (size_t)segs * ntiles * RADIX;  // look-back words of one pass
  const size_t head = (size_t)segs * SORT_PASSES * (RADIX + 1) * 4;
  const size_t head8 = (head + 7) / 8;
  TmpBuf<unsigned long long> space(w, head8 + (words * SORT_PASSES * (wide ? 8 : 4) + 7) / 8);
  check(cudaMemsetAsync(space.p, 0, space.bytes(), w.s), "memset");
  uint32_t* hist = reinterpret_cast<uint32_t*>(space.p);
  uint32_t* tickets = hist + (size_t)segs * SORT_PASSES * RADIX;  // [pass][seg]
  const unsigned hgrid = (unsigned)std::min<uint32_t>((n + 4 * SORT_THREADS - 1) / (4 * SORT_THREADS),
                                                      (uint32_t)multiprocessors() * 4u);
  k_sort_hist<<<dim3(hgrid, segs), SORT_THREADS, 0, w.s>>>(keys, n, hist);
  uint64_t* kin = keys;
  uint32_t* vin = vals;
  uint64_t* kout = keys_tmp;
  uint32_t* vout = vals_tmp;
  const dim3 grid(ntiles, segs);
  for (int p = 0; p < SORT_PASSES; p++) {  // an even number of passes: the result ends in keys, vals
    if (wide)
      k_sort_pass<unsigned long long><<<grid, SORT_THREADS, 0, w.s>>>(kin, vin, n, p, ntiles, hist,
                                                                      space.p + head8 + p * words,
                                                                      tickets + p * segs, kout, vout, err);
    else
      k_sort_pass<uint32_t><<<grid, SORT_THREADS, 0, w.s>>>(kin, vin, n, p, ntiles, hist,
                                                            reinterpret_cast<uint32_t*>(space.p + head8) + p * words,
                                                            tickets + p * segs, kout, vout, err);
    std::swap(kin, kout);
    std::swap(vin, vout);
  }
  check(cudaGetLastError(), "radix sort");
}

// ---- levels of a binary tree ------------------------------------------------
// order[b, e) lists the nodes of one level (any order within it); the
// children of its inner nodes, in that order, form the next level.
__global__ void k_level_flags(const int32_t* __restrict__ nodes5, const uint32_t* __restrict__ order, uint32_t b,
                              uint32_t e, uint32_t* __restrict__ flag) {
  const uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
  if (b + k >= e) return;
  flag[k] = nodes5[5 * (size_t)order[b + k] + 1] <= -1 ? 1u : 0u;
}
__global__ void k_level_children(const int32_t* __restrict__ nodes5, uint32_t* __restrict__ order, uint32_t b,
                                 uint32_t e, const uint32_t* __restrict__ rank, uint32_t n_nodes, uint32_t* err) {
  const uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
  if (b + k >= e) return;
  const uint32_t node = order[b + k];
  const int32_t* nd = nodes5 + 5 * (size_t)node;
  if (nd[1] > -1) return;
  const int32_t l = nd[0];
  if (l <= (int32_t)node || (uint32_t)l + 1 >= n_nodes) {  // children must come after their parent
    atomicOr(err, 1u);
    return;
  }
  order[e + 2 * rank[k]] = (uint32_t)l;
  order[e + 2 * rank[k] + 1] = (uint32_t)l + 1;
}

int tree_levels(const Scratch& w, const int32_t* nodes5, uint32_t n_nodes, TmpBuf<uint32_t>& order,
                std::vector<uint32_t>& level) {
  const cudaStream_t s = w.s;
  order.alloc(std::max<uint32_t>(n_nodes, 1u));
  check(cudaMemsetAsync(order.p, 0, 4, s), "memset");  // the root
  // tot: inner nodes of the level, a look-back's errors, the tree's errors
  TmpBuf<uint32_t> flag(w, std::max<uint32_t>(n_nodes, 1u)), tot(w, 3);
  check(cudaMemsetAsync(tot.p, 0, 12, s), "memset");
  level.assign(1, 0u);
  uint32_t b = 0, e = n_nodes ? 1u : 0u;
  uint32_t c[2] = {0, 0};
  while (b < e) {
    level.push_back(e);
    const unsigned blocks = (e - b + 127) / 128;
    k_level_flags<<<blocks, 128, 0, s>>>(nodes5, order.p, b, e, flag.p);
    scan_exclusive_u32(w, flag.p, flag.p, e - b, tot.p, tot.p + 1);
    check(cudaMemcpyAsync(c, tot.p, 8, cudaMemcpyDeviceToHost, s), "D2H");
    check(cudaStreamSynchronize(s), "sync");
    check_lookback(c[1], "tree levels");  // before the ranks place anything
    const uint64_t next_end = (uint64_t)e + 2ull * c[0];
    if (next_end > n_nodes) return 1;
    k_level_children<<<blocks, 128, 0, s>>>(nodes5, order.p, b, e, flag.p, n_nodes, tot.p + 2);
    b = e;
    e = (uint32_t)next_end;
  }
  uint32_t herr = 0;
  check(cudaMemcpyAsync(&herr, tot.p + 2, 4, cudaMemcpyDeviceToHost, s), "D2H");
  check(cudaStreamSynchronize(s), "sync");
  return (e != n_nodes || herr) ? 1 : 0;
}

}  // namespace pk
