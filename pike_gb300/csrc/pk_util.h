// pk_util.h -- small host helpers: owned device buffers, device-wide scans and sorts.
#pragma once
#include <cuda_runtime.h>
#include <cstddef>
#include <cstdint>
#include <stdexcept>
#include <string>
#include <utility>
#include <vector>

namespace pk {

struct CudaError : std::runtime_error {
  explicit CudaError(const std::string& s) : std::runtime_error(s) {}
};

inline void check(cudaError_t e, const char* what) {
  if (e != cudaSuccess) throw CudaError(std::string(what) + ": " + cudaGetErrorString(e));
}

// Makes the pages of a caller's pageable buffer resident, its contents kept, before the GPU
// copies into it: where the GPU reaches pageable memory through the host's page
// tables, the copy engine faulted fresh pages in one by one (49 MB in 16 buffers:
// 30-52 ms, touched by this thread first 17 ms, by eight threads 20 ms).
void touch_pages(void* p, size_t bytes);

// cudaMalloc.  When memory is short, what the scratch pools of this device's
// contexts hold between builds is given back first; throws when that is not
// enough, and leaves no CUDA error behind for the next call to find.
void* device_malloc(size_t bytes);

// Owned device allocation (device_malloc / cudaFree).  alloc() keeps the block it
// has when the new size fits it and fills at least half of it: a scene that is
// rebuilt at about its old size then costs no cudaMalloc and no cudaFree (which
// waits for the whole device).
template <class T>
struct DevBuf {
  T* p = nullptr;
  size_t n = 0;
  size_t cap = 0;  // bytes allocated
  DevBuf() = default;
  explicit DevBuf(size_t count) { alloc(count); }
  DevBuf(const DevBuf&) = delete;
  DevBuf& operator=(const DevBuf&) = delete;
  DevBuf(DevBuf&& o) noexcept : p(o.p), n(o.n), cap(o.cap) { o.p = nullptr; o.n = o.cap = 0; }
  DevBuf& operator=(DevBuf&& o) noexcept {
    if (this != &o) { release(); p = o.p; n = o.n; cap = o.cap; o.p = nullptr; o.n = o.cap = 0; }
    return *this;
  }
  ~DevBuf() { release(); }
  void alloc(size_t count) {
    const size_t need = count * sizeof(T);
    if (count && p && need <= cap && need >= cap / 2) {
      n = count;
      return;
    }
    release();
    if (count) {
      p = static_cast<T*>(device_malloc(need));
      n = count;
      cap = need;
    }
  }
  void release() {
    if (p) cudaFree(p);
    p = nullptr;
    n = cap = 0;
  }
  size_t bytes() const { return n * sizeof(T); }
};

// What a builder runs on: a stream, and a memory pool for its temporaries.
// The pool belongs to one context (pk_create), keeps at most SCRATCH_KEEP
// bytes between builds and goes with the context.  Allocation and release are
// stream-ordered: no host wait, no device-wide cudaFree.
constexpr uint64_t SCRATCH_KEEP = 512ull << 20;
struct Scratch {
  cudaStream_t s = nullptr;
  cudaMemPool_t pool = nullptr;
};
cudaMemPool_t create_scratch_pool(int device);
void destroy_scratch_pool(cudaMemPool_t pool);
void* scratch_malloc(const Scratch& w, size_t bytes);  // stream-ordered; short memory as in device_malloc

// A temporary of a builder; freed on the stream when it goes out of scope.
template <class T>
struct TmpBuf {
  Scratch w;
  T* p = nullptr;
  size_t n = 0;
  TmpBuf(const Scratch& scratch, size_t count) : w(scratch) { alloc(count); }
  explicit TmpBuf(const Scratch& scratch) : w(scratch) {}
  TmpBuf(const TmpBuf&) = delete;
  TmpBuf& operator=(const TmpBuf&) = delete;
  ~TmpBuf() { release(); }
  void alloc(size_t count) {
    release();
    if (!count) return;
    p = static_cast<T*>(scratch_malloc(w, count * sizeof(T)));
    n = count;
  }
  void release() {
    if (p) cudaFreeAsync(p, w.s);
    p = nullptr;
    n = 0;
  }
  void swap(TmpBuf& o) {
    std::swap(p, o.p);
    std::swap(n, o.n);
  }
  size_t bytes() const { return n * sizeof(T); }
};

// Exclusive prefix sum of n u32 values (in may alias out).  If total is not
// null it receives the sum (device pointer).  Counts must stay below 2^31.
// Enqueues and returns; a look-back that timed out sets ERR_LOOKBACK in *err
// (device).  The prefixes are then too small, each by some amount, and a sort's
// arrays hold words that were never written: whatever uses either as an index
// comes after a check of *err, on the host (check_lookback) or in a kernel.
void scan_exclusive_u32(const Scratch& w, const uint32_t* in, uint32_t* out, uint32_t n, uint32_t* total,
                        uint32_t* err);

// Throws when the look-back bit of `err` is set.
void check_lookback(uint32_t err, const char* what);

// Exclusive prefix sum of n u64 values (in may alias out); enqueues and returns.
void scan_exclusive_u64(const Scratch& w, const unsigned long long* in, unsigned long long* out, size_t n);

// Exclusive prefix sum of n doubles that are not negative (in may alias out);
// enqueues and returns.  For n < 2^33 (three levels) every prefix is the result of
// at most 96 additions, so it lies within 96 * 2^-53 (relative) of the exact sum.
void scan_exclusive_f64(const Scratch& w, const double* in, double* out, size_t n);

// Stable LSD radix sort of `segs` arrays of n (64-bit key, 32-bit value) pairs
// each, array k at keys + k * n and vals + k * n, ascending, in place using
// scratch arrays of the same size.  Enqueues and returns; errors as above.
void radix_sort_pairs_u64(const Scratch& w, uint64_t* keys, uint32_t* vals, uint64_t* keys_tmp, uint32_t* vals_tmp,
                          uint32_t n, uint32_t segs, uint32_t* err);

// The levels of a binary tree (nodes5: 5 words per node, word 0 the left
// child (the right child follows it), word 1 > -1 for a leaf; children after
// their parents): the nodes of depth d are order[level[d], level[d + 1]).
// Returns non-zero when the tree is malformed (a child not after its parent,
// or a node not reached exactly once).
int tree_levels(const Scratch& w, const int32_t* nodes5, uint32_t n_nodes, TmpBuf<uint32_t>& order,
                std::vector<uint32_t>& level);

// EnvironmentGenerator tables on the GPU (pk_env.cu).
int build_env_tables_gpu(const Scratch& scratch, const uchar4* rgbe, uint32_t w, uint32_t h, DevBuf<int2>& bins_out,
                         uint32_t& nb_out, DevBuf<int2>& coords_out, DevBuf<float>& pdf_out, std::string& why);
// The same tables for an FP32 RGB map (w x h x 3): radiance = luma of the
// stored values in double (the differentiable renderer's sampling tables).
int build_env_tables_gpu_f32(const Scratch& scratch, const float* rgb, uint32_t w, uint32_t h, DevBuf<int2>& bins_out,
                             uint32_t& nb_out, DevBuf<int2>& coords_out, DevBuf<float>& pdf_out, std::string& why);

// PK_ENV_ALIAS's alias table for a w x h RGBE image on the device (pk_env.cu):
// {keep threshold, alias} per texel and the pdf texture of the table's exact
// selection probabilities.  Returns non-zero with a reason on failure.
int build_env_alias_gpu(const Scratch& scratch, const uchar4* rgbe, uint32_t w, uint32_t h, DevBuf<uint2>& table_out,
                        DevBuf<float>& pdf_out, std::string& why);

}  // namespace pk
