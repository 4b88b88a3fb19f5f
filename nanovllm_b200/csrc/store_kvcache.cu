// store_kvcache: scatter of the step's new K and V rows into the paged cache through
// slot_mapping.  Replaces the reference's Triton kernel (nanovllm/layers/attention.py:10-40).
//
// HBM-bound byte copy: every thread moves 16-byte vectors, consecutive threads take consecutive
// vectors of one row (fully coalesced 128-byte lines on both sides), four independent vectors
// are in flight per thread, offsets are 64-bit, and the grid is a multiple of the SM count.
#include <atomic>

#include "../../include/b200_attn.h"
#include "common.cuh"

namespace b200 {
extern std::atomic<long long> g_launches;

constexpr int kStoreThreads = 256;
constexpr int kStoreUnroll = 4;

// Index: unsigned while twice the number of vectors fits in it (the division by the row's length is an eighth of the 64-bit
// one's instructions), else long long.
template <typename Index>
__global__ void __launch_bounds__(kStoreThreads)
store_kvcache_kernel(const char* key, const char* value, long long key_stride_b,
                     long long value_stride_b, char* k_cache, char* v_cache, const int* slot_mapping, Index total_vecs, Index row_vecs, long long n_slots) {
  // Let a dependent launch (the decode kernel that follows in the stream) start its prologue
  // now; it still waits for this grid to finish before it reads the cache.
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  const long long row_bytes = static_cast<long long>(row_vecs) * 16;
  const Index step = static_cast<Index>(gridDim.x) * kStoreThreads * kStoreUnroll;
  for (Index base = static_cast<Index>(blockIdx.x) * kStoreThreads * kStoreUnroll + threadIdx.x;
       base < total_vecs; base += step) {
    const char* src[kStoreUnroll];
    char* dst[kStoreUnroll];
#pragma unroll
    for (int u = 0; u < kStoreUnroll; ++u) {
      const Index idx = base + u * kStoreThreads;
      dst[u] = nullptr;
      if (idx < total_vecs) {
        const Index row = idx / row_vecs;               // (token, K|V) pair
        const long long vec = idx - row * row_vecs;
        const long long tok = row >> 1;
        const bool is_v = (row & 1) != 0;
        const long long slot = slot_mapping[tok];
        if (slot >= 0 && slot < n_slots) {
          src[u] = (is_v ? value + tok * value_stride_b : key + tok * key_stride_b) + vec * 16;
          dst[u] = (is_v ? v_cache : k_cache) + slot * row_bytes + vec * 16;
        }
      }
    }
    // The slots are not written by any kernel that lets this one start early, so the first pass has its places by the time
    // the kernel in front ends; K, V and the cache are touched behind the wait (which costs the later passes nothing).  Their loads
    // must not be left to the compiler: through the read-only path it had them ahead of the wait, as the times showed (256 tokens
    // 1.08 us per launch in a graph of stores, an eager layer of 256 sequences of 100 .. 2048 tokens, store and decode, 160.3 us).
    // With the 32-bit division, per launch in a graph of stores, 8 kv heads: 256 tokens 2.33 -> 1.34 us, 4096 5.45 -> 4.4,
    // 16384 21.9 -> 20.9, 140000 184.8 -> 186.7; the eager layer 163.1.
    asm volatile("griddepcontrol.wait;" ::: "memory");
    uint4 data[kStoreUnroll];
#pragma unroll
    for (int u = 0; u < kStoreUnroll; ++u)
      if (dst[u]) data[u] = ld_row16(src[u]);
#pragma unroll
    for (int u = 0; u < kStoreUnroll; ++u)
      if (dst[u]) *reinterpret_cast<uint4*>(dst[u]) = data[u];
  }
}

}  // namespace b200

extern "C" int b200_store_kvcache(const void* key, const void* value, int64_t key_row_stride,
                                  int64_t value_row_stride, void* k_cache, void* v_cache,
                                  const int32_t* slot_mapping, int32_t n_tokens, int32_t row_elems,
                                  int32_t elem_bytes, int64_t n_slots, void* stream) {
  using namespace b200;
  if (n_tokens < 0 || row_elems <= 0 || elem_bytes <= 0 || n_slots < 0 || key_row_stride < 0 || value_row_stride < 0)
    return set_error(kErrBadShape, "store_kvcache: negative or zero size (n_tokens=%d row_elems=%d elem_bytes=%d)",
                     n_tokens, row_elems, elem_bytes);
  if (n_tokens == 0) return kOk;
  if (!key || !value || !k_cache || !v_cache || !slot_mapping)
    return set_error(kErrNullPointer, "store_kvcache: null pointer argument");
  const long long row_bytes = static_cast<long long>(row_elems) * elem_bytes;
  const long long ks = key_row_stride * elem_bytes, vs = value_row_stride * elem_bytes;
  if (row_bytes % 16 || ks % 16 || vs % 16)
    return set_error(kErrMisaligned, "store_kvcache: row bytes (%lld) and row strides (%lld, %lld bytes) must be multiples of 16",
                     row_bytes, ks, vs);
  if ((reinterpret_cast<uintptr_t>(key) | reinterpret_cast<uintptr_t>(value) | reinterpret_cast<uintptr_t>(k_cache) |
       reinterpret_cast<uintptr_t>(v_cache)) & 15)
    return set_error(kErrMisaligned, "store_kvcache: pointers must be 16-byte aligned");
  if (ks < row_bytes || vs < row_bytes)
    return set_error(kErrBadShape, "store_kvcache: row stride smaller than the row");
  const int row_vecs = static_cast<int>(row_bytes / 16);
  const long long total = 2LL * n_tokens * row_vecs;
  const long long per_block = static_cast<long long>(kStoreThreads) * kStoreUnroll;
  long long blocks = (total + per_block - 1) / per_block;
  const int sms = sm_count();
  if (sms <= 0) return set_error(kErrNoDriver, "store_kvcache: no CUDA device");
  const long long cap = static_cast<long long>(sms) * 16;
  if (blocks > cap) blocks = cap;
  auto launch = [&](auto kernel, auto total_vecs, auto vecs) {
    return launch_early(kernel, static_cast<unsigned>(blocks), kStoreThreads, 0, static_cast<cudaStream_t>(stream),
                        static_cast<const char*>(key), static_cast<const char*>(value), ks, vs, static_cast<char*>(k_cache),
                        static_cast<char*>(v_cache), slot_mapping, total_vecs, vecs, static_cast<long long>(n_slots));
  };
  const cudaError_t le = total < (1LL << 31) ? launch(store_kvcache_kernel<unsigned>, static_cast<unsigned>(total), static_cast<unsigned>(row_vecs))
                                             : launch(store_kvcache_kernel<long long>, total, static_cast<long long>(row_vecs));
  g_launches.fetch_add(1);
  return check_cuda(le != cudaSuccess ? le : cudaGetLastError(), "store_kvcache launch");
}
