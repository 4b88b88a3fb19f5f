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
  bool first = true;
  for (Index base = static_cast<Index>(blockIdx.x) * kStoreThreads * kStoreUnroll + threadIdx.x;
       base < total_vecs; base += step) {
    const char* src[kStoreUnroll];
    Index vec[kStoreUnroll];
    int tok[kStoreUnroll], slot[kStoreUnroll];
    unsigned is_v = 0;                                  // a bit per vector
#pragma unroll
    for (int u = 0; u < kStoreUnroll; ++u) {
      const Index idx = base + u * kStoreThreads;
      tok[u] = -1;
      if (idx < total_vecs) {
        const Index row = idx / row_vecs;               // (token, K|V) pair
        vec[u] = idx - row * row_vecs;
        tok[u] = static_cast<int>(row >> 1);
        is_v |= static_cast<unsigned>(row & 1) << u;
        src[u] = (row & 1 ? value + tok[u] * value_stride_b : key + tok[u] * key_stride_b) + static_cast<long long>(vec[u]) * 16;
        if (first) {
          const int hint = (threadIdx.x & 7) == 0 ? ld_cg_s32(slot_mapping + tok[u]) : -1;
          if (hint >= 0 && hint < n_slots) prefetch_l2(src[u]);
        }
      }
    }
    // Everything is read behind the wait, so the kernel in front may write any of it.  Ahead of it the first pass finds its
    // places and, going by what the slots are then, has them and its rows on their way into L2.  Loads of K and V must not be left to
    // the compiler: through the read-only path it had them ahead of the wait, as the times showed (first figures below).
    // Us per launch in a graph of stores, 8 kv heads, __ldg | slots ahead of the wait | this form: 256 tokens 1.08 | 1.34 | 1.50,
    // 4096 4.0 | 4.4 | 5.3, 16384 20.1 | 20.9 | 21.2, 140000 185 | 186.7 | 185.5 (everything behind the wait and a 64-bit division: 2.33,
    // 5.45, 21.9, 184.8); an eager layer of 256 sequences of 100 .. 2048 tokens, store and decode, 160.3 | 163.1 | 161.6.
    if (first) asm volatile("griddepcontrol.wait;" ::: "memory");
    first = false;
#pragma unroll
    for (int u = 0; u < kStoreUnroll; ++u) slot[u] = tok[u] >= 0 ? ld_s32(slot_mapping + tok[u]) : -1;
    uint4 data[kStoreUnroll];
#pragma unroll
    for (int u = 0; u < kStoreUnroll; ++u)
      if (slot[u] >= 0 && slot[u] < n_slots) data[u] = ld_row16(src[u]);
#pragma unroll
    for (int u = 0; u < kStoreUnroll; ++u)
      if (slot[u] >= 0 && slot[u] < n_slots)
        *reinterpret_cast<uint4*>((is_v >> u & 1 ? v_cache : k_cache) + slot[u] * row_bytes + static_cast<long long>(vec[u]) * 16) = data[u];
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
