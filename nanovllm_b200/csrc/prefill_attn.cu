// C-ABI entry points of prefill attention: argument checks, tensor maps, kernel selection.
#include "../../include/b200_attn.h"
#include "kernels.cuh"

#include <cmath>

namespace b200 {

// Which kernel a batch goes to, from what the host knows of it.  A tcgen05 item is a chain of some 8 us however short the
// prompt; the mma.sync kernel with 64-row CTAs is through a short one in 4 to 6, but pays 1.05 us per 64 keys where
// tcgen05 pays half, and its CTAs come in waves of one per SM.  The lines below are fits, in us, to both kernels'
// times over 29 batches of 1 .. 128 prompts of 1 .. 1000 tokens at 1 .. 8 kv heads (within 20 % of all of them; one prompt
// of 137 tokens 12.8 -> 6.0 us, 16 of up to 100: 14.9 -> 10.9, 2 of 1000: stays at 27 instead of 43).
// Where the tcgen05 launch has few items its length is that of one item's chain, 0.9 us per 64 keys.  With the keys shared
// between the halves (`split`) it is half of that, for twice as many items of half the rows, each with the same start and
// end to pay: worth it up to some 1.2 whole items per SM, by the same kind of fit over 85 batches of 1 .. 64 prompts of
// 50 .. 8192 tokens (one of 2048 at 8/4 heads 36.8 -> 24.2 us, of 8192 at 4/2 heads 124 -> 67, 4 of 200 .. 2000 at
// 16/8 heads, 2.1 items per SM, stay at 42 instead of 44).
struct PrefillChoice {
  bool tc;           // tcgen05 (where it takes the head ratio)
  bool split;        // tcgen05: items of one tile of rows, the keys shared between the halves
  bool small_ctas;   // mma.sync: 64 rows per CTA, not 128
};
static PrefillChoice prefill_choice(int total_q, int batch, int Hkv, int G, int max_k) {
  PrefillChoice c = {true, false, false};
  if (G > 64) return c;   // (no room for a group in 64 rows)
  const double sms = sm_count() > 0 ? sm_count() : 1;
  const double tiles = (max_k + 63) / 64;                                                          // of 64 keys
  const double small_waves = (static_cast<double>(total_q) / (64 / G) + batch) * Hkv / sms;        // CTAs per SM
  const double tc_items = (static_cast<double>(total_q) / (256 / G) + batch) * Hkv / sms;          // items per SM
  const double t_small = 1.5 + fmax(2 + 1.05 * tiles, small_waves * (3 + 0.6 * tiles));
  const double split_items = (static_cast<double>(total_q) / (128 / G) + batch) * Hkv / sms;
  const double t_full = fmax(8 + 0.9 * tiles, 4 + tc_items * (5.2 + 0.5 * tiles));
  const double t_split = fmax(8.6 + 0.47 * tiles, 4 + split_items * (5.2 + 0.235 * tiles));
  c.split = t_split < t_full;
  c.tc = t_small > fmin(t_split, t_full);
  c.small_ctas = t_small <= t_full || small_waves <= 2;   // (!c.tc, and the head ratios that tcgen05 does not take)
  return c;
}

struct StoreArgs {
  const int* slots;
  void *k_cache, *v_cache;
  long long n_slots;
};

// `store` != nullptr (dense K/V only): k and v also go to the cache rows store->slots names.
static int prefill(const void* q, int64_t q_row_stride, const void* k, const void* v,
                                 int64_t k_row_stride, int64_t v_row_stride, int64_t total_k, const void* k_cache,
                                 const void* v_cache, int64_t num_blocks, int32_t block_size,
                                 const int32_t* block_tables, int64_t bt_row_stride, int32_t bt_cols,
                                 const int32_t* cu_seqlens_q, const int32_t* cu_seqlens_k, int32_t batch,
                                 int32_t total_q, int32_t max_seqlen_q, int32_t max_seqlen_k, void* out,
                                 int32_t num_heads, int32_t num_kv_heads, int32_t head_dim, float scale,
                                 int32_t kernel_variant, void* stream, const StoreArgs* store) {
  if (batch < 0 || total_q < 0) return set_error(kErrBadShape, "prefill_attn: negative batch or total_q");
  if (batch == 0 || total_q == 0) return kOk;
  if (!q || !out || !cu_seqlens_q || !cu_seqlens_k) return set_error(kErrNullPointer, "prefill_attn: null pointer argument");
  if (head_dim != 128) return set_error(kErrBadShape, "prefill_attn: head_dim must be 128 (got %d)", head_dim);
  if (num_heads <= 0 || num_kv_heads <= 0 || num_heads % num_kv_heads)
    return set_error(kErrBadShape, "prefill_attn: num_heads (%d) must be a positive multiple of num_kv_heads (%d)",
                     num_heads, num_kv_heads);
  const int G = num_heads / num_kv_heads;
  if (G > 128) return set_error(kErrBadShape, "prefill_attn: at most 128 query heads per kv head");
  if (q_row_stride < static_cast<long long>(num_heads) * 128 || q_row_stride % 8)
    return set_error(kErrMisaligned, "prefill_attn: q_row_stride must be >= H*128 and a multiple of 8 elements");
  if ((reinterpret_cast<uintptr_t>(q) | reinterpret_cast<uintptr_t>(out)) & 15)
    return set_error(kErrMisaligned, "prefill_attn: q and out must be 16-byte aligned");
  if (max_seqlen_q <= 0 || max_seqlen_k <= 0)
    return set_error(kErrBadShape, "prefill_attn: max_seqlen_q/k must be positive");

  if (kernel_variant < 0 || kernel_variant > 2)
    return set_error(kErrBadShape, "prefill_attn: kernel_variant must be 0 .. 2");
  const bool tc_ok = 128 % G == 0;
  if (kernel_variant == 2 && !tc_ok)
    return set_error(kErrBadShape, "prefill_attn: the tcgen05 kernel needs 128 %% (num_heads / num_kv_heads) == 0 (got %d)", G);
  const PrefillChoice choice = prefill_choice(total_q, batch, num_kv_heads, G, max_seqlen_k);
  const bool use_tc = kernel_variant == 2 || (kernel_variant == 0 && tc_ok && choice.tc);
  const uint32_t kv_box = use_tc ? 128 : 64;
  CUtensorMap map_k, map_v;
  const bool paged = block_tables != nullptr;
  int rc;
  if (paged) {
    if (!k_cache || !v_cache) return set_error(kErrNullPointer, "prefill_attn: block_tables given without caches");
    if (block_size <= 0 || block_size % 256)
      return set_error(kErrBadShape, "prefill_attn: block_size must be a positive multiple of 256 (got %d)", block_size);
    if (num_blocks <= 0 || num_blocks * block_size >= (1LL << 31))
      return set_error(kErrBadShape, "prefill_attn: num_blocks * block_size must be in (0, 2^31)");
    if (bt_cols <= 0 || bt_row_stride < bt_cols)
      return set_error(kErrBadShape, "prefill_attn: bad block table geometry");
    if ((reinterpret_cast<uintptr_t>(k_cache) | reinterpret_cast<uintptr_t>(v_cache)) & 15)
      return set_error(kErrMisaligned, "prefill_attn: caches must be 16-byte aligned");
    const uint64_t rows = static_cast<uint64_t>(num_blocks) * block_size;
    rc = make_tokens_heads_map(&map_k, k_cache, rows, num_kv_heads, static_cast<uint64_t>(num_kv_heads) * 128, kv_box);
    if (rc) return rc;
    rc = make_tokens_heads_map(&map_v, v_cache, rows, num_kv_heads, static_cast<uint64_t>(num_kv_heads) * 128, kv_box);
    if (rc) return rc;
  } else {
    if (!k || !v) return set_error(kErrNullPointer, "prefill_attn: dense k/v missing");
    if (total_k <= 0 || total_k >= (1LL << 31)) return set_error(kErrBadShape, "prefill_attn: total_k out of range");
    if (k_row_stride < static_cast<long long>(num_kv_heads) * 128 || v_row_stride < static_cast<long long>(num_kv_heads) * 128 ||
        k_row_stride % 8 || v_row_stride % 8)
      return set_error(kErrMisaligned, "prefill_attn: k/v row strides must be >= Hkv*128 and multiples of 8 elements");
    if ((reinterpret_cast<uintptr_t>(k) | reinterpret_cast<uintptr_t>(v)) & 15)
      return set_error(kErrMisaligned, "prefill_attn: k and v must be 16-byte aligned");
    rc = make_tokens_heads_map(&map_k, k, static_cast<uint64_t>(total_k), num_kv_heads, static_cast<uint64_t>(k_row_stride), kv_box);
    if (rc) return rc;
    rc = make_tokens_heads_map(&map_v, v, static_cast<uint64_t>(total_k), num_kv_heads, static_cast<uint64_t>(v_row_stride), kv_box);
    if (rc) return rc;
  }

  PrefillParams p;
  p.q = static_cast<const __nv_bfloat16*>(q);
  p.q_row_stride = q_row_stride;
  p.out = static_cast<__nv_bfloat16*>(out);
  p.cu_q = cu_seqlens_q;
  p.cu_k = cu_seqlens_k;
  p.block_tables = block_tables;
  p.bt_row_stride = bt_row_stride;
  p.bt_cols = bt_cols;
  p.block_size = paged ? block_size : 256;
  p.num_blocks = num_blocks;
  p.batch = batch;
  p.H = num_heads;
  p.Hkv = num_kv_heads;
  p.G = G;
  p.QT = 128 / G;
  p.n_slots = total_q / p.QT + batch;
  p.scale_log2 = scale * 1.4426950408889634f;
  p.total_q = total_q;
  p.max_seqlen_q = max_seqlen_q;
  p.max_seqlen_k = max_seqlen_k;
  p.out_tma = 0;
  p.st_slots = nullptr;
  if (store) {
    p.st_k = static_cast<const char*>(k);
    p.st_v = static_cast<const char*>(v);
    p.st_k_cache = static_cast<char*>(store->k_cache);
    p.st_v_cache = static_cast<char*>(store->v_cache);
    p.st_slots = store->slots;
    p.st_k_stride = k_row_stride * 2;
    p.st_v_stride = v_row_stride * 2;
    p.st_n_slots = store->n_slots;
    p.st_tokens = static_cast<int>(total_k);
  }
  if (use_tc) {
    CUtensorMap map_q;
    rc = make_tokens_heads_map(&map_q, q, static_cast<uint64_t>(total_q), num_heads, static_cast<uint64_t>(q_row_stride),
                               static_cast<uint32_t>(p.QT), static_cast<uint32_t>(G));
    if (rc) return rc;
    // output map of the persistent kernel: boxes of 32 tile rows = (32 / G tokens) x (G heads) x 32 dims
    CUtensorMap map_o = map_q;
    p.out_tma = 32 % G == 0;
    if (p.out_tma) {
      rc = make_tokens_heads_map_cols32(&map_o, out, static_cast<uint64_t>(total_q), num_heads,
                                        static_cast<uint64_t>(num_heads) * 128, static_cast<uint32_t>(32 / G),
                                        static_cast<uint32_t>(G));
      if (rc) return rc;
    }
    CUtensorMap map_kc = map_k, map_vc = map_v;
    if (p.st_slots) {
      rc = make_tokens_heads_map(&map_kc, store->k_cache, static_cast<uint64_t>(store->n_slots), num_kv_heads,
                                 static_cast<uint64_t>(num_kv_heads) * 128, 32);
      if (rc) return rc;
      rc = make_tokens_heads_map(&map_vc, store->v_cache, static_cast<uint64_t>(store->n_slots), num_kv_heads,
                                 static_cast<uint64_t>(num_kv_heads) * 128, 32);
      if (rc) return rc;
    }
    return launch_prefill_tc2(p, choice.split, map_q, map_k, map_v, map_o, map_kc, map_vc, static_cast<cudaStream_t>(stream));
  }
  return launch_prefill_mma(p, map_k, map_v, choice.small_ctas, static_cast<cudaStream_t>(stream));
}

}  // namespace b200

extern "C" int b200_prefill_attn(const void* q, int64_t q_row_stride, const void* k, const void* v,
                                 int64_t k_row_stride, int64_t v_row_stride, int64_t total_k, const void* k_cache,
                                 const void* v_cache, int64_t num_blocks, int32_t block_size,
                                 const int32_t* block_tables, int64_t bt_row_stride, int32_t bt_cols,
                                 const int32_t* cu_seqlens_q, const int32_t* cu_seqlens_k, int32_t batch,
                                 int32_t total_q, int32_t max_seqlen_q, int32_t max_seqlen_k, void* out,
                                 int32_t num_heads, int32_t num_kv_heads, int32_t head_dim, float scale,
                                 int32_t kernel_variant, void* stream) {
  return b200::prefill(q, q_row_stride, k, v, k_row_stride, v_row_stride, total_k, k_cache, v_cache, num_blocks, block_size,
                       block_tables, bt_row_stride, bt_cols, cu_seqlens_q, cu_seqlens_k, batch, total_q, max_seqlen_q,
                       max_seqlen_k, out, num_heads, num_kv_heads, head_dim, scale, kernel_variant, stream, nullptr);
}

extern "C" int b200_store_prefill_attn(const void* q, int64_t q_row_stride, const void* k, const void* v,
                                       int64_t k_row_stride, int64_t v_row_stride, int64_t total_k, void* k_cache,
                                       void* v_cache, const int32_t* slot_mapping, int64_t n_slots,
                                       const int32_t* cu_seqlens_q, const int32_t* cu_seqlens_k, int32_t batch,
                                       int32_t total_q, int32_t max_seqlen_q, int32_t max_seqlen_k, void* out,
                                       int32_t num_heads, int32_t num_kv_heads, int32_t head_dim, float scale,
                                       void* stream) {
  using namespace b200;
  if (!k_cache || !v_cache || !slot_mapping)
    return set_error(kErrNullPointer, "store_prefill_attn: null cache or slot_mapping");
  if (n_slots < 0 || n_slots >= (1LL << 31)) return set_error(kErrBadShape, "store_prefill_attn: n_slots must be in [0, 2^31)");
  if ((reinterpret_cast<uintptr_t>(k_cache) | reinterpret_cast<uintptr_t>(v_cache)) & 15)
    return set_error(kErrMisaligned, "store_prefill_attn: caches must be 16-byte aligned");
  if (batch == 0 || total_q == 0)     // nothing to attend: the store alone
    return b200_store_kvcache(k, v, k_row_stride, v_row_stride, k_cache, v_cache, slot_mapping, static_cast<int32_t>(total_k),
                              num_kv_heads * head_dim, 2, n_slots, stream);
  const StoreArgs store = {slot_mapping, k_cache, v_cache, n_slots};
  return prefill(q, q_row_stride, k, v, k_row_stride, v_row_stride, total_k, nullptr, nullptr, 0, 0, nullptr, 0, 0, cu_seqlens_q,
                 cu_seqlens_k, batch, total_q, max_seqlen_q, max_seqlen_k, out, num_heads, num_kv_heads, head_dim, scale, 0, stream,
                 &store);
}
