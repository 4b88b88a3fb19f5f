// Producer side of the attention layer in one launch: per-head RMSNorm of q and k, rotary
// embedding, and the store of k and v into the paged cache.  Replaces, for one decoder layer,
//   q_norm / k_norm      nanovllm/layers/layernorm.py:16-26    (called at nanovllm/models/qwen3.py:76-77)
//   rotary_emb           nanovllm/layers/rotary_embedding.py:6-14, 37-48  (called at models/qwen3.py:79)
//   store_kvcache        nanovllm/layers/attention.py:10-40    (called at layers/attention.py:62-63)
// which the reference runs as three compiled element-wise kernels plus one Triton kernel.
//
// A half-warp owns one 128-element head vector at a time (four consecutive heads of a token per pass):
// lane j of 16 holds elements [8j, 8j + 8)
// (16-byte accesses), so the rotary partner (element i +- 64) of every element sits in lane j ^ 8.  q heads and k heads are
// normalised in fp32, cast to bf16, multiplied by the bf16 weight, rotated in fp32 (products and
// sums rounded separately, as the reference's eager arithmetic does) and written out contiguous;
// k is also written to its cache slot.  v heads are copied bit-for-bit from the strided qkv row to
// their cache slot.  Pure streaming: HBM / launch bound, no tensor-core work.
//
// Large batches are bound by latency and issue slots, not yet by the memory: 16384 tokens at 16/8 heads take 58.9 us,
// 5.1 TB/s (71.3 us with a 64-bit division and two dependent trips per pass, scalar squares and fp32 weight products).
// Three CTAs per SM (80 registers) are the best of 2, 3, 4 and 5, four heads per pass the best of 2, 4 and 8.
#include <atomic>

#include <cuda_bf16.h>

#include "../../include/b200_attn.h"
#include "common.cuh"

namespace b200 {
extern std::atomic<long long> g_launches;

struct QkNormRopeParams {
  const __nv_bfloat16* qkv;
  long long qkv_row_stride;            // elements
  const long long* positions;          // (n_tokens) int64
  const __nv_bfloat16* q_weight;       // (128)
  const __nv_bfloat16* k_weight;       // (128)
  const float* cos_sin;                // (max_position, 128): 64 cos then 64 sin
  int max_position;
  bool wide_table;                     // cos_sin lies at a multiple of 32 bytes
  float eps;
  __nv_bfloat16* q_out;                // (n_tokens, H, 128)
  __nv_bfloat16* k_out;                // (n_tokens, Hkv, 128)
  __nv_bfloat16* k_cache;              // flat rows of Hkv * 128 elements, or nullptr
  __nv_bfloat16* v_cache;
  const int* slot_mapping;             // (n_tokens) or nullptr
  long long n_slots;
  int n_tokens, H, Hkv;
};

constexpr int kQkThreads = 256;     // 16 half-warps per CTA
constexpr int kQkCtas = 3;          // CTAs per SM, all resident, in the large form
constexpr int kQkGroup = 4;         // head vectors of one token a half-warp works through per pass (large batches)

__device__ __forceinline__ unsigned long long f32x2_mul(unsigned long long a, unsigned long long b) {
  unsigned long long d;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}

// bf16 pair -> packed fp32 pair (exact)
__device__ __forceinline__ unsigned long long bf16x2_to_f32x2(uint32_t v) {
  return f32x2_pack(__uint_as_float(v << 16), __uint_as_float(v & 0xffff0000u));
}

// What a half-warp needs once per token (not once per head): where the token goes in the cache and this
// lane's eight cos / sin values of its position.
struct QkTokenCtx {
  long long slot;                      // -1: no store
  unsigned long long cosv[4], sinv[4]; // packed pairs; sin carries the sign of this lane's half (-sin for the first)
};

// This lane's part of the table row of a position: eight cos there, eight sin 64 floats on.
__device__ __forceinline__ const float* qk_table_row(const QkNormRopeParams& p, long long pos, int sub) {
  pos = pos < 0 ? 0 : (pos >= p.max_position ? p.max_position - 1 : pos);
  return p.cos_sin + pos * 128 + (sub & 7) * 8;
}

struct QkTableRow {
  float4 c0, c1, s0, s1;
};
__device__ __forceinline__ float4 qk_float4(const uint4& v) {
  return make_float4(__uint_as_float(v.x), __uint_as_float(v.y), __uint_as_float(v.z), __uint_as_float(v.w));
}
__device__ __forceinline__ QkTableRow qk_load_table(const QkNormRopeParams& p, long long pos, int sub) {
  const float* cs = qk_table_row(p, pos, sub);
  QkTableRow t;
  if (p.wide_table) {
    ld_row32(cs, t.c0, t.c1);
    ld_row32(cs + 64, t.s0, t.s1);
  } else {
    t.c0 = qk_float4(ld_row16(cs));
    t.c1 = qk_float4(ld_row16(cs + 4));
    t.s0 = qk_float4(ld_row16(cs + 64));
    t.s1 = qk_float4(ld_row16(cs + 68));
  }
  return t;
}

__device__ __forceinline__ QkTokenCtx qk_token_ctx(const QkNormRopeParams& p, const QkTableRow& t, int slot, int sub) {
  QkTokenCtx c;
  c.slot = slot < p.n_slots ? slot : -1;                 // never write outside the cache
  // first half:  y1 = x1 * cos - x2 * sin      second half:  y2 = x2 * cos + x1 * sin
  // (negating sin is exact, and a + (-t) rounds like a - t)
  const float sg = sub < 8 ? -1.f : 1.f;
  c.cosv[0] = f32x2_pack(t.c0.x, t.c0.y); c.cosv[1] = f32x2_pack(t.c0.z, t.c0.w);
  c.cosv[2] = f32x2_pack(t.c1.x, t.c1.y); c.cosv[3] = f32x2_pack(t.c1.z, t.c1.w);
  c.sinv[0] = f32x2_pack(sg * t.s0.x, sg * t.s0.y); c.sinv[1] = f32x2_pack(sg * t.s0.z, sg * t.s0.w);
  c.sinv[2] = f32x2_pack(sg * t.s1.x, sg * t.s1.y); c.sinv[3] = f32x2_pack(sg * t.s1.z, sg * t.s1.w);
  return c;
}

// One q or k head vector: `raw` holds this lane's 8 elements; `w` the lane's 8 weights as bf16 pairs.
// Every product and every sum is rounded on its own (mul.rn / add.rn, packed two at a time), in the order the
// reference's eager arithmetic takes them.  First half: normalised and weighted, exact bf16 values as packed pairs.
__device__ __forceinline__ void qk_normalise(const uint4& raw, const uint32_t (&w)[4], float eps, unsigned half_mask, uint32_t (&ap)[4]) {
  const uint32_t r[4] = {raw.x, raw.y, raw.z, raw.w};
  unsigned long long x[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) x[i] = bf16x2_to_f32x2(r[i]);
  // mean of squares over the 128 elements, fp32 (the order of this sum is the one thing the reference leaves open)
  float ss, s1;
  f32x2_unpack(f32x2_fma(x[3], x[3], f32x2_fma(x[2], x[2], f32x2_fma(x[1], x[1], f32x2_mul(x[0], x[0])))), ss, s1);
  ss += s1;
#pragma unroll
  for (int o = 8; o > 0; o >>= 1) ss += __shfl_xor_sync(half_mask, ss, o);
  const float rinv = __frsqrt_rn(__fadd_rn(__fmul_rn(ss, 1.f / 128.f), eps));      // (a division by 128 is this product, exactly)
  const unsigned long long rinv2 = f32x2_pack(rinv, rinv);
  // normalise in fp32, round to bf16, scale by the bf16 weight (rounded to bf16 again)
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    float n0, n1;
    f32x2_unpack(f32x2_mul(x[i], rinv2), n0, n1);
    // (the product of two bf16 values is exact in fp32, so the packed bf16 product rounds once, as the reference does)
    const __nv_bfloat162 m = __hmul2(__floats2bfloat162_rn(n0, n1), *reinterpret_cast<const __nv_bfloat162*>(&w[i]));
    ap[i] = *reinterpret_cast<const uint32_t*>(&m);
  }
}
// Second half: rotated.  (The packed pairs travel to the partner lane, 4 shuffles instead of 8.)
__device__ __forceinline__ uint4 qk_rotate(const uint32_t (&ap)[4], const QkTokenCtx& c, unsigned half_mask) {
  uint32_t y[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const uint32_t bp = __shfl_xor_sync(half_mask, ap[i], 8);       // the elements 64 away
    float y0, y1;
    f32x2_unpack(f32x2_add(f32x2_mul(bf16x2_to_f32x2(ap[i]), c.cosv[i]), f32x2_mul(bf16x2_to_f32x2(bp), c.sinv[i])), y0, y1);
    y[i] = pack_bf16(y0, y1);
  }
  return make_uint4(y[0], y[1], y[2], y[3]);
}

__device__ __forceinline__ void qk_weight_pairs(const __nv_bfloat16* wt, int sub, uint32_t (&w)[4]) {
  const uint4 wraw = *reinterpret_cast<const uint4*>(wt + sub * 8);
  w[0] = wraw.x; w[1] = wraw.y; w[2] = wraw.z; w[3] = wraw.w;
}

// Where a head vector of a token goes (slot -1: not to the cache).
__device__ __forceinline__ void qk_put_q(const QkNormRopeParams& p, int tok, int hd, int sub, const uint4& out) {
  *reinterpret_cast<uint4*>(p.q_out + (static_cast<long long>(tok) * p.H + hd) * 128 + sub * 8) = out;
}
__device__ __forceinline__ void qk_put_k(const QkNormRopeParams& p, int tok, int hd, int sub, long long slot, const uint4& out) {
  const int kh = hd - p.H;
  *reinterpret_cast<uint4*>(p.k_out + (static_cast<long long>(tok) * p.Hkv + kh) * 128 + sub * 8) = out;
  if (slot >= 0) *reinterpret_cast<uint4*>(p.k_cache + (slot * p.Hkv + kh) * 128 + sub * 8) = out;
}
__device__ __forceinline__ void qk_put_v(const QkNormRopeParams& p, int hd, int sub, long long slot, const uint4& raw) {
  if (slot >= 0) *reinterpret_cast<uint4*>(p.v_cache + (slot * p.Hkv + (hd - p.H - p.Hkv)) * 128 + sub * 8) = raw;     // a bit copy
}

template <int GROUP>
__global__ void __launch_bounds__(kQkThreads, GROUP == 1 ? 4 : kQkCtas)
qk_norm_rope_store_kernel(const QkNormRopeParams p) {
  // A half-warp owns one head vector at a time: lane j of 16 holds elements [8j, 8j + 8) (one 16-byte access),
  // the rotary partner (element i +- 64) of each of them sits in lane j ^ 8.  It takes GROUP consecutive
  // heads of one token per pass -- all loads of the pass go out first -- so that what belongs to the token
  // (slot, position, the lane's cos / sin values) and to the head kind (the norm weight) is fetched once per
  // pass instead of once per head.  GROUP = 1 for decode-sized batches, where the launch is latency bound
  // and more half-warps in flight matter more than the instructions saved.
  const int sub = threadIdx.x & 15;
  const int heads = p.H + 2 * p.Hkv;
  const int groups = (heads + GROUP - 1) / GROUP;                       // per token
  // A half-warp keeps its group of heads and walks over tokens, so there is one division in the kernel, not one per pass.
  const int worker = blockIdx.x * (kQkThreads / 16) + (threadIdx.x >> 4);
  const int stride = gridDim.x * (kQkThreads / 16) / groups;              // tokens (the host sees to it that it is >= 1)
  const int tok0 = worker / groups, hd0 = (worker - tok0 * groups) * GROUP;
  const unsigned half_mask = 0xffffu << (threadIdx.x & 16);
  // Launched with programmatic stream serialization (a decode kernel in front lets it start early).  Everything that counts is read
  // behind the wait, so the kernel in front may write any of it.
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  const bool store = p.slot_mapping && p.k_cache && p.v_cache, any = tok0 < stride && tok0 < p.n_tokens;
  uint32_t wq[4], wk[4];
  long long pos;
  int slot = -1;
  if constexpr (GROUP == 1) {
    // One pass, one head, and one trip behind the wait: the position is read ahead of it as a hint, and what hangs on it or is known
    // anyway is on its way into L2.  The table row of the hint comes with everything else (in 32-byte loads: four of 16 bytes
    // cost a layer 0.2 us); position and row are looked at behind the normalisation, and the row is fetched again if the
    // position has changed.  28 layers of a decode graph, producer and attention, everything behind the wait | this form | table,
    // weights, slot and position in registers ahead of the wait, which a kernel in front must then not write: one sequence 201 |
    // 189 | 187 us, 37 of 100 .. 1024 tokens 564 | 535 | 521, 256 of 100 .. 2048 at 2/1 heads 845 | 803 | 795.
    const __nv_bfloat16* row = p.qkv + static_cast<long long>(tok0) * p.qkv_row_stride + hd0 * 128 + sub * 8;
    const __nv_bfloat16* wt = hd0 < p.H ? p.q_weight : p.k_weight;
    const bool rotated = hd0 < p.H + p.Hkv;
    long long hint = 0;
    if (any) {
      if ((sub & 7) == 0) prefetch_l2(row);
      // (what many half-warps share is asked for by a few of them: requests for one line queue up)
      if (store && threadIdx.x == 0) prefetch_l2(p.slot_mapping + tok0);
      if (blockIdx.x < 2 && threadIdx.x < 4) prefetch_l2((threadIdx.x < 2 ? p.q_weight : p.k_weight) + (threadIdx.x & 1) * 64);
      if (rotated) {
        hint = ld_cg_s64(p.positions + tok0);
        if ((sub & 3) == 0) prefetch_l2(qk_table_row(p, hint, sub) + (sub & 8) * 8);
      }
    }
    asm volatile("griddepcontrol.wait;" ::: "memory");
    if (!any) return;
    uint4 out = ld_row16(row);
    if (rotated) {
      qk_weight_pairs(wt, sub, wq);
      QkTableRow t = qk_load_table(p, hint, sub);
      pos = ld_s64(p.positions + tok0);
      if (store && hd0 >= p.H) slot = ld_s32(p.slot_mapping + tok0);
      uint32_t ap[4];
      qk_normalise(out, wq, p.eps, half_mask, ap);
      if (pos != hint) t = qk_load_table(p, pos, sub);
      out = qk_rotate(ap, qk_token_ctx(p, t, slot, sub), half_mask);
    } else if (store) {
      slot = ld_s32(p.slot_mapping + tok0);
    }
    const long long to = slot < p.n_slots ? slot : -1;       // never write outside the cache
    if (hd0 < p.H) {
      qk_put_q(p, tok0, hd0, sub, out);
    } else if (rotated) {
      qk_put_k(p, tok0, hd0, sub, to, out);
    } else {
      qk_put_v(p, hd0, sub, to, out);
    }
    return;
  }
  asm volatile("griddepcontrol.wait;" ::: "memory");
  if (!any) return;
  qk_weight_pairs(p.q_weight, sub, wq);
  qk_weight_pairs(p.k_weight, sub, wk);
  pos = p.positions[tok0];
  if (store) slot = p.slot_mapping[tok0];
  // Position and slot are fetched a token ahead: the table row hangs on the position, and two trips in a row are what a
  // pass would otherwise wait for.
  for (int tok = tok0; tok < p.n_tokens; tok += stride) {
    const __nv_bfloat16* row = p.qkv + static_cast<long long>(tok) * p.qkv_row_stride + sub * 8;
    uint4 raw[GROUP];
#pragma unroll
    for (int g = 0; g < GROUP; ++g)
      if (hd0 + g < heads) raw[g] = *reinterpret_cast<const uint4*>(row + (hd0 + g) * 128);
    const float* cs = qk_table_row(p, pos, sub);
    QkTableRow t;
    t.c0 = *reinterpret_cast<const float4*>(cs);
    t.c1 = *reinterpret_cast<const float4*>(cs + 4);
    t.s0 = *reinterpret_cast<const float4*>(cs + 64);
    t.s1 = *reinterpret_cast<const float4*>(cs + 68);
    const QkTokenCtx c = qk_token_ctx(p, t, slot, sub);
    if (tok + stride < p.n_tokens) {
      pos = p.positions[tok + stride];
      if (store) slot = p.slot_mapping[tok + stride];
    }
#pragma unroll
    for (int g = 0; g < GROUP; ++g) {
      const int hd = hd0 + g;
      if (hd >= heads) break;
      if (hd >= p.H + p.Hkv) {
        qk_put_v(p, hd, sub, c.slot, raw[g]);
      } else if (hd < p.H) {
        uint32_t ap[4];
        qk_normalise(raw[g], wq, p.eps, half_mask, ap);
        qk_put_q(p, tok, hd, sub, qk_rotate(ap, c, half_mask));
      } else {
        uint32_t ap[4];
        qk_normalise(raw[g], wk, p.eps, half_mask, ap);
        qk_put_k(p, tok, hd, sub, c.slot, qk_rotate(ap, c, half_mask));
      }
    }
  }
}

}  // namespace b200

extern "C" int b200_qk_norm_rope_store(const void* qkv, int64_t qkv_row_stride, const int64_t* positions,
                                       const void* q_weight, const void* k_weight, const float* cos_sin_cache,
                                       int32_t max_position, float eps, void* q_out, void* k_out, void* k_cache,
                                       void* v_cache, const int32_t* slot_mapping, int64_t n_slots, int32_t n_tokens,
                                       int32_t num_heads, int32_t num_kv_heads, int32_t head_dim, void* stream) {
  using namespace b200;
  if (n_tokens == 0) return kOk;
  if (!qkv || !positions || !q_weight || !k_weight || !cos_sin_cache || !q_out || !k_out)
    return set_error(kErrNullPointer, "qk_norm_rope_store: null pointer");
  if (head_dim != 128 || num_heads <= 0 || num_kv_heads <= 0 || n_tokens < 0 || max_position <= 0)
    return set_error(kErrBadShape, "qk_norm_rope_store: head_dim must be 128 and the counts positive (H=%d Hkv=%d D=%d n=%d)",
                     num_heads, num_kv_heads, head_dim, n_tokens);
  if ((k_cache == nullptr) != (v_cache == nullptr))
    return set_error(kErrNullPointer, "qk_norm_rope_store: k_cache and v_cache must both be given or both be null");
  if (k_cache && !slot_mapping) return set_error(kErrNullPointer, "qk_norm_rope_store: a cache needs slot_mapping");
  if (k_cache && n_slots <= 0) return set_error(kErrBadShape, "qk_norm_rope_store: n_slots must be positive");
  const long long width = static_cast<long long>(num_heads + 2 * num_kv_heads) * 128;
  if (qkv_row_stride < width || qkv_row_stride % 8 != 0)
    return set_error(kErrMisaligned, "qk_norm_rope_store: qkv_row_stride must be >= (H + 2 Hkv) * 128 and a multiple of 8 elements");
  auto mis = [](const void* ptr, uintptr_t a) { return ptr && (reinterpret_cast<uintptr_t>(ptr) & (a - 1)) != 0; };
  if (mis(qkv, 16) || mis(q_out, 16) || mis(k_out, 16) || mis(k_cache, 16) || mis(v_cache, 16) || mis(q_weight, 16) ||
      mis(k_weight, 16) || mis(cos_sin_cache, 16))
    return set_error(kErrMisaligned, "qk_norm_rope_store: every tensor must be 16-byte aligned");
  QkNormRopeParams p;
  p.qkv = static_cast<const __nv_bfloat16*>(qkv);
  p.qkv_row_stride = qkv_row_stride;
  p.positions = reinterpret_cast<const long long*>(positions);
  p.q_weight = static_cast<const __nv_bfloat16*>(q_weight);
  p.k_weight = static_cast<const __nv_bfloat16*>(k_weight);
  p.cos_sin = cos_sin_cache;
  p.max_position = max_position;
  p.wide_table = reinterpret_cast<uintptr_t>(cos_sin_cache) % 32 == 0;
  p.eps = eps;
  p.q_out = static_cast<__nv_bfloat16*>(q_out);
  p.k_out = static_cast<__nv_bfloat16*>(k_out);
  p.k_cache = static_cast<__nv_bfloat16*>(k_cache);
  p.v_cache = static_cast<__nv_bfloat16*>(v_cache);
  p.slot_mapping = slot_mapping;
  p.n_slots = n_slots;
  p.n_tokens = n_tokens;
  p.H = num_heads;
  p.Hkv = num_kv_heads;
  const int sms = sm_count();
  if (sms <= 0) return set_error(kErrNoDriver, "qk_norm_rope_store: no CUDA device");
  const int heads = num_heads + 2 * num_kv_heads;
  // one head per pass while that still leaves fewer half-warps than the device can hold
  const bool small = static_cast<long long>(n_tokens) * heads <= static_cast<long long>(sms) * 6 * (kQkThreads / 16);
  const int group = small ? 1 : kQkGroup;
  const long long n_units = static_cast<long long>(n_tokens) * ((heads + group - 1) / group);
  const long long want = (n_units + kQkThreads / 16 - 1) / (kQkThreads / 16);
  const long long per_token = ((heads + group - 1) / group + kQkThreads / 16 - 1) / (kQkThreads / 16);   // CTAs one token takes
  long long cap = static_cast<long long>(sms) * (small ? 8 : kQkCtas);
  if (cap < per_token) cap = per_token;
  const int grid = static_cast<int>(want < cap ? want : cap);
  const cudaError_t le = launch_early(small ? qk_norm_rope_store_kernel<1> : qk_norm_rope_store_kernel<kQkGroup>, grid, kQkThreads,
                                      0, static_cast<cudaStream_t>(stream), p);
  g_launches.fetch_add(1);
  return check_cuda(le != cudaSuccess ? le : cudaGetLastError(), "qk_norm_rope_store launch");
}
