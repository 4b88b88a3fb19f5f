// Building blocks shared by the two decode kernels (decode_attn.cu, decode_cluster.cu): the tile of 64 tokens, the
// work of one consumer warp on its 16-token slab of it, and the states that are combined at the end.
#pragma once
#include "kernels.cuh"

namespace b200 {

constexpr int kTile = 64;                       // tokens per stage
constexpr int kSubTileBytes = kTile * 128;      // 64 tokens x 64 dims bf16
constexpr int kStageBytes = 4 * kSubTileBytes;  // K lo, K hi, V lo, V hi
constexpr int kDecConsumerWarps = 4;
constexpr int kDecConsumers = kDecConsumerWarps * 32;
constexpr int kMaxG = 16;

struct DecodeParams {
  const __nv_bfloat16* q;
  long long q_row_stride;
  __nv_bfloat16* out;
  const int* context_lens;
  const int* block_tables;
  long long bt_row_stride;
  int bt_cols;
  int batch, H, Hkv, G;
  int block_size;
  long long num_blocks;
  float scale_log2;
  int n_merge;    // hand-off buffers between the consumer warps and the epilogue warp (1 or 2)
  float* ws_o;    // [slots][G][128] unnormalised partial outputs
  float* ws_ml;   // [slots][G][2]   running max (log2 domain) and sum
  int* counters;  // [batch * Hkv], zero between launches
  unsigned int* ticket;  // unit scheduler, zero between launches
  // the step's cache store in the same launch: row i of st_k / st_v to slot st_slots[i]; nullptr: none
  const int* st_slots;
  const __nv_bfloat16 *st_k, *st_v;
  long long st_k_stride, st_v_stride, st_n_slots;   // elements; slots of the cache
  __nv_bfloat16 *st_k_cache, *st_v_cache;
};

// One 16-byte chunk per lane of head h of the step's row `tok`: lanes 0 .. 15 K, 16 .. 31 V.
__device__ __forceinline__ uint4 step_chunk(const DecodeParams& p, int tok, int h, int lane) {
  const __nv_bfloat16* src = lane < 16 ? p.st_k + tok * p.st_k_stride : p.st_v + tok * p.st_v_stride;
  return ld_row16(src + h * 128 + (lane & 15) * 8);
}

// 1-D bulk copy global -> shared, completion counted on an mbarrier (addresses and size multiples of 16).
__device__ __forceinline__ void bulk_load_1d(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
               ::"r"(smem_u32(dst)), "l"(reinterpret_cast<uint64_t>(src)), "r"(bytes), "r"(smem_u32(bar))
               : "memory");
}

// Running state of one consumer warp over one (sequence, kv head): rows of the accumulator fragment = query heads.
struct DecAcc {
  float o[16][4];
  float m0, m1, l0, l1;
  __device__ __forceinline__ void reset() {
#pragma unroll
    for (int n = 0; n < 16; ++n) o[n][0] = o[n][1] = o[n][2] = o[n][3] = 0.f;
    m0 = m1 = -INFINITY;
    l0 = l1 = 0.f;
  }
};

// The G query rows (in shared memory) as the A operand: rows = the query heads that share the kv head.
__device__ __forceinline__ void dec_query_fragments(const __nv_bfloat16* q, int G, int lane, uint32_t (&qa)[8][4]) {
  const int row = lane >> 2, quad = lane & 3;
  const uint32_t* q0 = reinterpret_cast<const uint32_t*>(q + row * 128);
  const uint32_t* q1 = q0 + 8 * 64;
#pragma unroll
  for (int ks = 0; ks < 8; ++ks) {
    qa[ks][0] = row < G ? q0[ks * 8 + quad] : 0u;
    qa[ks][1] = row + 8 < G ? q1[ks * 8 + quad] : 0u;
    qa[ks][2] = row < G ? q0[ks * 8 + 4 + quad] : 0u;
    qa[ks][3] = row + 8 < G ? q1[ks * 8 + 4 + quad] : 0u;
  }
}

// One warp's 16-token slab of a tile in shared memory (`valid` > 0 of its tokens exist): S = Q K^T, online softmax in
// the log2 domain, O += P V.
__device__ __forceinline__ void dec_tile(unsigned char* stage, int warp, int lane, int valid, float scale_log2,
                                         const uint32_t (&qa)[8][4], DecAcc& a) {
  const int quad = lane & 3;
  const uint32_t st = smem_u32(stage);
  const uint32_t k_base = st, v_base = st + 2 * kSubTileBytes;
  if (valid < 16) {
    // rows past the sequence end hold whatever the cache block holds: zero the V rows so
    // that 0 * garbage cannot produce NaN (K garbage is masked by select below)
    unsigned char* vb = stage + 2 * kSubTileBytes;
    for (int e = lane; e < 16 * 16; e += 32) {
      const int r = warp * 16 + (e >> 4), c = e & 15;
      if ((e >> 4) >= valid)
        *reinterpret_cast<uint4*>(vb + (c >> 3) * kSubTileBytes + r * 128 + (((c & 7) ^ (r & 7)) << 4)) =
            make_uint4(0, 0, 0, 0);
    }
    fence_proxy_async_smem();
    __syncwarp();
  }
  // ---- S = Q K^T (16 x 16 tokens) ----
  float s[2][4];
#pragma unroll
  for (int j = 0; j < 2; ++j) s[j][0] = s[j][1] = s[j][2] = s[j][3] = 0.f;
  {
    const int tok = warp * 16 + ((lane >> 4) << 3) + (lane & 7);
    const int dsel = ((lane >> 3) & 1) << 3;
#pragma unroll
    for (int ks = 0; ks < 8; ++ks) {
      uint32_t b0, b1, b2, b3;
      ldmatrix_x4(k_base + tile_offset(tok, ks * 16 + dsel, kTile), b0, b1, b2, b3);
      mma_bf16_16816(s[0], qa[ks], b0, b1);
      mma_bf16_16816(s[1], qa[ks], b2, b3);
    }
  }
  // ---- online softmax (log2 domain) ----
  float mx0 = -INFINITY, mx1 = -INFINITY;
#pragma unroll
  for (int j = 0; j < 2; ++j) {
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      const bool in = (j * 8 + quad * 2 + e) < valid;
      s[j][e] = in ? s[j][e] * scale_log2 : -INFINITY;
      s[j][2 + e] = in ? s[j][2 + e] * scale_log2 : -INFINITY;
      mx0 = fmaxf(mx0, s[j][e]);
      mx1 = fmaxf(mx1, s[j][2 + e]);
    }
  }
  mx0 = fmaxf(mx0, __shfl_xor_sync(0xffffffffu, mx0, 1));
  mx0 = fmaxf(mx0, __shfl_xor_sync(0xffffffffu, mx0, 2));
  mx1 = fmaxf(mx1, __shfl_xor_sync(0xffffffffu, mx1, 1));
  mx1 = fmaxf(mx1, __shfl_xor_sync(0xffffffffu, mx1, 2));
  const float mn0 = fmaxf(a.m0, mx0), mn1 = fmaxf(a.m1, mx1);
  const float a0 = fast_exp2(a.m0 - mn0), a1 = fast_exp2(a.m1 - mn1);
  a.m0 = mn0; a.m1 = mn1;
  float ps0 = 0.f, ps1 = 0.f;
#pragma unroll
  for (int j = 0; j < 2; ++j) {
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      s[j][e] = fast_exp2(s[j][e] - mn0);
      s[j][2 + e] = fast_exp2(s[j][2 + e] - mn1);
      ps0 += s[j][e];
      ps1 += s[j][2 + e];
    }
  }
  a.l0 = a.l0 * a0 + ps0;
  a.l1 = a.l1 * a1 + ps1;
  if (a0 != 1.f || a1 != 1.f) {
#pragma unroll
    for (int n = 0; n < 16; ++n) { a.o[n][0] *= a0; a.o[n][1] *= a0; a.o[n][2] *= a1; a.o[n][3] *= a1; }
  }
  // ---- O += P V ----
  uint32_t pa[4];
  pa[0] = pack_bf16(s[0][0], s[0][1]);
  pa[1] = pack_bf16(s[0][2], s[0][3]);
  pa[2] = pack_bf16(s[1][0], s[1][1]);
  pa[3] = pack_bf16(s[1][2], s[1][3]);
  {
    const int tok = warp * 16 + (((lane >> 3) & 1) << 3) + (lane & 7);
    const int dsel = (lane >> 4) << 3;
#pragma unroll
    for (int n2 = 0; n2 < 8; ++n2) {
      uint32_t b0, b1, b2, b3;
      ldmatrix_x4_trans(v_base + tile_offset(tok, n2 * 16 + dsel, kTile), b0, b1, b2, b3);
      mma_bf16_16816(a.o[2 * n2], pa, b0, b1);
      mma_bf16_16816(a.o[2 * n2 + 1], pa, b2, b3);
    }
  }
}

// Drops the warp's state where the combining warp finds it: O as [G][128] floats, (max, sum) as [G][2].
__device__ __forceinline__ void dec_hand_off(DecAcc& a, float* mo, float* ml, int G, int lane) {
  const int row = lane >> 2, quad = lane & 3;
  a.l0 += __shfl_xor_sync(0xffffffffu, a.l0, 1);
  a.l0 += __shfl_xor_sync(0xffffffffu, a.l0, 2);
  a.l1 += __shfl_xor_sync(0xffffffffu, a.l1, 1);
  a.l1 += __shfl_xor_sync(0xffffffffu, a.l1, 2);
#pragma unroll
  for (int n = 0; n < 16; ++n) {
    if (row < G) *reinterpret_cast<float2*>(mo + row * 128 + n * 8 + quad * 2) = make_float2(a.o[n][0], a.o[n][1]);
    if (row + 8 < G) *reinterpret_cast<float2*>(mo + (row + 8) * 128 + n * 8 + quad * 2) = make_float2(a.o[n][2], a.o[n][3]);
  }
  if (quad == 0) {
    if (row < G) { ml[row * 2] = a.m0; ml[row * 2 + 1] = a.l0; }
    if (row + 8 < G) { ml[(row + 8) * 2] = a.m1; ml[(row + 8) * 2 + 1] = a.l1; }
  }
}

// The consumer warps' states of query head gq combined; lane owns dims [4 * lane, 4 * lane + 4).  (The sums are written
// out as fused operations: every place this is expanded in must give the same bits.)
struct DecPart {
  float M, L;
  float4 v;
};
template <int WARPS = kDecConsumerWarps>
__device__ __forceinline__ DecPart dec_combine_warps(const float* mo, const float* ml, int G, int gq, int lane) {
  DecPart r;
  r.M = -INFINITY;
#pragma unroll
  for (int w = 0; w < WARPS; ++w) r.M = fmaxf(r.M, ml[(w * G + gq) * 2]);
  r.L = 0.f;
  r.v = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
  for (int w = 0; w < WARPS; ++w) {
    const float wgt = fast_exp2(ml[(w * G + gq) * 2] - r.M);
    r.L = fmaf(ml[(w * G + gq) * 2 + 1], wgt, r.L);
    const float4 v = *reinterpret_cast<const float4*>(mo + (w * G + gq) * 128 + lane * 4);
    r.v.x = fmaf(v.x, wgt, r.v.x); r.v.y = fmaf(v.y, wgt, r.v.y); r.v.z = fmaf(v.z, wgt, r.v.z); r.v.w = fmaf(v.w, wgt, r.v.w);
  }
  return r;
}
__device__ __forceinline__ void dec_store_row(__nv_bfloat16* out_row, const DecPart& a, int lane) {
  const float inv = 1.f / a.L;
  uint2 o2;
  o2.x = pack_bf16(a.v.x * inv, a.v.y * inv);
  o2.y = pack_bf16(a.v.z * inv, a.v.w * inv);
  *reinterpret_cast<uint2*>(out_row + lane * 4) = o2;
}

__device__ __forceinline__ DecPart dec_nothing() {
  DecPart r;
  r.M = -INFINITY;
  r.L = 0.f;
  r.v = make_float4(0.f, 0.f, 0.f, 0.f);
  return r;
}

// The TMA loads of one tile (K lo / hi, V lo / hi; 16-token boxes where only part of it holds tokens).  Returns nothing
// about completion: the bytes arrive on `bar`, whose transaction count the caller has raised by dec_tile_bytes().
__device__ __forceinline__ int dec_tile_slabs(int valid) { return valid >= kTile - 15 ? 4 : (valid + 15) >> 4; }
__device__ __forceinline__ uint32_t dec_tile_bytes(int nslab) { return nslab == 4 ? kStageBytes : nslab * 4 * 2048; }
__device__ __forceinline__ void dec_load_tile(unsigned char* st, uint64_t* bar, const CUtensorMap* map_k, const CUtensorMap* map_v,
                                              const CUtensorMap* map_k16, const CUtensorMap* map_v16, int h, int slot0, int nslab) {
  if (nslab == 4) {
    tma_load_3d(st, map_k, bar, 0, h, slot0);
    tma_load_3d(st + kSubTileBytes, map_k, bar, 64, h, slot0);
    tma_load_3d(st + 2 * kSubTileBytes, map_v, bar, 0, h, slot0);
    tma_load_3d(st + 3 * kSubTileBytes, map_v, bar, 64, h, slot0);
  } else {
    for (int sl = 0; sl < nslab; ++sl) {
      unsigned char* d = st + sl * 2048;
      tma_load_3d(d, map_k16, bar, 0, h, slot0 + sl * 16);
      tma_load_3d(d + kSubTileBytes, map_k16, bar, 64, h, slot0 + sl * 16);
      tma_load_3d(d + 2 * kSubTileBytes, map_v16, bar, 0, h, slot0 + sl * 16);
      tma_load_3d(d + 3 * kSubTileBytes, map_v16, bar, 64, h, slot0 + sl * 16);
    }
  }
}

// Launches the cluster kernel for batches with few (sequence, kv head) pairs; see decode_cluster.cu.
int launch_decode_cluster(const DecodeParams& p, const CUtensorMap& map_k, const CUtensorMap& map_v, const CUtensorMap& map_k16,
                          const CUtensorMap& map_v16, int ctas_per_pair, cudaStream_t stream);
int decode_cluster_ctas(int batch, int Hkv, int G, int max_tiles);

}  // namespace b200
