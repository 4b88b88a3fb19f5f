// Varlen causal prefill attention on warp-level mma.sync: head ratios that the tcgen05 kernel
// (prefill_attn_tc2.cu) does not take, and prompts too short for it.  Replaces flash_attn_varlen_func as called at
// nanovllm/layers/attention.py:64-70, for dense K/V and for K/V read from the paged cache.
//
// One CTA owns `QT = 16 * WARPS / G` consecutive query tokens of one sequence for one kv head: its
// 16-row-per-warp M dimension is the (token, query-head-of-the-group) product, so each K/V tile
// is loaded once for all G query heads that share it.  K/V arrive as 64-token TMA tiles through
// a 4-stage mbarrier ring fed by a producer warp; the consumer warps run QK^T, online softmax and
// PV in registers.  A tile costs a scheduler 1.05 us per warp that it holds (the mma.sync rate), so short prompts, where
// CTAs are few and latency is all there is, take 4 warps per CTA, one per scheduler, and large batches 8.  Two more
// warps do the layer's cache store where the call asks for it.
#include <atomic>

#include "../../include/b200_attn.h"
#include "kernels.cuh"

namespace b200 {
extern std::atomic<long long> g_launches;

constexpr int kPfTile = 64;
constexpr int kPfSub = kPfTile * 128;
constexpr int kPfStageBytes = 4 * kPfSub;
constexpr int kPfStages = 4;
constexpr int kPfStoreThreads = 64;      // one warp for K, one for V

static __device__ int g_status_prefill_mma = 0;

// The layer's cache store (nanovllm/layers/attention.py:10-40) on the side: attention over dense K and V does not read the
// cache.  A CTA sends on the rows of its own query tokens (they are keys of its last tiles) from shared memory.
__device__ __forceinline__ void pf_store_tile(const PrefillParams& p, char* cache, const unsigned char* tile, int h, int r0,
                                              int r1, const int (&slots)[2], int lane) {
  const long long row_bytes = static_cast<long long>(p.Hkv) * 256;
  for (int r2 = r0; r2 < r1; r2 += 2) {               // two rows per pass, half a warp each
    const int r = r2 + (lane >> 4), c = lane & 15;
    const int s_lo = __shfl_sync(0xffffffffu, slots[0], r & 31), s_hi = __shfl_sync(0xffffffffu, slots[1], r & 31);
    const int slot = r < 32 ? s_lo : s_hi;
    if (r < r1 && slot >= 0 && slot < p.st_n_slots)
      *reinterpret_cast<uint4*>(cache + slot * row_bytes + h * 256 + c * 16) =
          *reinterpret_cast<const uint4*>(tile + (c >> 3) * kPfSub + r * 128 + (((c & 7) ^ (r & 7)) << 4));
  }
}
// Rows [row0, row1) from memory, kv heads [h0, h1): what no CTA has as its own query tokens.
__device__ __forceinline__ void pf_store_rows(const PrefillParams& p, const char* src, long long stride, char* cache, int row0, int row1,
                                              int h0, int h1, int lane) {
  const int vecs = p.Hkv * 16;
  for (int r = row0; r < row1; ++r) {
    const long long slot = ld_s32(p.st_slots + r);
    if (slot < 0 || slot >= p.st_n_slots) continue;
    for (int v = h0 * 16 + lane; v < h1 * 16; v += 32)
      reinterpret_cast<uint4*>(cache)[slot * vecs + v] = ld_row16(src + r * stride + v * 16);
  }
}

template <int kPfConsumerWarps>
__global__ void __launch_bounds__(kPfConsumerWarps * 32 + 32 + kPfStoreThreads, 1)
prefill_attn_mma_kernel(const PrefillParams p, const __grid_constant__ CUtensorMap map_k,
                        const __grid_constant__ CUtensorMap map_v) {
  extern __shared__ unsigned char smem_raw[];
  unsigned char* stages = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  __shared__ __align__(8) uint64_t bar_full[kPfStages];
  __shared__ __align__(8) uint64_t bar_empty[kPfStages];
  __shared__ __align__(8) uint64_t bar_last;     // the last tile's load is under way
  __shared__ int s_abort;

  constexpr int kPfConsumers = kPfConsumerWarps * 32;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int G = p.G, QT = p.QT;
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  if (tid == kPfConsumers) {
    tma_prefetch_desc(&map_k);
    tma_prefetch_desc(&map_v);
  }
  if (tid == 0) {
    s_abort = 0;
    for (int s = 0; s < kPfStages; ++s) {
      mbar_init(&bar_full[s], 1);
      mbar_init(&bar_empty[s], kPfConsumerWarps);
    }
    mbar_init(&bar_last, 1);
    mbar_fence_init();
  }
  const int h = blockIdx.x % p.Hkv;
  const int x = p.n_slots - 1 - static_cast<int>(blockIdx.x / p.Hkv);  // later (heavier) tiles first
  // Everything is read behind the wait, so the kernel in front may write any of it.  Every CTA waits, those with nothing to do as
  // well, so that this launch ends behind that kernel.
  asm volatile("griddepcontrol.wait;" ::: "memory");

  // slot -> (sequence, query tile): sequence i owns slots [cu_q[i] / QT + i, ... + ceil(Lq_i / QT)).  Each warp looks for itself, 32
  // places at a time; the last look has the sequence's bounds as well.  Per launch in a graph of launches, a binary search behind the
  // wait | ahead of it, which bars the kernel in front from writing cu_seqlens | this: 16/8 heads, 1 prompt of 33 tokens 3.98 | 3.85 |
  // 4.11 us, 8 of 60 5.5 | 4.9 | 5.1, 128 of 20 36.0 | 35.1 | 30.1; 4/2, 32 of 100 10.5 | 10.0 | 9.7; 2/1, 256 of 10 10.7 | 9.5 | 8.1.
  int seq = 0, left = p.batch;
  while (left > 31) {
    const int step = (left + 31) / 32, i = seq + lane * step;
    const unsigned below = __ballot_sync(0xffffffffu, lane * step < left && ld_s32(p.cu_q + min(i, p.batch)) / QT + i <= x);
    const int skip = max(__popc(below) - 1, 0) * step;
    seq += skip;
    left = min(step, left - skip);
  }
  const int cq = ld_s32(p.cu_q + min(seq + lane, p.batch)), ck = ld_s32(p.cu_k + min(seq + lane, p.batch));
  int at = 0;
  if (left > 1) at = max(__popc(__ballot_sync(0xffffffffu, lane < left && cq / QT + seq + lane <= x)) - 1, 0);
  seq += at;
  const int q_begin = __shfl_sync(0xffffffffu, cq, at), Lq = __shfl_sync(0xffffffffu, cq, at + 1) - q_begin;
  const int k_begin = __shfl_sync(0xffffffffu, ck, at), Lk = __shfl_sync(0xffffffffu, ck, at + 1) - k_begin;
  const int qt = x - (q_begin / QT + seq);
  const bool storing = warp > kPfConsumerWarps, st_v = warp == kPfConsumerWarps + 2;
  char* const st_cache = st_v ? p.st_v_cache : p.st_k_cache;
  const char* const st_src = st_v ? p.st_v : p.st_k;
  const long long st_stride = st_v ? p.st_v_stride : p.st_k_stride;
  if (storing) {
    if (!p.st_slots) return;
    // rows that belong to no query block: sequences without queries, rows outside cu_seqlens_k
    for (int i = blockIdx.x; i < p.batch; i += gridDim.x)
      if (ld_s32(p.cu_q + i) == ld_s32(p.cu_q + i + 1))
        pf_store_rows(p, st_src, st_stride, st_cache, ld_s32(p.cu_k + i), min(ld_s32(p.cu_k + i + 1), p.st_tokens), 0, p.Hkv, lane);
    if (blockIdx.x == 0) {
      pf_store_rows(p, st_src, st_stride, st_cache, 0, min(ld_s32(p.cu_k), p.st_tokens), 0, p.Hkv, lane);
      pf_store_rows(p, st_src, st_stride, st_cache, ld_s32(p.cu_k + p.batch), p.st_tokens, 0, p.Hkv, lane);
    }
  }
  if (qt < 0 || qt * QT >= Lq) return;
  const int tq0 = qt * QT;                       // first query token of this CTA within the sequence
  const int tq1 = min(tq0 + QT, Lq);
  const int shift = Lk - Lq;                     // bottom-right causal alignment
  const int kv_end = min(Lk, shift + tq1);       // keys [0, kv_end) are visible to at least one row
  const int n_tiles = (kv_end + kPfTile - 1) / kPfTile;
  if (storing && shift != 0) {
    // queries and keys do not start together: the CTA of the last query block stores the sequence's rows of its head
    if (tq1 == Lq) pf_store_rows(p, st_src, st_stride, st_cache, k_begin, min(k_begin + Lk, p.st_tokens), h, h + 1, lane);
    return;
  }
  if (n_tiles <= 0) {
    if (storing) return;
    // no visible key (Lk < Lq rows): zeros, as the reference's attention library does
    for (int e = tid; e < (tq1 - tq0) * G * 128; e += kPfConsumers + 32) {
      const int r = e >> 7, d = e & 127;
      p.out[(static_cast<long long>(q_begin + tq0 + r / G) * p.H + h * G + r % G) * 128 + d] = __float2bfloat16(0.f);
    }
    return;
  }

  // (the store warps take part only where they get this far)
  named_bar_sync(2, kPfConsumers + 32 + (p.st_slots && shift == 0 ? kPfStoreThreads : 0));
  volatile int* abort_flag = &s_abort;

  if (storing) {
    for (int t = tq0 / kPfTile; t <= (tq1 - 1) / kPfTile; ++t) {
      const int key0 = t * kPfTile, row0 = k_begin + key0;
      const int r0 = max(tq0 - key0, 0), r1 = min(min(tq1 - key0, kPfTile), p.st_tokens - row0);
      int slots[2];
#pragma unroll
      for (int u = 0; u < 2; ++u) slots[u] = u * 32 + lane >= r0 && u * 32 + lane < r1 ? ld_s32(p.st_slots + row0 + u * 32 + lane) : -1;
      // These are among the CTA's last tiles: once the very last is under way their stages are not loaded again, and each
      // full-barrier is in its tile's phase.
      if (!mbar_wait(&bar_last, 0, abort_flag) || !mbar_wait(&bar_full[t % kPfStages], (t / kPfStages) & 1, abort_flag)) return;
      pf_store_tile(p, st_cache, stages + (t % kPfStages) * kPfStageBytes + (st_v ? 2 * kPfSub : 0), h, r0, r1, slots, lane);
    }
    return;
  }

  if (warp == kPfConsumerWarps) {
    if (lane == 0) {
      const int* bt_row = p.block_tables ? p.block_tables + seq * p.bt_row_stride : nullptr;
      for (int t = 0; t < n_tiles; ++t) {
        const int stage = t % kPfStages;
        const uint32_t ph = (t / kPfStages) & 1;
        if (!mbar_wait(&bar_empty[stage], ph ^ 1, abort_flag)) { atomicExch(&g_status_prefill_mma, 1); break; }
        int row0;
        if (bt_row) {
          const int tok0 = t * kPfTile;
          const int col = tok0 / p.block_size;
          const long long blk = col < p.bt_cols ? bt_row[col] : -1;
          row0 = (blk >= 0 && blk < p.num_blocks) ? static_cast<int>(blk * p.block_size + (tok0 - col * p.block_size))
                                                  : -kPfTile;
        } else {
          row0 = k_begin + t * kPfTile;
        }
        unsigned char* st = stages + stage * kPfStageBytes;
        mbar_expect_tx(&bar_full[stage], kPfStageBytes);
        tma_load_3d(st, &map_k, &bar_full[stage], 0, h, row0);
        tma_load_3d(st + kPfSub, &map_k, &bar_full[stage], 64, h, row0);
        tma_load_3d(st + 2 * kPfSub, &map_v, &bar_full[stage], 0, h, row0);
        tma_load_3d(st + 3 * kPfSub, &map_v, &bar_full[stage], 64, h, row0);
        if (t + 1 == n_tiles) mbar_arrive(&bar_last);
      }
    }
    return;
  }

  // ------------------------------- consumers -------------------------------
  const int quad = lane & 3;
  const int r0 = warp * 16 + (lane >> 2), r1 = r0 + 8;      // rows of the (token, head) product
  const int tok0 = tq0 + r0 / G, tok1 = tq0 + r1 / G;       // query token within the sequence
  const bool ok0 = r0 < QT * G && tok0 < Lq, ok1 = r1 < QT * G && tok1 < Lq;
  const int kmax0 = ok0 ? shift + tok0 : -1;                // last visible key (inclusive)
  const int kmax1 = ok1 ? shift + tok1 : -1;
  int wmax = max(kmax0, kmax1), wmin = min(kmax0, kmax1);
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) {
    wmax = max(wmax, __shfl_xor_sync(0xffffffffu, wmax, off));
    wmin = min(wmin, __shfl_xor_sync(0xffffffffu, wmin, off));
  }

  uint32_t qa[8][4];
  {
    const uint32_t* q0 = reinterpret_cast<const uint32_t*>(
        p.q + static_cast<long long>(q_begin + tok0) * p.q_row_stride + (h * G + r0 % G) * 128);
    const uint32_t* q1 = reinterpret_cast<const uint32_t*>(
        p.q + static_cast<long long>(q_begin + tok1) * p.q_row_stride + (h * G + r1 % G) * 128);
#pragma unroll
    for (int ks = 0; ks < 8; ++ks) {
      qa[ks][0] = ok0 ? ld_u32(q0 + ks * 8 + quad) : 0u;
      qa[ks][1] = ok1 ? ld_u32(q1 + ks * 8 + quad) : 0u;
      qa[ks][2] = ok0 ? ld_u32(q0 + ks * 8 + 4 + quad) : 0u;
      qa[ks][3] = ok1 ? ld_u32(q1 + ks * 8 + 4 + quad) : 0u;
    }
  }
  float o[16][4];
#pragma unroll
  for (int n = 0; n < 16; ++n) o[n][0] = o[n][1] = o[n][2] = o[n][3] = 0.f;
  float m0 = -INFINITY, m1 = -INFINITY, l0 = 0.f, l1 = 0.f;

  for (int t = 0; t < n_tiles; ++t) {
    const int stage = t % kPfStages;
    const uint32_t ph = (t / kPfStages) & 1;
    if (!mbar_wait(&bar_full[stage], ph, abort_flag)) { if (lane == 0) atomicExch(&g_status_prefill_mma, 1); return; }
    const int key0 = t * kPfTile;
    if (key0 + kPfTile > Lk) {
      // ragged last tile: rows past the sequence end are foreign data; zero V there
      unsigned char* vb = stages + stage * kPfStageBytes + 2 * kPfSub;
      const int first = Lk - key0;
      for (int e = tid; e < (kPfTile - first) * 16; e += kPfConsumers) {
        const int r = first + (e >> 4), c = e & 15;
        *reinterpret_cast<uint4*>(vb + (c >> 3) * kPfSub + r * 128 + (((c & 7) ^ (r & 7)) << 4)) = make_uint4(0, 0, 0, 0);
      }
      fence_proxy_async_smem();
      named_bar_sync(1, kPfConsumers);
    }
    if (key0 <= wmax) {
      const uint32_t st = smem_u32(stages + stage * kPfStageBytes);
      const uint32_t k_base = st, v_base = st + 2 * kPfSub;
      float s[8][4];
#pragma unroll
      for (int j = 0; j < 8; ++j) s[j][0] = s[j][1] = s[j][2] = s[j][3] = 0.f;
      {
        const int trow = ((lane >> 4) << 3) + (lane & 7);
        const int dsel = ((lane >> 3) & 1) << 3;
#pragma unroll
        for (int ks = 0; ks < 8; ++ks) {
#pragma unroll
          for (int j2 = 0; j2 < 4; ++j2) {
            uint32_t b0, b1, b2, b3;
            ldmatrix_x4(k_base + tile_offset(j2 * 16 + trow, ks * 16 + dsel, kPfTile), b0, b1, b2, b3);
            mma_bf16_16816(s[2 * j2], qa[ks], b0, b1);
            mma_bf16_16816(s[2 * j2 + 1], qa[ks], b2, b3);
          }
        }
      }
      const bool need_mask = key0 + kPfTile - 1 > wmin;
      float mx0 = -INFINITY, mx1 = -INFINITY;
#pragma unroll
      for (int j = 0; j < 8; ++j) {
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          const int key = key0 + j * 8 + quad * 2 + e;
          float v0 = s[j][e] * p.scale_log2, v1 = s[j][2 + e] * p.scale_log2;
          if (need_mask) {
            if (key > kmax0) v0 = -INFINITY;
            if (key > kmax1) v1 = -INFINITY;
          }
          s[j][e] = v0;
          s[j][2 + e] = v1;
          mx0 = fmaxf(mx0, v0);
          mx1 = fmaxf(mx1, v1);
        }
      }
      mx0 = fmaxf(mx0, __shfl_xor_sync(0xffffffffu, mx0, 1));
      mx0 = fmaxf(mx0, __shfl_xor_sync(0xffffffffu, mx0, 2));
      mx1 = fmaxf(mx1, __shfl_xor_sync(0xffffffffu, mx1, 1));
      mx1 = fmaxf(mx1, __shfl_xor_sync(0xffffffffu, mx1, 2));
      const float mn0 = fmaxf(m0, mx0), mn1 = fmaxf(m1, mx1);
      const float ms0 = mn0 == -INFINITY ? 0.f : mn0, ms1 = mn1 == -INFINITY ? 0.f : mn1;
      const float a0 = fast_exp2(m0 - ms0), a1 = fast_exp2(m1 - ms1);
      m0 = mn0; m1 = mn1;
      float ps0 = 0.f, ps1 = 0.f;
#pragma unroll
      for (int j = 0; j < 8; ++j) {
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          s[j][e] = fast_exp2(s[j][e] - ms0);
          s[j][2 + e] = fast_exp2(s[j][2 + e] - ms1);
          ps0 += s[j][e];
          ps1 += s[j][2 + e];
        }
      }
      l0 = l0 * a0 + ps0;
      l1 = l1 * a1 + ps1;
      if (a0 != 1.f || a1 != 1.f) {
#pragma unroll
        for (int n = 0; n < 16; ++n) { o[n][0] *= a0; o[n][1] *= a0; o[n][2] *= a1; o[n][3] *= a1; }
      }
      {
        const int trow = (((lane >> 3) & 1) << 3) + (lane & 7);
        const int dsel = (lane >> 4) << 3;
#pragma unroll
        for (int kk = 0; kk < 4; ++kk) {
          uint32_t pa[4];
          pa[0] = pack_bf16(s[2 * kk][0], s[2 * kk][1]);
          pa[1] = pack_bf16(s[2 * kk][2], s[2 * kk][3]);
          pa[2] = pack_bf16(s[2 * kk + 1][0], s[2 * kk + 1][1]);
          pa[3] = pack_bf16(s[2 * kk + 1][2], s[2 * kk + 1][3]);
#pragma unroll
          for (int n2 = 0; n2 < 8; ++n2) {
            uint32_t b0, b1, b2, b3;
            ldmatrix_x4_trans(v_base + tile_offset(kk * 16 + trow, n2 * 16 + dsel, kPfTile), b0, b1, b2, b3);
            mma_bf16_16816(o[2 * n2], pa, b0, b1);
            mma_bf16_16816(o[2 * n2 + 1], pa, b2, b3);
          }
        }
      }
    }
    __syncwarp();
    if (lane == 0) mbar_arrive(&bar_empty[stage]);
  }

  l0 += __shfl_xor_sync(0xffffffffu, l0, 1);
  l0 += __shfl_xor_sync(0xffffffffu, l0, 2);
  l1 += __shfl_xor_sync(0xffffffffu, l1, 1);
  l1 += __shfl_xor_sync(0xffffffffu, l1, 2);
  const float inv0 = l0 > 0.f ? 1.f / l0 : 0.f, inv1 = l1 > 0.f ? 1.f / l1 : 0.f;
  if (ok0) {
    uint32_t* dst = reinterpret_cast<uint32_t*>(p.out + (static_cast<long long>(q_begin + tok0) * p.H + h * G + r0 % G) * 128);
#pragma unroll
    for (int n = 0; n < 16; ++n) dst[n * 4 + quad] = pack_bf16(o[n][0] * inv0, o[n][1] * inv0);
  }
  if (ok1) {
    uint32_t* dst = reinterpret_cast<uint32_t*>(p.out + (static_cast<long long>(q_begin + tok1) * p.H + h * G + r1 % G) * 128);
#pragma unroll
    for (int n = 0; n < 16; ++n) dst[n * 4 + quad] = pack_bf16(o[n][2] * inv1, o[n][3] * inv1);
  }
}

int launch_prefill_mma(PrefillParams p, const CUtensorMap& map_k, const CUtensorMap& map_v, bool small, cudaStream_t stream) {
  const size_t smem = 1024 + static_cast<size_t>(kPfStages) * kPfStageBytes;
  static std::atomic<size_t> configured[2][kMaxDevices];
  const int warps = small ? 4 : 8;
  auto* const kernel = small ? prefill_attn_mma_kernel<4> : prefill_attn_mma_kernel<8>;
  const int rc = ensure_dynamic_smem(reinterpret_cast<const void*>(kernel), smem, configured[small],
                                     "prefill_attn(mma.sync): cudaFuncSetAttribute");
  if (rc) return rc;
  p.QT = 16 * warps / p.G;
  p.n_slots = p.total_q / p.QT + p.batch;
  const long long blocks = static_cast<long long>(p.n_slots) * p.Hkv;
  if (blocks <= 0) return kOk;
  if (blocks > 0x7fffffffLL) return set_error(kErrBadShape, "prefill_attn: too many query tiles");
  const cudaError_t le = launch_early(kernel, static_cast<unsigned>(blocks), warps * 32 + 32 + kPfStoreThreads, smem, stream, p, map_k, map_v);
  g_launches.fetch_add(1);
  return check_cuda(le != cudaSuccess ? le : cudaGetLastError(), "prefill_attn launch");
}

int read_status_prefill_mma() {
  int v = 0;
  cudaMemcpyFromSymbol(&v, g_status_prefill_mma, sizeof(int));
  return v;
}

int reset_state_prefill_mma() {
  const int zero = 0;
  return check_cuda(cudaMemcpyToSymbol(g_status_prefill_mma, &zero, sizeof(int)), "device_status: clearing the mma.sync status word");
}

}  // namespace b200
