// Paged single-token decode attention for batches with few (sequence, kv head) pairs: one thread-block cluster per pair.
//
// Latency bound: a single request of 562 tokens is 2.3 MB, 0.35 us of HBM time, and the launch is a chain of dependent
// trips.  A cut through global memory costs store, fence, arrival counter and reload: 5 us, half of the launch (11.4 us
// before, of equal pieces of one tile list).  With few pairs the CTAs of one cluster share the tiles of one pair and push
// their (max, sum, O) through distributed shared memory into the first of them, which writes the row.  Nothing goes
// through global memory, no workspace, and the batch is not scanned: a CTA needs the length and the block-table row
// of one sequence, which it reads in one trip, ahead of the programmatic-launch wait.  Measured in a graph, with the
// producer kernel in front: one sequence of 562 tokens 12.4 -> 7.1 us, 8 of 100 .. 1024 tokens 19.0 -> 9.9 us.
#include "../../include/b200_attn.h"
#include "decode_common.cuh"

namespace b200 {
extern std::atomic<long long> g_launches;

constexpr int kCluStages = 4;          // even: a stage belongs to one of the two groups of consumer warps
constexpr int kCluWarps = 8;           // consumer warps: two groups of four that take the CTA's tiles in turn
constexpr int kCluThreads = kCluWarps * 32 + 32;
constexpr int kCluSlots = 5;           // slots per lane: a batch with a store has at most 32 * kCluSlots sequences
constexpr int kCluMaxG = 8;            // query heads per kv head that the hand-off buffers have room for
static __device__ int g_status_decode_cluster = 0;

__device__ __forceinline__ uint32_t cluster_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }
// Shared-memory address of CTA `rank` of the cluster that corresponds to this CTA's `addr`.
__device__ __forceinline__ uint32_t cluster_addr(uint32_t addr, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
  return r;
}
__device__ __forceinline__ void cluster_store(uint32_t addr, const float4& v) {
  asm volatile("st.shared::cluster.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "f"(v.x), "f"(v.y), "f"(v.z), "f"(v.w) : "memory");
}
__device__ __forceinline__ void cluster_store(uint32_t addr, float a, float b) {
  asm volatile("st.shared::cluster.v2.f32 [%0], {%1, %2};" ::"r"(addr), "f"(a), "f"(b) : "memory");
}
__device__ __forceinline__ void cluster_mbar_arrive(uint32_t bar) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(bar) : "memory");
}
// mbar_wait() for a barrier that other CTAs of the cluster arrive on.
__device__ __forceinline__ bool cluster_mbar_wait(uint64_t* bar, uint32_t parity) {
  const long long t0 = clock64();
  while (true) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok) : "r"(smem_u32(bar)), "r"(parity) : "memory");
    if (ok) return true;
    if (clock64() - t0 > kSpinLimitCycles) return false;
  }
}

// kStore: the step's cache store (nanovllm/layers/attention.py:62-63) in the same launch; as one of its own it is half of what
// an eager step of a small batch costs the host.  Nothing orders this launch's CTAs, so none of them relies on finding
// another's row in the cache: rank 0 of (sequence i, head h) writes row i of head h to its slot, and whoever loads a tile
// that covers ANY slot of the step puts the new row into its copy of the tile.
template <bool kStore>
__global__ void __launch_bounds__(kCluThreads, 1)
decode_cluster_kernel(const DecodeParams p, const __grid_constant__ CUtensorMap map_k,
                      const __grid_constant__ CUtensorMap map_v, const __grid_constant__ CUtensorMap map_k16,
                      const __grid_constant__ CUtensorMap map_v16, const int ctas) {
  extern __shared__ unsigned char smem_raw[];
  unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  const int G = p.G;
  unsigned char* stages = smem;
  __nv_bfloat16* s_q = reinterpret_cast<__nv_bfloat16*>(smem + kCluStages * kStageBytes);          // [G][128]
  float* merge_o = reinterpret_cast<float*>(s_q + G * 128);                                       // [8][G][128]
  float* inbox_o = merge_o + kCluWarps * G * 128;                                         // [ctas][G][128]
  float* merge_ml = inbox_o + ctas * G * 128;                                                     // [8][G][2]
  float* inbox_ml = merge_ml + kCluWarps * G * 2;                                         // [ctas][G][2]
  __shared__ __align__(8) uint64_t bar_full[kCluStages];
  __shared__ __align__(8) uint64_t bar_empty[kCluStages];
  __shared__ __align__(8) uint64_t bar_q, bar_merge, bar_inbox;
  __shared__ int s_abort, s_slot0[kCluStages];

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int rank = static_cast<int>(cluster_rank());
  const int pair = blockIdx.x / ctas;
  const int seq = pair / p.Hkv, h = pair - seq * p.Hkv;
  // Metadata, ahead of the wait for the kernel in front (see decode_attn.cu): length and block-table row in one trip.
  const int* bt_row = p.block_tables + seq * p.bt_row_stride;
  const int max_len = p.bt_cols * p.block_size;
  int len = p.context_lens[seq];
  const int my_blk = warp == kCluWarps && lane < p.bt_cols ? bt_row[lane] : -1;
  if (tid == 0) {
    s_abort = 0;
    for (int s = 0; s < kCluStages; ++s) {
      mbar_init(&bar_full[s], 1);
      mbar_init(&bar_empty[s], kDecConsumerWarps);
    }
    mbar_init(&bar_q, 1);
    mbar_init(&bar_merge, kCluWarps);
    mbar_fence_init();
  }
  if (tid == kCluWarps * 32) {
    tma_prefetch_desc(&map_k);
    tma_prefetch_desc(&map_v);
    tma_prefetch_desc(&map_k16);
    tma_prefetch_desc(&map_v16);
  }
  __syncthreads();
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  len = len < 0 ? 0 : (len > max_len ? max_len : len);
  int slots[kCluSlots];                    // consumer warps: the step's slots, lane l those of sequences l, l + 32, ..
  uint4 own = make_uint4(0, 0, 0, 0);      // and this sequence's new row: lanes 0 .. 15 a K chunk each, 16 .. 31 a V chunk
  if (kStore && warp < kCluWarps) {
    asm volatile("griddepcontrol.wait;" ::: "memory");
    own = step_chunk(p, seq, h, lane);
#pragma unroll
    for (int u = 0; u < kCluSlots; ++u) {
      slots[u] = u * 32 + lane < p.batch ? p.st_slots[u * 32 + lane] : -1;
      if (slots[u] >= p.st_n_slots) slots[u] = -1;
    }
    if (rank == 0 && warp == 0) {
      const long long slot = p.st_slots[seq];
      if (slot >= 0 && slot < p.st_n_slots)
        *reinterpret_cast<uint4*>((lane < 16 ? p.st_k_cache : p.st_v_cache) + (slot * p.Hkv + h) * 128 + (lane & 15) * 8) = own;
    }
  }
  if (len == 0) {
    // no context: zeros (the whole cluster agrees, nobody waits for anybody)
    asm volatile("griddepcontrol.wait;" ::: "memory");
    if (rank == 0) {
      uint2* o = reinterpret_cast<uint2*>(p.out + (static_cast<long long>(seq) * p.H + h * G) * 128);
      for (int v = tid; v < G * 32; v += kCluThreads) o[v] = make_uint2(0, 0);
    }
    return;
  }
  // tiles [t0, t1) of the pair are this CTA's; rank 0 always has some, and min(nt, ctas) of the ranks do
  const int nt = (len + kTile - 1) / kTile;
  const int t0 = (rank * nt + ctas - 1) / ctas, t1 = ((rank + 1) * nt + ctas - 1) / ctas;
  const int active = nt < ctas ? nt : ctas;
  if (tid == 0) {
    mbar_init(&bar_inbox, active * kCluWarps);
    mbar_fence_init();
  }
  __syncwarp();
  cluster_arrive();                       // waited for only in front of the push: by then everybody has long arrived
  if (t0 == t1) return;
  volatile int* abort_flag = &s_abort;

  if (warp == kCluWarps) {
    // =========================== producer warp ===========================
    // The first tiles start on their way into L2 while the kernel in front still runs (nothing is read yet).
    for (int t = t0; t < t1 && t < t0 + kCluStages; ++t) {
      const int tok0 = t * kTile, col = tok0 / p.block_size;
      const int blk = col < 32 ? __shfl_sync(0xffffffffu, my_blk, col) : bt_row[col];
      if (lane < 4 && tok0 + kTile <= len && blk >= 0 && blk < p.num_blocks)
        tma_prefetch_l2_3d(lane < 2 ? &map_k : &map_v, (lane & 1) * 64, h, blk * p.block_size + (tok0 - col * p.block_size));
    }
    asm volatile("griddepcontrol.wait;" ::: "memory");   // from here on: query rows and the cache
    if (lane == 0) {
      mbar_expect_tx(&bar_q, G * 256);
      bulk_load_1d(s_q, p.q + seq * p.q_row_stride + static_cast<long long>(h) * G * 128, G * 256, &bar_q);
    }
    for (int t = t0; t < t1; ++t) {
      const int it = t - t0, stage = it % kCluStages;
      const int tok0 = t * kTile, col = tok0 / p.block_size;
      const int blk = col < 32 ? __shfl_sync(0xffffffffu, my_blk, col) : bt_row[col];
      if (it >= kCluStages && !mbar_wait(&bar_empty[stage], ((it / kCluStages) & 1) ^ 1, abort_flag)) {
        if (lane == 0) atomicExch(&g_status_decode_cluster, 1);
        return;
      }
      __syncwarp();
      if (lane == 0) {
        int slot0 = -kTile;  // out-of-range block id: the box lies outside the tensor and reads zeros
        if (blk >= 0 && blk < p.num_blocks) slot0 = blk * p.block_size + (tok0 - col * p.block_size);
        const int nslab = dec_tile_slabs(len - tok0);
        if (kStore) s_slot0[stage] = slot0;
        mbar_expect_tx(&bar_full[stage], dec_tile_bytes(nslab));
        dec_load_tile(stages + stage * kStageBytes, &bar_full[stage], &map_k, &map_v, &map_k16, &map_v16, h, slot0, nslab);
      }
    }
    return;
  }

  // ============================= consumer warps =============================
  bool ok = true;
  uint32_t qa[8][4];
  DecAcc acc;
  acc.reset();
  // One warp's slab of a tile is a chain of some 1400 cycles, and with one CTA per SM nothing else runs there: a second
  // group of warps on every other tile halves the time of a long sequence (16/8 heads, 8192 tokens: 17.3 -> 14.2 us with the producer kernel in front).
  const int group = warp >> 2, slab = warp & 3;
  for (int it = group; it < t1 - t0; it += 2) {
    const int stage = it % kCluStages;
    if (!mbar_wait(&bar_full[stage], (it / kCluStages) & 1, abort_flag)) { ok = false; break; }
    if (it < 2) {
      if (!mbar_wait(&bar_q, 0, abort_flag)) { ok = false; break; }
      dec_query_fragments(s_q, G, lane, qa);
    }
    const int valid = len - ((t0 + it) * kTile + slab * 16);
    if (kStore && valid > 0) {
      // rows of this slab that the step replaces
      const int first = s_slot0[stage] + slab * 16;
#pragma unroll
      for (int u = 0; u < kCluSlots; ++u) {
        const int row = slots[u] - first;
        unsigned hits = __ballot_sync(0xffffffffu, slots[u] >= 0 && row >= 0 && row < 16 && row < valid);
        while (hits) {
          const int l = __ffs(hits) - 1;
          hits &= hits - 1;
          const int r = slab * 16 + __shfl_sync(0xffffffffu, row, l), tok = u * 32 + l, c = lane & 15;
          const uint4 w = tok == seq ? own : step_chunk(p, tok, h, lane);
          *reinterpret_cast<uint4*>(stages + stage * kStageBytes + (lane < 16 ? 0 : 2 * kSubTileBytes) + (c >> 3) * kSubTileBytes +
                                    r * 128 + (((c & 7) ^ (r & 7)) << 4)) = w;
          fence_proxy_async_smem();          // (a later load writes over it)
        }
      }
      __syncwarp();
    }
    if (valid > 0) dec_tile(stages + stage * kStageBytes, slab, lane, valid, p.scale_log2, qa, acc);
    __syncwarp();
    if (lane == 0) mbar_arrive(&bar_empty[stage]);
  }
  ok = __all_sync(0xffffffffu, ok);
  if (ok) {
    dec_hand_off(acc, merge_o + warp * G * 128, merge_ml + warp * G * 2, G, lane);
    __syncwarp();
    if (lane == 0) mbar_arrive(&bar_merge);
    ok = __all_sync(0xffffffffu, mbar_wait(&bar_merge, 0, abort_flag));
  }
  __nv_bfloat16* out_row = p.out + (static_cast<long long>(seq) * p.H + h * G) * 128;
  if (ok && active == 1) {
    for (int gq = warp; gq < G; gq += kCluWarps)
      dec_store_row(out_row + gq * 128, dec_combine_warps<kCluWarps>(merge_o, merge_ml, G, gq, lane), lane);
    return;
  }
  cluster_wait();                         // rank 0's inbox barrier is initialised (all threads arrived at the start)
  if (ok) {
    // Push: warp w combines the warps' states of head w and sends them to rank 0.
    for (int gq = warp; gq < G; gq += kCluWarps) {
      const DecPart r = dec_combine_warps<kCluWarps>(merge_o, merge_ml, G, gq, lane);
      cluster_store(cluster_addr(smem_u32(inbox_o + (rank * G + gq) * 128 + lane * 4), 0), r.v);
      if (lane == 0) cluster_store(cluster_addr(smem_u32(inbox_ml + (rank * G + gq) * 2), 0), r.M, r.L);
    }
    __syncwarp();
    if (lane == 0) cluster_mbar_arrive(cluster_addr(smem_u32(&bar_inbox), 0));
  }
  if (rank == 0 && ok) ok = __all_sync(0xffffffffu, cluster_mbar_wait(&bar_inbox, 0));
  if (!ok) {
    // A wait gave up: report it, and leave only when every other CTA of the cluster has (an exited thread counts as
    // arrived), so that no late push finds this CTA's shared memory gone.
    if (lane == 0) atomicExch(&g_status_decode_cluster, 1);
    cluster_arrive();
    cluster_wait();
    return;
  }
  if (rank != 0) return;
  for (int gq = warp; gq < G; gq += kCluWarps) {
    float M = -INFINITY;
    for (int r = 0; r < ctas; ++r) {
      if ((r * nt + ctas - 1) / ctas == ((r + 1) * nt + ctas - 1) / ctas) continue;     // that rank had no tile
      M = fmaxf(M, inbox_ml[(r * G + gq) * 2]);
    }
    DecPart a;
    a.M = M;
    a.L = 0.f;
    a.v = make_float4(0.f, 0.f, 0.f, 0.f);
    for (int r = 0; r < ctas; ++r) {
      if ((r * nt + ctas - 1) / ctas == ((r + 1) * nt + ctas - 1) / ctas) continue;
      const float w = fast_exp2(inbox_ml[(r * G + gq) * 2] - M);
      const float4 v = *reinterpret_cast<const float4*>(inbox_o + (r * G + gq) * 128 + lane * 4);
      a.L += inbox_ml[(r * G + gq) * 2 + 1] * w;
      a.v.x += v.x * w; a.v.y += v.y * w; a.v.z += v.z * w; a.v.w += v.w * w;
    }
    dec_store_row(out_row + gq * 128, a, lane);
  }
}

int read_status_decode_cluster() {
  int v = 0;
  cudaMemcpyFromSymbol(&v, g_status_decode_cluster, sizeof(int));
  return v;
}

int reset_state_decode_cluster() {
  const int zero = 0;
  return check_cuda(cudaMemcpyToSymbol(g_status_decode_cluster, &zero, sizeof(int)), "device_status: clearing the decode status word");
}

static size_t cluster_smem_bytes(int G, int ctas) {
  return 1024 + static_cast<size_t>(kCluStages) * kStageBytes + static_cast<size_t>(G) * 256 +
         static_cast<size_t>(kCluWarps + ctas) * G * 130 * 4;
}

// CTAs per (sequence, kv head), or 0: leave the batch to the general kernel.  What is known on the host is the number of pairs
// and the width of the block table, not the lengths.
//
// Size: the largest of which all pairs are on the chip at once, a second round costs as much as the first.  How many are is the
// runtime's answer for this kernel (one CTA per SM; what a GPC has left over stays idle): 15 clusters of 8, 33 of 4, 74 of 2
// on a B200.  Us per layer of a decode graph with the producer in front, one kv head: 13 sequences of 50 .. 2000 tokens on clusters
// of 8 | 4 7.8 | 8.9, 16 of them 12.5 | 9.1; 33 of 562 on 4 | 2 7.3 | 7.7, 34 of them 11.8 | 7.7; 74 of 562 on 2 | 1
// 9.5 | 9.1, 75 of them 15.3 | 9.2.  (More than 8 CTAs: of clusters of 16 only a few fit.)
//
// Table: a pair's CTAs must be able to bear the longest pair that it allows, which the general kernel cuts as it needs.  Both
// sides as above, this kernel | the general one, at the line and beyond it, tables filled evenly from 50 tokens on; one
// sequence filling the table among ones of 200; and sequences of 562 (200) tokens under it, which is what the line costs:
//   clusters of 8, 128 tiles   9 sequences 13.0 | 12.6; 13.0 | 11.1; 6.3 | 8.3      (64 tiles 9.3 | 10.5; 9.0 | 9.5; 6.3 | 8.3)
//   clusters of 4, 64 tiles   24 sequences 12.7 | 11.8; 12.6 | 9.8; 7.0 | 9.0       (48 tiles 10.8 | 11.2; 10.5 | 9.6; 7.0 | 8.9)
//   clusters of 2, 20 tiles   50 sequences 10.1 | 10.6; 9.8 | 9.2; 8.0 | 9.9        (32 tiles 12.8 | 11.8; 12.7 | 9.1; 8.0 | 9.9)
//   lone CTAs, 16 tiles      110 sequences 12.0 | 12.9; 11.8 | 10.0; 6.4 | 7.8      (75 sequences 11.9 | 10.9; 11.6 | 9.7; 6.5 | 7.6)
// 16/8 heads, filled evenly: clusters of 2, 32 tiles, 5 sequences 12.1 | 10.9, 9 14.2 | 13.4; lone CTAs, 16 tiles, 12 sequences
// 11.3 | 11.9, 18 13.2 | 13.8.  So the line lies where tables that are filled stop gaining; clusters of 4 and 8 go beyond that, to
// the 16 columns of 256 tokens under which an engine of 4096 tokens runs all its batches, short ones for the most part.
constexpr int kCluSizes = 4;                            // of 8, 4, 2 and 1 CTAs
constexpr int kCluMaxTiles[kCluSizes] = {128, 64, 20, 16};
int decode_cluster_rule(long long pairs, int G, int max_tiles, const int* on_chip) {
  if (G > kCluMaxG) return 0;
  for (int i = 0; i < kCluSizes; ++i) {
    const int c = 8 >> i;
    if (pairs <= on_chip[i] && c * G <= 32 && c / 2 < max_tiles) return max_tiles <= kCluMaxTiles[i] ? c : 0;
  }
  return 0;
}

// Leave for the largest launch there is.
static int cluster_configure(bool store) {
  static std::atomic<size_t> configured[2][kMaxDevices];
  auto* const kernel = store ? decode_cluster_kernel<true> : decode_cluster_kernel<false>;
  return ensure_dynamic_smem(reinterpret_cast<const void*>(kernel), cluster_smem_bytes(kCluMaxG, 8), configured[store],
                             "decode_attn(cluster): cudaFuncSetAttribute");
}

// How many clusters of 8 >> i CTAs the current device holds at a time (0: not known).
static int clusters_on_chip(int i) {
  static std::atomic<int> known[kMaxDevices][kCluSizes];
  int dev = 0, n = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) return 0;
  if ((n = known[dev][i].load(std::memory_order_acquire)) > 0) return n;
  if (cluster_configure(false)) return 0;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(8u >> i);
  cfg.blockDim = dim3(kCluThreads);
  cfg.dynamicSmemBytes = cluster_smem_bytes(kCluMaxG, 8);  // (one CTA per SM with any number of heads)
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 8u >> i;
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  if (cudaOccupancyMaxActiveClusters(&n, decode_cluster_kernel<false>, &cfg) != cudaSuccess) {
    cudaGetLastError();
    return 0;
  }
  known[dev][i].store(n, std::memory_order_release);
  return n;
}

int decode_cluster_ctas(int batch, int Hkv, int G, int max_tiles) {
  const long long pairs = static_cast<long long>(batch) * Hkv;
  if (G > kCluMaxG || pairs > sm_count()) return 0;
  int on_chip[kCluSizes];
  for (int i = 0; i < kCluSizes; ++i) on_chip[i] = clusters_on_chip(i);
  return decode_cluster_rule(pairs, G, max_tiles, on_chip);
}

int launch_decode_cluster(const DecodeParams& p, const CUtensorMap& map_k, const CUtensorMap& map_v, const CUtensorMap& map_k16,
                          const CUtensorMap& map_v16, int ctas_per_pair, cudaStream_t stream) {
  auto* const kernel = p.st_slots ? decode_cluster_kernel<true> : decode_cluster_kernel<false>;
  const int rc = cluster_configure(p.st_slots != nullptr);
  if (rc) return rc;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(static_cast<unsigned>(p.batch * p.Hkv * ctas_per_pair));
  cfg.blockDim = dim3(kCluThreads);
  cfg.dynamicSmemBytes = cluster_smem_bytes(p.G, ctas_per_pair);
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = static_cast<unsigned>(ctas_per_pair);
  attr[1].val.clusterDim.y = attr[1].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 2;
  const cudaError_t le = cudaLaunchKernelEx(&cfg, kernel, p, map_k, map_v, map_k16, map_v16, ctas_per_pair);
  g_launches.fetch_add(1);
  return check_cuda(le != cudaSuccess ? le : cudaGetLastError(), "decode_attn(cluster) launch");
}

}  // namespace b200
