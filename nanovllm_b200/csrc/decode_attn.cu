// Paged single-token decode attention (replaces flash_attn_with_kvcache as called at
// nanovllm/layers/attention.py:71-74).
//
// HBM-bound: every K and V byte of every context token is read exactly once.  Design:
//  * Work unit = one (sequence, kv head) pair, whole, or, where the batch's longest pair is well above a CTA's equal share
//    of the tiles (the rule and its lines stand where the units are laid out), one of the equal parts it is cut into.  Persistent CTAs (2 per SM) take the units longest first: the
//    first ones statically, the others through an atomic ticket, so that CTAs that stream faster take more and the
//    short units level the end.  Order and cuts are derived on the device from context_lens by every CTA alike: the
//    launch geometry never depends on device data, as CUDA-graph replay requires.  (Equal static pieces of
//    one flat tile list, the earlier form, cut nearly every pair of a batch of a few hundred pairs and paid for it
//    with partials at the end of the launch; whole pairs in HBM order also stream faster: 176 -> 164 us on 256
//    sequences of 100 .. 2048 tokens, 16/8 heads, 7.0 TB/s.)  Batches with few pairs go to decode_cluster.cu.
//  * The producer warp (one elected lane) walks the CTA's units.  For every unit it publishes a descriptor in shared
//    memory, bulk-copies the G query rows into a small ring, and issues the TMA tile loads (64 tokens: two 64x64
//    boxes for K, two for V, 128-byte swizzle; 16-token boxes for the ragged last tile of a sequence) into a
//    ring of stages guarded by full/empty mbarriers.  The descriptor and the query rows ride on the full-barrier of the
//    unit's first tile, and the next unit and its metadata are fetched one unit ahead, so the ring never drains at
//    unit boundaries.
//  * Four consumer warps take 16 tokens of each tile: QK^T and PV on mma.sync.m16n8k16 (the G
//    query heads of the kv head are rows of the 16-row A operand), online softmax in fp32 with
//    quad shuffles.  At the end of a unit they only drop their running (m, l, O) into shared
//    memory and go on with the next tile; the CTA's last unit they finish themselves.
//  * An epilogue warp combines the four warps' states and writes the bf16 row, or, for a part of a cut pair, a
//    partial (m, l, unnormalised O) to the workspace; the last part to arrive (one atomic counter per pair, reset by
//    that warp) merges the partials in the order of the parts.  No CTA ever waits for another; every mbarrier wait is bounded.
#include "../../include/b200_attn.h"
#include "decode_common.cuh"

namespace b200 {
extern std::atomic<long long> g_launches;

constexpr int kDecStages = 3;
// Tiles that a CTA's first unit has on their way into L2 ahead of the wait (at most 8), while the kernel in front ends and the
// memory is idle: as many as the ring has stages, or, from kDecAheadShare tiles per CTA on, five.  Us per layer of a graph with the
// producer in front, by tiles per CTA, at 3 | 5 tiles:
//   4.4   90 of 20 .. 400 tokens, 8/4 heads      12.9 | 13.4      10.5  200 of 30 .. 900, 4/2          23.3 | 23.2
//   4.8   256 of 50 .. 600, 2/1                  14.2 | 14.8      12.3  400 of 100 .. 1000, 4/1        27.0 | 26.0
//   6.2   200 of 30 .. 500, 4/2                  15.9 | 16.7      12.5  50 of 100 .. 1024, 16/8        24.2 | 24.4
//   7.3   400 of 30 .. 600, 4/1                  18.0 | 18.9      14.9  256 of 100 .. 2048, 2/1        28.9 | 28.5
//   8.4   200 of 30 .. 700, 4/2                  18.9 | 19.3      15.8  512 of 100 .. 1000, 4/1        30.3 | 29.2
//   9.4   400 of 30 .. 800, 4/1                  23.5 | 23.0      11.8  12 of 300 .. 9000, 16/4        26.5 | 26.1
// (6.0, 90 of 500 .. 700, 4/2: 15.4 | 14.9).  Six and eight: the same as five within 0.3 us except 37 of 100 .. 1024, 16/8, at 8
// (19.1, 20.0) and the last (25.8).  Blocks of 512 and 1024 tokens give the same picture.
constexpr int kDecAhead = 5, kDecAheadShare = 9;
constexpr int kDecProducerWarp = kDecConsumerWarps;
constexpr int kDecEpilogueWarp = kDecConsumerWarps + 1;
constexpr int kDecThreads = kDecConsumers + 64;
constexpr int kDecWarps = kDecThreads / 32;
constexpr int kDecMaxBatch = 512;               // per launch; the host splits larger batches
constexpr int kDecPer = (kDecMaxBatch + kDecThreads - 1) / kDecThreads;
constexpr int kWsStatusBytes = 256;  // header: word 0 is the ticket counter of the scheduler
constexpr int kWsCounterInts = kDecMaxBatch * 128;   // arrival counters: fixed region, up to 128 kv heads
constexpr int kUnitRing = kDecStages + 1;  // unit descriptors / query rows in flight
constexpr int kDecPending = 8;             // partials written but not yet counted, per CTA
constexpr int kDecClasses = 64;            // length classes of the sort
constexpr int kSortRows = kDecPer * kDecWarps;
constexpr int kDecMinPart = 4;             // tiles: shorter parts would cost more to merge than to stream
// Sequences up to which the cache store rides in the launch (its slots take the place of the other tables' upper halves).  Beyond,
// going through the slots for every last tile costs what the launch of its own does: eager layer, 128 sequences of 100 .. 2048
// (16/8 heads) 90.2 -> 87.6 us, 160: 110.6 -> 109.9, 200: 135.3 -> 137.0.
constexpr int kDecStoreBatch = 160;
constexpr int kBloomWords = 64, kBloomBits = 11;  // (256 bytes: what static shared memory has left of its 1 KiB)
constexpr int kDecOneWaveShare = 12;       // tiles per CTA up to which parts get a CTA each (measured where it is used)
constexpr int kPartialSlots = 12;          // of the workspace, per CTA of the grid
static __device__ int g_status_decode = 0;

// One unit as the producer hands it to the other warps.
struct UnitDesc {
  int seq, h;
  int t0, t1;            // tiles [t0, t1) of the pair
  int len;               // context length, clamped to the block table's capacity
  int parts;             // parts the pair is cut into (1: whole)
  int part0, slot;       // workspace slots of the pair's first part and of this one (consecutive parts: Hkv apart)
};

// The units of a launch, the same in every CTA.  Chunk x of [0, chunks) in order of length is part (x - base[r]) of the
// r-th longest sequence; unit u is kv head u % Hkv of chunk u / Hkv.
struct DecUnits {
  const unsigned short *order, *base, *nt;   // shared memory: sequences by length, first chunk of each, tiles by sequence
  const unsigned char* tail;                 // tokens of a sequence's last tile - 1
  int cap;                                   // tiles a part may have
  int live;                                  // sequences with tokens
  int ahead;                                 // tiles of a CTA's first unit to fetch ahead of the wait
  bool split, wide;                          // some pair is cut; some tile count does not fit 16 bits
  __device__ __forceinline__ UnitDesc get(const DecodeParams& p, int u) const {
    UnitDesc d;
    const int x = u / p.Hkv;
    d.h = u - x * p.Hkv;
    int r = x, part = 0;
    if (split) {
      int lo = 0, hi = live;
      while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (base[mid] <= x) lo = mid; else hi = mid;
      }
      r = lo;
      part = x - base[r];
    }
    d.seq = order[r];
    int n = nt[d.seq];
    d.len = (n - 1) * kTile + tail[d.seq] + 1;
    if (wide) {
      d.len = min(p.context_lens[d.seq], p.bt_cols * p.block_size);
      n = (d.len + kTile - 1) / kTile;
    }
    d.parts = split ? (n + cap - 1) / cap : 1;
    d.t0 = split ? static_cast<int>(static_cast<long long>(part) * n / d.parts) : 0;
    d.t1 = split ? static_cast<int>(static_cast<long long>(part + 1) * n / d.parts) : n;
    d.slot = u;
    d.part0 = u - part * p.Hkv;
    return d;
  }
};

__device__ __forceinline__ int ld_acquire_gpu(const int* ptr) {
  int v;
  asm volatile("ld.acquire.gpu.global.s32 %0, [%1];" : "=r"(v) : "l"(ptr) : "memory");
  return v;
}

// Merges the n partials of a pair (query head gq) into r.  `own` >= 0: that part is not in the workspace but in r.  Eight
// partials a trip, their maxima and sums together with their rows, always in the order of the parts: whichever CTA
// merges, and from where, depends on timing, so the sums must not.
__device__ __forceinline__ void dec_merge_partials(const DecodeParams& p, int part0, int n, int own, int gq, int lane, DecPart& r) {
  const DecPart mine = r;
  r = dec_nothing();
#pragma unroll 1
  for (int first = 0; first < n; first += 8) {
    // lane j (mod 8) looks after partial first + j
    const int j = first + (lane & 7);
    const int row = (part0 + (j < n ? j : n - 1) * p.Hkv) * p.G + gq;
    float2 ml = make_float2(mine.M, mine.L);
    if (j != own) ml = __ldcg(reinterpret_cast<const float2*>(p.ws_ml + row * 2));
    float4 v[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      const int ru = __shfl_sync(0xffffffffu, row, u);
      v[u] = mine.v;
      if (first + u < n && first + u != own) v[u] = __ldcg(reinterpret_cast<const float4*>(p.ws_o + static_cast<long long>(ru) * 128 + lane * 4));
    }
    if (j >= n) ml = make_float2(-INFINITY, 0.f);
    float M = ml.x;
#pragma unroll
    for (int off = 4; off > 0; off >>= 1) M = fmaxf(M, __shfl_xor_sync(0xffffffffu, M, off));
    M = fmaxf(M, r.M);
    const float w = fast_exp2(ml.x - M), w0 = fast_exp2(r.M - M);
    float L = __fmul_rn(ml.y, w);
#pragma unroll
    for (int off = 4; off > 0; off >>= 1) L += __shfl_xor_sync(0xffffffffu, L, off);
    r.M = M;
    // (written out: the function is expanded in three places, which must not contract products and sums differently)
    r.L = fmaf(r.L, w0, L);
    r.v.x = __fmul_rn(r.v.x, w0); r.v.y = __fmul_rn(r.v.y, w0); r.v.z = __fmul_rn(r.v.z, w0); r.v.w = __fmul_rn(r.v.w, w0);
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      const float wu = __shfl_sync(0xffffffffu, w, u);
      if (first + u < n) {
        r.v.x = fmaf(v[u].x, wu, r.v.x); r.v.y = fmaf(v[u].y, wu, r.v.y);
        r.v.z = fmaf(v[u].z, wu, r.v.z); r.v.w = fmaf(v[u].w, wu, r.v.w);
      }
    }
  }
}

// L2 prefetch of the full tiles among [t0, t1), at most eight, which lie in the blocks of table columns col0 and col0 + 1: a box
// (half of the K or V rows' columns) per lane.
__device__ __forceinline__ void dec_prefetch_tiles(const DecodeParams& p, const CUtensorMap& map_k, const CUtensorMap& map_v, int h,
                                                   int t0, int t1, int len, int lane, int col0, int blk0, int blk1) {
  const int t = t0 + (lane >> 2), tok0 = t * kTile, col = tok0 / p.block_size;
  const int blk = col == col0 ? blk0 : col == col0 + 1 ? blk1 : -1;
  if (t >= t1 || tok0 + kTile > len || blk < 0 || blk >= p.num_blocks) return;
  tma_prefetch_l2_3d(lane & 2 ? &map_v : &map_k, (lane & 1) * 64, h, static_cast<int>(blk * static_cast<long long>(p.block_size)) + (tok0 - col * p.block_size));
}

__device__ __forceinline__ void dec_store_partial(const DecodeParams& p, int slot, int gq, int lane, const DecPart& r) {
  *reinterpret_cast<float4*>(p.ws_o + (static_cast<long long>(slot) * p.G + gq) * 128 + lane * 4) = r.v;
  if (lane == 0) *reinterpret_cast<float2*>(p.ws_ml + (slot * p.G + gq) * 2) = make_float2(r.M, r.L);
}

// kStore: the step's cache store in the same launch, as in decode_cluster.cu: nobody relies on finding another CTA's row in
// the cache.  The epilogue warps write the step's rows, and whoever loads a tile that covers any slot of the step puts the
// new rows into its copy.  Which tiles may do so every CTA knows from a small Bloom filter over the slots' tiles; only for
// those do the consumer warps go through the slots (eager layer, 37 sequences of 100 .. 1024, 16/8 heads: 19.9 -> 17.1 us).
__device__ __forceinline__ uint32_t dec_bloom_a(int slot) { return (slot >> 6) & (kBloomWords * 32 - 1); }
__device__ __forceinline__ uint32_t dec_bloom_b(int slot) { return (static_cast<uint32_t>(slot >> 6) * 2654435761u) >> (32 - kBloomBits); }

// The step's rows among this warp's 16 rows of the tile that starts at slot0.
__device__ __forceinline__ void dec_patch_rows(const DecodeParams& p, const int* s_slots, unsigned char* stage, int warp, int lane,
                                               int slot0, int h) {
  bool any = false;
  for (int i0 = 0; i0 < p.batch; i0 += 32) {
    const int slot = i0 + lane < p.batch ? s_slots[i0 + lane] : -1;
    const int row = slot - slot0 - warp * 16;
    unsigned found = __ballot_sync(0xffffffffu, slot >= 0 && row >= 0 && row < 16);
    while (found) {
      const int src = __ffs(found) - 1;
      found &= found - 1;
      const int r = warp * 16 + __shfl_sync(0xffffffffu, row, src), c = lane & 15;
      *reinterpret_cast<uint4*>(stage + (lane < 16 ? 0 : 2 * kSubTileBytes) + (c >> 3) * kSubTileBytes + r * 128 +
                                (((c & 7) ^ (r & 7)) << 4)) = step_chunk(p, i0 + src, h, lane);
      any = true;
    }
  }
  if (any) {
    fence_proxy_async_smem();
    __syncwarp();
  }
}

template <bool kStore>
__global__ void __launch_bounds__(kDecThreads, 2)
decode_attn_kernel(const DecodeParams p, const __grid_constant__ CUtensorMap map_k,
                   const __grid_constant__ CUtensorMap map_v, const __grid_constant__ CUtensorMap map_k16,
                   const __grid_constant__ CUtensorMap map_v16) {
  extern __shared__ __align__(1024) unsigned char smem[];
  const int G = p.G, Hkv = p.Hkv;
  unsigned char* stages = smem;
  __nv_bfloat16* s_q = reinterpret_cast<__nv_bfloat16*>(smem + kDecStages * kStageBytes);          // [kUnitRing][G][128]
  float* merge_o = reinterpret_cast<float*>(s_q + kUnitRing * G * 128);                           // [n_merge][4][G][128]
  float* merge_ml = merge_o + p.n_merge * kDecConsumerWarps * G * 128;                              // [n_merge][4][G][2]
  unsigned short* s_order = reinterpret_cast<unsigned short*>(merge_ml + p.n_merge * kDecConsumerWarps * G * 2);
  constexpr int kMaxBatch = kStore ? kDecStoreBatch : kDecMaxBatch;
  unsigned short* s_base = s_order + kMaxBatch;
  unsigned short* s_nt = s_base + kMaxBatch;
  unsigned char* s_tail = reinterpret_cast<unsigned char*>(s_nt + kMaxBatch);
  int* s_slots = reinterpret_cast<int*>(s_tail + kMaxBatch);                 // kStore: [batch], -1 where nothing is stored
  __shared__ __align__(8) uint64_t bar_full[kDecStages];
  __shared__ __align__(8) uint64_t bar_empty[kDecStages];
  __shared__ __align__(8) uint64_t bar_merge_full[2];
  __shared__ __align__(8) uint64_t bar_merge_empty[2];
  __shared__ __align__(8) uint64_t bar_decide, bar_part, bar_final;
  __shared__ __align__(16) UnitDesc s_desc[kUnitRing];
  __shared__ __align__(16) UnitDesc s_merge_desc[2];
  __shared__ __align__(16) UnitDesc s_pending[kDecPending];
  __shared__ int s_parts[kDecWarps];
  __shared__ uint32_t s_bloom[kStore ? kBloomWords : 1];
  __shared__ int s_patch[kStore ? kDecStages : 1];       // a stage's first slot, or -1: no row of the step in it
  __shared__ int s_warp_sums[kDecWarps], s_warp_max[kDecWarps], s_warp_live[kDecWarps];
  __shared__ int s_abort, s_known, s_last, s_decision, s_merge_all;

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int max_len = p.bt_cols * p.block_size;

  if (tid == 0) {
    s_abort = 0;
    s_known = 0;
    s_last = -1;
    mbar_init(&bar_decide, 1);
    mbar_init(&bar_part, kDecConsumerWarps);
    mbar_init(&bar_final, 1);
    for (int s = 0; s < kDecStages; ++s) {
      mbar_init(&bar_full[s], 1);
      mbar_init(&bar_empty[s], kDecConsumerWarps);
    }
    for (int s = 0; s < 2; ++s) {
      mbar_init(&bar_merge_full[s], kDecConsumerWarps);
      mbar_init(&bar_merge_empty[s], 1);
    }
    mbar_fence_init();
  }

  // Launched with programmatic stream serialization: the kernel may start while the previous kernel
  // of the stream is still running, if that kernel allows it (griddepcontrol.launch_dependents; of this library
  // the store, producer, decode and mma.sync prefill kernels do; any other kernel has completed before this one
  // starts).  Those kernels write K/V rows of the cache, query and key rows and outputs, never the metadata, so
  // the scan over context_lens, the first block-table reads and (kStore) the slots below run ahead;
  // every thread that goes on to touch q, the cache, the output or the workspace first executes
  // griddepcontrol.wait (the consumer warps only touch them after data that was loaded behind it).

  // ---- the units of the launch: lengths -> parts -> order ----
  DecUnits un;
  un.order = s_order;
  un.base = s_base;
  un.nt = s_nt;
  un.tail = s_tail;
  int units;
  {
    // scratch of the sort, in the stage memory that no load has been issued into yet: sequences per (round, warp) and class
    uint32_t* const s_cnt = reinterpret_cast<uint32_t*>(stages);                    // [kSortRows][kDecClasses / 2], two a word
    unsigned short* const cnt = reinterpret_cast<unsigned short*>(s_cnt);
    for (int i = tid; i < kSortRows * kDecClasses / 2; i += kDecThreads) s_cnt[i] = 0;
    const int per = (p.batch + kDecThreads - 1) / kDecThreads;
    const int i0 = tid * per;
    int local[kDecPer];
    int sum = 0, longest = 0, live = 0;
    if (kStore && tid < kBloomWords) s_bloom[tid] = 0;
#pragma unroll
    for (int k = 0; k < kDecPer; ++k) {
      int nt = 0;
      const int i = i0 + k;
      if (k < per && i < p.batch) {
        int len = p.context_lens[i];
        len = len < 0 ? 0 : (len > max_len ? max_len : len);
        nt = (len + kTile - 1) / kTile;
        s_nt[i] = static_cast<unsigned short>(nt < 65535 ? nt : 65535);
        s_tail[i] = static_cast<unsigned char>((len - 1) & (kTile - 1));
      }
      local[k] = nt;
      sum += nt;
      longest = max(longest, nt);
      live += nt > 0;
    }
    sum = __reduce_add_sync(0xffffffffu, sum);
    longest = __reduce_max_sync(0xffffffffu, longest);
    live = __reduce_add_sync(0xffffffffu, live);
    if (lane == 0) { s_warp_sums[warp] = sum; s_warp_max[warp] = longest; s_warp_live[warp] = live; }
    __syncthreads();
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    if constexpr (kStore) {
      for (int i = tid; i < p.batch; i += kDecThreads) {
        const int slot = __ldg(p.st_slots + i);
        const bool stored = slot >= 0 && slot < p.st_n_slots;
        s_slots[i] = stored ? slot : -1;
        if (!stored) continue;
        atomicOr(&s_bloom[dec_bloom_a(slot) >> 5], 1u << (dec_bloom_a(slot) & 31));
        atomicOr(&s_bloom[dec_bloom_b(slot) >> 5], 1u << (dec_bloom_b(slot) & 31));
      }
    }
    long long total = 0;
    longest = live = 0;
#pragma unroll
    for (int w = 0; w < kDecWarps; ++w) {
      total += s_warp_sums[w];
      longest = max(longest, s_warp_max[w]);
      live += s_warp_live[w];
    }
    // Pairs are cut only if the longest one is well above a CTA's equal share of the tiles: whole pairs, longest first,
    // level out well enough below that and leave nothing to merge.  The line is 1.25 shares, or 1.85 where
    // every CTA has at most one pair (short and long ones share an SM then, and the long one, which ends the launch, goes
    // faster when the others are done: a tile takes a CTA 1.38 us while all 296 stream and 0.57 us, its chain, on its own; us per layer with the producer, whole | cut, at 1.46 shares 25.7 | 27.2, 1.73 20.3 | 22.4, 1.93
    // 26.7 | 26.6, with 32 tiles a share 59.0 | 54.0, 2.05 19.4 | 20.5, 2.3 25.2 | 23.2, 2.9 49.3 | 39.1), and 3 tiles, which is what a merge costs (90 sequences of 20 .. 400 tokens, 4 kv heads:
    // 14.6 -> 11.5 us uncut).  Above it, pairs longer than 2/3 of a share (and kDecMinPart tiles) are cut into
    // equal parts: 1/2 and 1/3 leave parts of a size that do not add up to a share, and cost more merges (measured over
    // batches of 16 .. 500 sequences of 1 .. 8192 tokens).  The parts come first in the order, so that their merging
    // happens while the whole pairs stream.  A part is longer than a third of a share, so there are at most
    // 3 x grid of them: the workspace's kPartialSlots x grid slots hold every partial.
    // With fewer pairs than CTAs and a small share, the parts are instead as short as they can be with a CTA for
    // each, 1 .. 1.5 shares: no CTA starts a second unit, and there are half as many partials.  5 sequences of 47 ..
    // 4381 tokens, 8 kv heads: 21.1 -> 14.2 us; 20 of 500 .. 1500, 4 kv heads: 17.7 -> 13.2; 128 of 30 .. 600, 2 kv heads: 16.3 ->
    // 12.4.  From kDecOneWaveShare on, levelling through the tickets is as good or better unless the longest pair is far above
    // a share (us per layer with the producer, a CTA for each | through tickets: 4.7 tiles a share 14.8 | 17.6, 9.4
    // 22.4 | 24.2, 11 24.2 | 24.5, 14.7 30.2 | 29.7, 20.7 38.1 | 38.0, 29.5 52.0 | 50.3; 14.9 with the longest at 9 shares 29.5 | 31.9).
    const long long tiles = total * Hkv;
    const int grid = static_cast<int>(gridDim.x);
    const bool one_wave = live * Hkv <= grid;
    un.cap = longest;
    if (static_cast<long long>(longest) * grid * 100 > (one_wave ? 185 : 125) * tiles && (longest - 3ll) * grid > tiles) {
      const long long part = 2 * tiles / (3 * grid) + 1;
      un.cap = static_cast<int>(part < kDecMinPart ? kDecMinPart : part < longest ? part : longest);
      if (one_wave && tiles <= kDecOneWaveShare * grid && longest < 65535) {       // (the same in every thread)
        const int share = static_cast<int>((tiles + grid - 1) / grid);
        // each warp counts the parts for one length
        const int step = (share + 9) / 10, cap = max(kDecMinPart, share + warp * step);
        int n = 0;
        for (int i = lane; i < p.batch; i += 32) n += (s_nt[i] + cap - 1) / cap;
        n = __reduce_add_sync(0xffffffffu, n);
        if (lane == 0) s_parts[warp] = n;
        __syncthreads();
#pragma unroll
        for (int w = kDecWarps - 1; w >= 0; --w)
          if (s_parts[w] * Hkv <= grid) un.cap = min(longest, max(kDecMinPart, share + w * step));
      }
    }
    un.live = live;
    un.ahead = tiles < static_cast<long long>(kDecAheadShare) * grid ? kDecStages : kDecAhead;
    un.split = longest > un.cap;
    un.wide = longest >= 65535;
    // size classes: without cuts all 64 for the whole pairs, else 32 for the parts and, behind them, 32 for the whole pairs
    const int top = un.split ? un.cap : longest, classes = un.split ? kDecClasses / 2 : kDecClasses;
    // Longest first: a stable counting sort by length class (longest -> class 0).  Every CTA must arrive at
    // the same order, so places within a class follow from (round, warp, lane), not from who comes first.
    int cls[kDecPer], pos[kDecPer];
#pragma unroll
    for (int k = 0; k < kDecPer; ++k) {
      cls[k] = -1;
      if (local[k] > 0) {
        const int parts = (local[k] + un.cap - 1) / un.cap;
        const int part = parts == 1 ? local[k] : (local[k] + parts - 1) / parts;
        cls[k] = static_cast<int>(static_cast<unsigned>(top - part) * (classes - 1) / static_cast<unsigned>(top));
        if (un.split && parts == 1) cls[k] += classes;
      }
      const unsigned same = __match_any_sync(0xffffffffu, cls[k]);
      pos[k] = __popc(same & ((1u << lane) - 1));
      if (pos[k] == 0 && cls[k] >= 0) cnt[(k * kDecWarps + warp) * kDecClasses + cls[k]] = static_cast<unsigned short>(__popc(same));
    }
    __syncthreads();
    if (warp == 0) {
      // lane owns classes 2 * lane and 2 * lane + 1 (the halves of a word; no sum exceeds kDecMaxBatch)
      uint32_t v[kSortRows], sum2 = 0;
#pragma unroll
      for (int r = 0; r < kSortRows; ++r) v[r] = s_cnt[r * (kDecClasses / 2) + lane];
#pragma unroll
      for (int r = 0; r < kSortRows; ++r) sum2 += v[r];
      const uint32_t both = (sum2 & 0xffff) + (sum2 >> 16);
      uint32_t in = both;
#pragma unroll
      for (int off = 1; off < 32; off <<= 1) {
        const uint32_t x = __shfl_up_sync(0xffffffffu, in, off);
        if (lane >= off) in += x;
      }
      uint32_t at = (in - both) | ((in - (sum2 >> 16)) << 16);        // first place of either class
#pragma unroll
      for (int r = 0; r < kSortRows; ++r) {
        s_cnt[r * (kDecClasses / 2) + lane] = at;
        at += v[r];
      }
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < kDecPer; ++k)
      if (cls[k] >= 0) s_order[cnt[(k * kDecWarps + warp) * kDecClasses + cls[k]] + pos[k]] = static_cast<unsigned short>(i0 + k);
    units = live * Hkv;
    if (un.split) {
      // first chunk of every sequence, in that order
      __syncthreads();
      int parts[kDecPer], mine = 0;
#pragma unroll
      for (int k = 0; k < kDecPer; ++k) {
        parts[k] = 0;
        if (k < per && i0 + k < live) {
          int n = s_nt[s_order[i0 + k]];
          if (un.wide) n = (min(p.context_lens[s_order[i0 + k]], max_len) + kTile - 1) / kTile;
          parts[k] = (n + un.cap - 1) / un.cap;
        }
        mine += parts[k];
      }
      int incl = mine;
#pragma unroll
      for (int off = 1; off < 32; off <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, incl, off);
        if (lane >= off) incl += v;
      }
      if (lane == 31) s_warp_live[warp] = incl;     // (its first use is two barriers back)
      __syncthreads();
      int at = incl - mine, chunks = 0;
#pragma unroll
      for (int w = 0; w < kDecWarps; ++w) {
        if (w < warp) at += s_warp_live[w];
        chunks += s_warp_live[w];
      }
#pragma unroll
      for (int k = 0; k < kDecPer; ++k) {
        if (k < per && i0 + k < live) s_base[i0 + k] = static_cast<unsigned short>(at);
        at += parts[k];
      }
      units = chunks * Hkv;
    }
    fence_proxy_async_smem();                        // the loads write over the scratch
    __syncthreads();
  }

  // ---- sequences with no context produce zeros (the epilogue warp's job, before anything else) ----
  if (warp == kDecEpilogueWarp) {
    asm volatile("griddepcontrol.wait;" ::: "memory");
    for (int i = blockIdx.x; i < p.batch; i += gridDim.x) {
      if (s_nt[i] == 0) {
        uint4* o = reinterpret_cast<uint4*>(p.out + static_cast<long long>(i) * p.H * 128);
        for (int v = lane; v < p.H * 16; v += 32) o[v] = make_uint4(0, 0, 0, 0);
      }
    }
    if constexpr (kStore) {
      for (int i = blockIdx.x; i < p.batch; i += gridDim.x) {
        const long long slot = s_slots[i];
        if (slot < 0) continue;
#pragma unroll 4
        for (int h = 0; h < Hkv; ++h)
          *reinterpret_cast<uint4*>((lane < 16 ? p.st_k_cache : p.st_v_cache) + (slot * Hkv + h) * 128 + (lane & 15) * 8) =
              step_chunk(p, i, h, lane);
      }
    }
  }

  const int cta = blockIdx.x;
  const int n_first = min(units, static_cast<int>(gridDim.x));     // units handed out statically, one per CTA
  if (cta >= n_first) return;
  const int n_drawn = units - n_first;                             // units handed out through tickets
  volatile int* abort_flag = &s_abort;

  if (warp == kDecProducerWarp) {
    // =========================== producer warp ===========================
    if (lane == 0) {
      tma_prefetch_desc(&map_k);
      tma_prefetch_desc(&map_v);
      tma_prefetch_desc(&map_k16);
      tma_prefetch_desc(&map_v16);
    }
    int it = 0, n_unit = 0;
    bool ok = true;
    // The SM's second CTA (ids from the SM count on) counts from the short end, so that long and short units share an SM.
    const int half = gridDim.x / 2;
    UnitDesc cur = un.get(p, cta < half ? cta : n_first - 1 - (cta - half));
    // the unit's first two block ids, fetched one unit ahead
    const int* cur_bt = p.block_tables + cur.seq * p.bt_row_stride;
    int cur_col0 = (cur.t0 * kTile) / p.block_size;
    int cur_blk0 = cur_bt[cur_col0];
    int cur_blk1 = cur_col0 + 1 < p.bt_cols ? cur_bt[cur_col0 + 1] : -1;
    // Bring the first tiles into L2 while the kernel in front still runs: nothing is read, so it does not matter
    // that that kernel may be writing this step's rows.
    dec_prefetch_tiles(p, map_k, map_v, cur.h, cur.t0, min(cur.t1, cur.t0 + un.ahead), cur.len, lane, cur_col0, cur_blk0, cur_blk1);
    if (lane != 0) return;
    asm volatile("griddepcontrol.wait;" ::: "memory");   // from here on: query rows and the cache
    while (true) {
      const int last_col = (cur.len - 1) / p.block_size;
      int col_now = cur_col0;
      long long blk_now = cur_blk0;
      long long blk_next = cur_col0 < last_col ? cur_blk1 : -1;
      UnitDesc nxt;
      bool more = false;
      int nxt_col0 = 0, nxt_blk0 = -1, nxt_blk1 = -1;
      const int* nxt_bt = nullptr;
      for (int t = cur.t0; t < cur.t1; ++t, ++it) {
        const int stage = it % kDecStages;
        const uint32_t ph = (it / kDecStages) & 1;
        if (!mbar_wait(&bar_empty[stage], ph ^ 1, abort_flag)) { ok = false; break; }
        const int tok0 = t * kTile;
        const int col = tok0 / p.block_size;
        if (col != col_now) {
          col_now = col;
          blk_now = blk_next;
          blk_next = col_now < last_col ? cur_bt[col_now + 1] : -1;
        }
        int slot0 = -kTile;  // out-of-range block id: the box lies outside the tensor and reads zeros
        if (blk_now >= 0 && blk_now < p.num_blocks)
          slot0 = static_cast<int>(blk_now * p.block_size + (tok0 - col * p.block_size));
        const int nslab = dec_tile_slabs(cur.len - tok0);
        const bool first = t == cur.t0;
        // descriptor and query rows travel with the unit's first tile
        if (first) s_desc[n_unit % kUnitRing] = cur;
        if constexpr (kStore) {
          const uint32_t a = dec_bloom_a(slot0), b = dec_bloom_b(slot0);
          s_patch[stage] = slot0 >= 0 && ((s_bloom[a >> 5] >> (a & 31)) & (s_bloom[b >> 5] >> (b & 31)) & 1) ? slot0 : -1;
        }
        mbar_expect_tx(&bar_full[stage], dec_tile_bytes(nslab) + (first ? G * 256 : 0));
        if (first)
          bulk_load_1d(s_q + (n_unit % kUnitRing) * G * 128,
                       p.q + cur.seq * p.q_row_stride + static_cast<long long>(cur.h) * G * 128, G * 256, &bar_full[stage]);
        dec_load_tile(stages + stage * kStageBytes, &bar_full[stage], &map_k, &map_v, &map_k16, &map_v16, cur.h, slot0, nslab);
        if (first) {
          // With this unit under way, find the next one and start fetching its metadata: a ticket.  Each CTA
          // draws until it fails, so exactly n_drawn + n_first tickets are drawn per launch (none if n_drawn is 0); whoever
          // draws the last one resets the counter.
          unsigned int tk = 0;
          if (n_drawn > 0) {
            tk = atomicAdd(p.ticket, 1u);
            if (tk == static_cast<unsigned int>(units - 1)) atomicExch(p.ticket, 0u);
            more = tk < static_cast<unsigned int>(n_drawn);
          }
          if (!more) {
            *const_cast<volatile int*>(&s_last) = n_unit;
            __threadfence_block();
          }
          *const_cast<volatile int*>(&s_known) = n_unit + 1;     // whether anything follows this unit is settled
          if (more) {
            nxt = un.get(p, n_first + static_cast<int>(tk));
            nxt_bt = p.block_tables + nxt.seq * p.bt_row_stride;
            nxt_col0 = (nxt.t0 * kTile) / p.block_size;
            nxt_blk0 = nxt_bt[nxt_col0];
            nxt_blk1 = nxt_col0 + 1 < p.bt_cols ? nxt_bt[nxt_col0 + 1] : -1;
          }
        }
      }
      if (!ok) break;
      ++n_unit;
      if (!more) break;
      cur = nxt;
      cur_bt = nxt_bt;
      cur_col0 = nxt_col0;
      cur_blk0 = nxt_blk0;
      cur_blk1 = nxt_blk1;
    }
    if (!ok) atomicExch(&g_status_decode, 1);
    return;
  }

  if (warp == kDecEpilogueWarp) {
    // =========================== epilogue warp ===========================
    // Lane owns 4 of the 128 output dims.  Step 1 for every unit: combine the four consumer
    // warps' states and store the row (or the partial) -- no waiting on global memory, so the
    // consumers get their hand-off buffer back at once.  The slow part of a partial (fence, arrival
    // counter, merge: several dependent trips to L2) is queued and flushed when no hand-off is
    // waiting; one fence and one round of atomics then serve every queued partial.
    int n_pending = 0;
    auto flush = [&]() {
      if (n_pending == 0) return;
      __threadfence();
      __syncwarp();
      bool last = false;
      if (lane < n_pending) {
        const UnitDesc& d = s_pending[lane];
        last = atomicAdd(&p.counters[d.seq * Hkv + d.h], 1) == d.parts - 1;
      }
      const unsigned last_mask = __ballot_sync(0xffffffffu, last);
      if (last_mask) __threadfence();
      for (int k = 0; k < n_pending; ++k) {
        if (!((last_mask >> k) & 1u)) continue;
        // this CTA brought the last partial of pair k: merge them all
        const UnitDesc d = s_pending[k];
#pragma unroll 1
        for (int gq = 0; gq < G; ++gq) {
          DecPart r = dec_nothing();
          dec_merge_partials(p, d.part0, d.parts, -1, gq, lane, r);
          dec_store_row(p.out + (static_cast<long long>(d.seq) * p.H + d.h * G + gq) * 128, r, lane);
        }
        if (lane == 0) p.counters[d.seq * Hkv + d.h] = 0;
      }
      __syncwarp();
      n_pending = 0;
    };
    // (flush() is expanded in one place only: it is large, and three copies cost the kernel registers)
    bool finished = false, flush_now = false;
    for (int n = 0;;) {
      const int e = n % p.n_merge;
      const uint32_t ph = (n / p.n_merge) & 1;
      bool is_last = __shfl_sync(0xffffffffu, *const_cast<volatile int*>(&s_last), 0) == n;
      const bool ready = __all_sync(0xffffffffu, !finished && !flush_now && !is_last && mbar_try_wait(&bar_merge_full[e], ph));
      flush_now = false;
      if (!ready) {
        flush();                                     // nothing to combine right now: do the slow part
        if (finished) break;
        if (!is_last && !mbar_wait(&bar_merge_full[e], ph, abort_flag)) break;
      }
      // (settled by now: the consumers hand a unit over only when it is known what follows it)
      is_last = is_last || __shfl_sync(0xffffffffu, *const_cast<volatile int*>(&s_last), 0) == n;
      if (is_last) {
        const UnitDesc d = s_desc[n % kUnitRing];
        // The CTA's last unit: nothing is left to hide the trips to L2 behind, so all warps finish it together.
        // If it is a part and the pair's other parts have all arrived (looked up while the consumers still stream), the
        // row is finished from this CTA's own state and their partials, without a partial of its own.
        const bool whole = d.parts == 1;
        int* counter = &p.counters[d.seq * Hkv + d.h];
        bool arrived = whole, handed = false;
        const long long c0 = clock64();
        for (int look = 0; !arrived && !handed; ++look) {
          if ((look & 31) == 0) arrived = ld_acquire_gpu(counter) == d.parts - 1;
          handed = mbar_test_wait(&bar_merge_full[e], ph);
          if (*abort_flag || clock64() - c0 > kSpinLimitCycles) break;
        }
        arrived = __shfl_sync(0xffffffffu, arrived, 0);
        if (lane == 0) {
          s_decision = whole ? 0 : arrived ? 1 : 2;
          mbar_arrive(&bar_decide);
          if (arrived && !whole) *counter = 0;
        }
        if (!arrived) {
          if (!mbar_wait(&bar_part, 0, abort_flag)) break;
          if (lane == 0) {
            __threadfence();
            const bool merge = atomicAdd(counter, 1) == d.parts - 1;
            if (merge) { __threadfence(); *counter = 0; }
            s_merge_all = merge;
            mbar_arrive(&bar_final);
          }
        }
        finished = true;
        continue;
      }
      const UnitDesc d = s_merge_desc[e];
      const float* mo = merge_o + e * kDecConsumerWarps * G * 128;
      const float* ml = merge_ml + e * kDecConsumerWarps * G * 2;
      for (int gq = 0; gq < G; ++gq) {
        const DecPart r = dec_combine_warps(mo, ml, G, gq, lane);
        if (d.parts == 1)
          dec_store_row(p.out + (static_cast<long long>(d.seq) * p.H + d.h * G + gq) * 128, r, lane);
        else
          dec_store_partial(p, d.slot, gq, lane, r);
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(&bar_merge_empty[e]);   // the consumers may refill the hand-off buffer
      ++n;
      if (d.parts > 1) {
        if (lane == 0) s_pending[n_pending] = d;
        __syncwarp();
        if (++n_pending == kDecPending) flush_now = true;   // a full queue is flushed at the top of the loop
      }
    }
    return;
  }

  // ============================= consumer warps =============================
  int it = 0;
  bool ok = true;
  for (int n_unit = 0; ok; ++n_unit) {
    // ---- a new unit: its descriptor and query rows arrive with its first tile ----
    if (!mbar_wait(&bar_full[it % kDecStages], (it / kDecStages) & 1, abort_flag)) { ok = false; break; }
    const UnitDesc d = s_desc[n_unit % kUnitRing];
    uint32_t qa[8][4];   // query fragments: rows = the G heads sharing the kv head
    dec_query_fragments(s_q + (n_unit % kUnitRing) * G * 128, G, lane, qa);
    DecAcc acc;
    acc.reset();
    for (int t = d.t0; t < d.t1; ++t, ++it) {
      const int stage = it % kDecStages;
      const uint32_t ph = (it / kDecStages) & 1;
      if (t != d.t0 && !mbar_wait(&bar_full[stage], ph, abort_flag)) { ok = false; break; }
      const int valid = d.len - (t * kTile + warp * 16);  // valid tokens in this warp's 16-token slab
      if constexpr (kStore) {
        const int slot0 = s_patch[stage];
        if (slot0 >= 0 && valid > 0) dec_patch_rows(p, s_slots, stages + stage * kStageBytes, warp, lane, slot0, d.h);
      }
      if (valid > 0) dec_tile(stages + stage * kStageBytes, warp, lane, valid, p.scale_log2, qa, acc);
      __syncwarp();
      if (lane == 0) mbar_arrive(&bar_empty[stage]);
    }
    if (!ok) break;

    // ---- hand the warp's running state to the epilogue warp and move on ----
    const int e = n_unit % p.n_merge;
    const uint32_t ph = (n_unit / p.n_merge) & 1;
    if (!mbar_wait(&bar_merge_empty[e], ph ^ 1, abort_flag)) { ok = false; break; }
    dec_hand_off(acc, merge_o + (e * kDecConsumerWarps + warp) * G * 128, merge_ml + (e * kDecConsumerWarps + warp) * G * 2, G, lane);
    {
      const long long c0 = clock64();
      while (*const_cast<volatile int*>(&s_known) <= n_unit) {
        if (*abort_flag || clock64() - c0 > kSpinLimitCycles) { *abort_flag = 1; ok = false; break; }
      }
      __threadfence_block();
    }
    ok = __all_sync(0xffffffffu, ok);
    if (!ok) break;
    const bool is_last = *const_cast<volatile int*>(&s_last) == n_unit;
    if (tid == 0) s_merge_desc[e] = d;
    __syncwarp();
    if (lane == 0) mbar_arrive(&bar_merge_full[e]);
    if (is_last) {
      // finished by all warps together: warp w takes query heads w, w + 4, ..
      if (!mbar_wait(&bar_merge_full[e], ph, abort_flag) || !mbar_wait(&bar_decide, 0, abort_flag)) { ok = false; break; }
      const int decision = *const_cast<volatile int*>(&s_decision);
      const float* mo = merge_o + e * kDecConsumerWarps * G * 128;
      const float* ml = merge_ml + e * kDecConsumerWarps * G * 2;
      __nv_bfloat16* out_row = p.out + (static_cast<long long>(d.seq) * p.H + d.h * G) * 128;
#pragma unroll 1
      for (int gq = warp; gq < G; gq += kDecConsumerWarps) {
        DecPart r = dec_combine_warps(mo, ml, G, gq, lane);
        if (decision == 2) {
          dec_store_partial(p, d.slot, gq, lane, r);
        } else {
          if (decision == 1) dec_merge_partials(p, d.part0, d.parts, (d.slot - d.part0) / Hkv, gq, lane, r);
          dec_store_row(out_row + gq * 128, r, lane);
        }
      }
      if (decision == 2) {
        __syncwarp();
        if (lane == 0) mbar_arrive(&bar_part);
        if (!mbar_wait(&bar_final, 0, abort_flag)) { ok = false; break; }
        if (*const_cast<volatile int*>(&s_merge_all)) {
          // this CTA brought the last partial
#pragma unroll 1
          for (int gq = warp; gq < G; gq += kDecConsumerWarps) {
            DecPart r = dec_nothing();
            dec_merge_partials(p, d.part0, d.parts, -1, gq, lane, r);
            dec_store_row(out_row + gq * 128, r, lane);
          }
        }
      }
      return;
    }
  }
  if (lane == 0) atomicExch(&g_status_decode, 1);
}

int read_status_decode() {
  int v = 0;
  cudaMemcpyFromSymbol(&v, g_status_decode, sizeof(int));
  return v;
}

// Only the status word lives in the library; the ticket and arrival counters of an abandoned launch
// are in the caller's workspace, which the caller has to zero-fill again.
int reset_state_decode() {
  const int zero = 0;
  return check_cuda(cudaMemcpyToSymbol(g_status_decode, &zero, sizeof(int)), "device_status: clearing the decode status word");
}

// Two hand-off buffers between consumers and the epilogue warp when two CTAs still fit on an SM with them.
static int decode_merge_buffers(int G) { return G <= 2 ? 2 : 1; }

static size_t decode_smem_bytes(int G) {
  return static_cast<size_t>(kDecStages) * kStageBytes + static_cast<size_t>(kUnitRing) * G * 256 +
         static_cast<size_t>(decode_merge_buffers(G)) * kDecConsumerWarps * G * 130 * 4 + kDecMaxBatch * 7;
}

static int decode_grid() { return 2 * sm_count(); }

static long long decode_partial_slots(int grid) { return static_cast<long long>(kPartialSlots) * grid; }
static long long decode_partial_bytes(int grid, int G) { return decode_partial_slots(grid) * G * 130 * 4; }
static long long decode_ws_bytes(int grid, int G) {
  return kWsStatusBytes + static_cast<long long>(kWsCounterInts) * 4 + decode_partial_bytes(grid, G);
}

}  // namespace b200

extern "C" int64_t b200_decode_workspace_bytes(int32_t max_batch, int32_t num_heads, int32_t num_kv_heads,
                                               int32_t head_dim) {
  using namespace b200;
  if (max_batch <= 0 || num_heads <= 0 || num_kv_heads <= 0 || num_heads % num_kv_heads || head_dim != 128)
    return set_error(kErrBadShape, "decode_workspace_bytes: bad geometry (batch=%d H=%d Hkv=%d D=%d)", max_batch,
                     num_heads, num_kv_heads, head_dim);
  const int grid = decode_grid();
  if (grid <= 0) return set_error(kErrNoDriver, "decode_workspace_bytes: no CUDA device");
  if (num_kv_heads > 128 || num_heads / num_kv_heads > kMaxG)
    return set_error(kErrBadShape, "decode_workspace_bytes: at most 128 kv heads and %d query heads per kv head", kMaxG);
  return decode_ws_bytes(grid, num_heads / num_kv_heads);
}

namespace b200 {

struct DecodeStore {
  const int* slots;
  const void *k, *v;
  long long k_stride, v_stride;   // elements
};

// `store` != nullptr: row i of k and v also goes to slot store->slots[i] of the caches first.
static int decode(const void* q, int64_t q_row_stride, const void* k_cache, const void* v_cache,
                                int64_t num_blocks, int32_t block_size, const int32_t* block_tables,
                                int64_t bt_row_stride, int32_t bt_cols, const int32_t* context_lens, void* out,
                                void* workspace, int64_t workspace_bytes, int32_t batch, int32_t num_heads,
                                int32_t num_kv_heads, int32_t head_dim, float scale, void* stream, const DecodeStore* store) {
  if (batch < 0) return set_error(kErrBadShape, "decode_attn: negative batch");
  if (batch == 0) return kOk;
  if (!q || !k_cache || !v_cache || !block_tables || !context_lens || !out)
    return set_error(kErrNullPointer, "decode_attn: null pointer argument");
  if (head_dim != 128) return set_error(kErrBadShape, "decode_attn: head_dim must be 128 (got %d)", head_dim);
  if (num_heads <= 0 || num_kv_heads <= 0 || num_heads % num_kv_heads)
    return set_error(kErrBadShape, "decode_attn: num_heads (%d) must be a positive multiple of num_kv_heads (%d)",
                     num_heads, num_kv_heads);
  const int G = num_heads / num_kv_heads;
  if (G > kMaxG) return set_error(kErrBadShape, "decode_attn: at most %d query heads per kv head (got %d)", kMaxG, G);
  if (num_kv_heads > 128) return set_error(kErrBadShape, "decode_attn: at most 128 kv heads (got %d)", num_kv_heads);
  if (block_size <= 0 || block_size % 256)
    return set_error(kErrBadShape, "decode_attn: block_size must be a positive multiple of 256 (got %d)", block_size);
  if (num_blocks <= 0 || num_blocks * block_size >= (1LL << 31))
    return set_error(kErrBadShape, "decode_attn: num_blocks * block_size must be in (0, 2^31)");
  if (bt_cols <= 0 || bt_row_stride < bt_cols || static_cast<long long>(bt_cols) * block_size >= (1LL << 30))
    return set_error(kErrBadShape, "decode_attn: bad block table geometry (cols=%d stride=%lld)", bt_cols,
                     (long long)bt_row_stride);
  if (q_row_stride < static_cast<long long>(num_heads) * 128 || q_row_stride % 8)
    return set_error(kErrMisaligned, "decode_attn: q_row_stride must be >= H*128 and a multiple of 8 elements");
  if ((reinterpret_cast<uintptr_t>(q) | reinterpret_cast<uintptr_t>(k_cache) | reinterpret_cast<uintptr_t>(v_cache) |
       reinterpret_cast<uintptr_t>(out)) & 15)
    return set_error(kErrMisaligned, "decode_attn: q, caches and out must be 16-byte aligned");
  const int grid = decode_grid();
  if (grid <= 0) return set_error(kErrNoDriver, "decode_attn: no CUDA device");
  const long long need = decode_ws_bytes(grid, G);
  if (!workspace || workspace_bytes < need || (reinterpret_cast<uintptr_t>(workspace) & 15))
    return set_error(kErrWorkspace, "decode_attn: workspace of %lld bytes (16-byte aligned, zero-filled once) required, got %lld",
                     need, (long long)workspace_bytes);

  CUtensorMap map_k, map_v;
  int rc = make_tokens_heads_map(&map_k, k_cache, static_cast<uint64_t>(num_blocks) * block_size, num_kv_heads,
                                 static_cast<uint64_t>(num_kv_heads) * 128, kTile);
  if (rc) return rc;
  rc = make_tokens_heads_map(&map_v, v_cache, static_cast<uint64_t>(num_blocks) * block_size, num_kv_heads,
                             static_cast<uint64_t>(num_kv_heads) * 128, kTile);
  if (rc) return rc;
  CUtensorMap map_k16, map_v16;   // 16-token boxes for the ragged last tile of a sequence
  rc = make_tokens_heads_map(&map_k16, k_cache, static_cast<uint64_t>(num_blocks) * block_size, num_kv_heads,
                             static_cast<uint64_t>(num_kv_heads) * 128, 16);
  if (rc) return rc;
  rc = make_tokens_heads_map(&map_v16, v_cache, static_cast<uint64_t>(num_blocks) * block_size, num_kv_heads,
                             static_cast<uint64_t>(num_kv_heads) * 128, 16);
  if (rc) return rc;

  const size_t smem = decode_smem_bytes(G);
  static std::atomic<size_t> configured[2][kMaxDevices];

  unsigned char* ws = static_cast<unsigned char*>(workspace);
  DecodeParams p;
  p.bt_row_stride = bt_row_stride;
  p.bt_cols = bt_cols;
  p.H = num_heads;
  p.Hkv = num_kv_heads;
  p.G = G;
  p.block_size = block_size;
  p.num_blocks = num_blocks;
  p.scale_log2 = scale * 1.4426950408889634f;
  p.n_merge = decode_merge_buffers(G);
  p.ticket = reinterpret_cast<unsigned int*>(ws);
  p.counters = reinterpret_cast<int*>(ws + kWsStatusBytes);
  p.ws_o = reinterpret_cast<float*>(ws + kWsStatusBytes + static_cast<long long>(kWsCounterInts) * 4);
  p.ws_ml = p.ws_o + decode_partial_slots(grid) * G * 128;
  p.q_row_stride = q_row_stride;
  for (int b0 = 0; b0 < batch; b0 += kDecMaxBatch) {
    p.batch = batch - b0 < kDecMaxBatch ? batch - b0 : kDecMaxBatch;
    p.q = static_cast<const __nv_bfloat16*>(q) + b0 * q_row_stride;
    p.out = static_cast<__nv_bfloat16*>(out) + static_cast<long long>(b0) * num_heads * 128;
    p.context_lens = context_lens + b0;
    p.block_tables = block_tables + b0 * bt_row_stride;
    p.st_slots = nullptr;
    const int ctas = decode_cluster_ctas(p.batch, num_kv_heads, G, static_cast<int>(static_cast<long long>(bt_cols) * block_size / kTile));
    if (store && (ctas || batch <= kDecStoreBatch) && p.batch == batch) {
      p.st_slots = store->slots;
      p.st_k = static_cast<const __nv_bfloat16*>(store->k);
      p.st_v = static_cast<const __nv_bfloat16*>(store->v);
      p.st_k_stride = store->k_stride;
      p.st_v_stride = store->v_stride;
      p.st_n_slots = num_blocks * block_size;
      p.st_k_cache = static_cast<__nv_bfloat16*>(const_cast<void*>(k_cache));
      p.st_v_cache = static_cast<__nv_bfloat16*>(const_cast<void*>(v_cache));
    } else if (store && b0 == 0) {
      rc = b200_store_kvcache(store->k, store->v, store->k_stride, store->v_stride, const_cast<void*>(k_cache),
                              const_cast<void*>(v_cache), store->slots, batch, num_kv_heads * 128, 2, num_blocks * block_size, stream);
      if (rc) return rc;
    }
    if (ctas) {
      rc = launch_decode_cluster(p, map_k, map_v, map_k16, map_v16, ctas, static_cast<cudaStream_t>(stream));
      if (rc) return rc;
      continue;
    }
    auto* const kernel = p.st_slots ? decode_attn_kernel<true> : decode_attn_kernel<false>;
    rc = ensure_dynamic_smem(reinterpret_cast<const void*>(kernel), smem, configured[p.st_slots != nullptr], "decode_attn: cudaFuncSetAttribute");
    if (rc) return rc;
    const cudaError_t le = launch_early(kernel, grid, kDecThreads, smem, static_cast<cudaStream_t>(stream), p, map_k, map_v, map_k16, map_v16);
    g_launches.fetch_add(1);
    rc = check_cuda(le != cudaSuccess ? le : cudaGetLastError(), "decode_attn launch");
    if (rc) return rc;
  }
  return kOk;
}

}  // namespace b200

extern "C" int b200_decode_attn(const void* q, int64_t q_row_stride, const void* k_cache, const void* v_cache,
                                int64_t num_blocks, int32_t block_size, const int32_t* block_tables,
                                int64_t bt_row_stride, int32_t bt_cols, const int32_t* context_lens, void* out,
                                void* workspace, int64_t workspace_bytes, int32_t batch, int32_t num_heads,
                                int32_t num_kv_heads, int32_t head_dim, float scale, void* stream) {
  return b200::decode(q, q_row_stride, k_cache, v_cache, num_blocks, block_size, block_tables, bt_row_stride, bt_cols, context_lens, out,
                      workspace, workspace_bytes, batch, num_heads, num_kv_heads, head_dim, scale, stream, nullptr);
}

extern "C" int b200_store_decode_attn(const void* q, int64_t q_row_stride, const void* k, const void* v, int64_t k_row_stride,
                                      int64_t v_row_stride, const int32_t* slot_mapping, void* k_cache, void* v_cache,
                                      int64_t num_blocks, int32_t block_size, const int32_t* block_tables,
                                      int64_t bt_row_stride, int32_t bt_cols, const int32_t* context_lens, void* out,
                                      void* workspace, int64_t workspace_bytes, int32_t batch, int32_t num_heads,
                                      int32_t num_kv_heads, int32_t head_dim, float scale, void* stream) {
  using namespace b200;
  if (batch > 0) {
    if (!k || !v || !slot_mapping) return set_error(kErrNullPointer, "store_decode_attn: null k, v or slot_mapping");
    const int64_t row = static_cast<int64_t>(num_kv_heads) * head_dim;
    if (k_row_stride < row || v_row_stride < row || k_row_stride % 8 || v_row_stride % 8 ||
        ((reinterpret_cast<uintptr_t>(k) | reinterpret_cast<uintptr_t>(v)) & 15))
      return set_error(kErrMisaligned, "store_decode_attn: k and v must be 16-byte aligned, their row strides >= Hkv*128 and multiples of 8 elements");
  }
  const DecodeStore store = {slot_mapping, k, v, k_row_stride, v_row_stride};
  return decode(q, q_row_stride, k_cache, v_cache, num_blocks, block_size, block_tables, bt_row_stride, bt_cols, context_lens, out,
                workspace, workspace_bytes, batch, num_heads, num_kv_heads, head_dim, scale, stream, &store);
}

// ---------------------------------------------------------------------------------------------
// Decode attention for callers that cannot allocate device memory.
//
// Some hosts of this library have nowhere to get a workspace from: a serving engine that has
// already handed every free byte of the GPU to its KV cache (nano-vllm sizes the cache from the
// free memory it finds, so a later cudaMalloc can fail), a plugin slot whose contract forbids
// allocation inside the call, or code that runs where the framework's caching allocator must not
// be touched.  For them the scratch of the decode kernel lives in the library image itself: a
// file-scope __device__ array that every GPU loading the library holds until the process exits.
// ---------------------------------------------------------------------------------------------
namespace b200 {

constexpr int kStaticMaxGridTimesG = 320 * 4;   // persistent CTAs x query heads per kv head the scratch has room for
constexpr long long kStaticScratchBytes =
    kWsStatusBytes + static_cast<long long>(kWsCounterInts) * 4 + static_cast<long long>(kPartialSlots) * kStaticMaxGridTimesG * 130 * 4;

static __device__ __align__(256) unsigned char g_decode_static_scratch[kStaticScratchBytes];

// Device address of the array above on the current device.  In host code the array's name is only a
// handle for the runtime, never an address a kernel may be given, so the address is asked for
// once per device (with that device current) and remembered.
static int static_scratch_address(void** out) {
  static void* cached[64];
  static std::atomic<int> ready[64];
  int dev = 0;
  int rc = check_cuda(cudaGetDevice(&dev), "decode_attn_static: cudaGetDevice");
  if (rc) return rc;
  if (dev < 0 || dev >= 64) return set_error(kErrDevice, "decode_attn_static: device ordinal %d not supported", dev);
  if (!ready[dev].load(std::memory_order_acquire)) {
    void* ptr = nullptr;
    rc = check_cuda(cudaGetSymbolAddress(&ptr, g_decode_static_scratch), "decode_attn_static: cudaGetSymbolAddress");
    if (rc) return rc;
    if (!ptr) return set_error(kErrDevice, "decode_attn_static: the scratch array has no address on device %d", dev);
    cached[dev] = ptr;
    ready[dev].store(1, std::memory_order_release);
  }
  *out = cached[dev];
  return kOk;
}

}  // namespace b200

extern "C" int64_t b200_decode_static_scratch_bytes(void) { return b200::kStaticScratchBytes; }

extern "C" int b200_decode_attn_static(const void* q, int64_t q_row_stride, const void* k_cache, const void* v_cache,
                                       int64_t num_blocks, int32_t block_size, const int32_t* block_tables,
                                       int64_t bt_row_stride, int32_t bt_cols, const int32_t* context_lens, void* out,
                                       int32_t batch, int32_t num_heads, int32_t num_kv_heads, int32_t head_dim,
                                       float scale, void* stream) {
  using namespace b200;
  if (batch < 0) return set_error(kErrBadShape, "decode_attn_static: negative batch");
  if (batch == 0) return kOk;
  if (num_heads <= 0 || num_kv_heads <= 0 || num_heads % num_kv_heads)
    return set_error(kErrBadShape, "decode_attn_static: num_heads (%d) must be a positive multiple of num_kv_heads (%d)",
                     num_heads, num_kv_heads);
  const int grid = decode_grid();
  if (grid <= 0) return set_error(kErrNoDriver, "decode_attn_static: no CUDA device");
  const int G = num_heads / num_kv_heads;
  if (static_cast<long long>(grid) * G > kStaticMaxGridTimesG || num_kv_heads > 128)
    return set_error(kErrWorkspace,
                     "decode_attn_static: %d persistent CTAs x %d query heads per kv head exceeds the built-in scratch's "
                     "limit of %d (and kv heads must be <= 128); use b200_decode_attn with a caller-owned workspace",
                     grid, G, kStaticMaxGridTimesG);
  void* scratch = nullptr;
  int rc = static_scratch_address(&scratch);
  if (rc) return rc;
  // The array keeps whatever the previous call left.  Partials are always written before they are
  // read; the ticket counter and the arrival counters are what must start at zero, so clear them here.
  const long long per_launch = batch < kDecMaxBatch ? batch : kDecMaxBatch;
  rc = check_cuda(cudaMemsetAsync(scratch, 0, kWsStatusBytes + static_cast<size_t>(per_launch) * num_kv_heads * 4,
                                  static_cast<cudaStream_t>(stream)),
                  "decode_attn_static: clearing the counters");
  if (rc) return rc;
  return b200_decode_attn(q, q_row_stride, k_cache, v_cache, num_blocks, block_size, block_tables, bt_row_stride, bt_cols,
                          context_lens, out, scratch, kStaticScratchBytes, batch, num_heads, num_kv_heads, head_dim,
                          scale, stream);
}
