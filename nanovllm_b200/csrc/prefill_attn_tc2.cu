// Varlen causal prefill attention, tcgen05 / TMEM, persistent and ping-ponged: the fast path.
// Replaces flash_attn_varlen_func as called at nanovllm/layers/attention.py:64-70, for dense K/V
// and for K/V read from the paged cache.
//
// One persistent CTA per SM.  A work item is (sequence, kv head, block of 2 * QT query tokens),
// QT = 128 / G, handed out through an atomic ticket counter from the longest sequence down (t2_order), and
// within a sequence from its last, longest query block.  The two
// halves of the block ("A" = first QT tokens, "B" = next QT) are two independent 128-row tiles that
// share every K/V tile, so K/V traffic per query row is halved and, more to the point, the tensor
// core always has the other half's MMA to run while one half is in its softmax (launches with few items: kSplit below):
//   warp 0        TMA producer: draws tickets, publishes item descriptors, loads Q_A / Q_B and
//                 feeds two-deep rings of 128-token K tiles and V tiles;
//   warp 1        one elected thread issues tcgen05.mma:  S_X = Q_X K^T  (M128 N128 K16 x 8) and
//                 O_X += P_X V  (A operand = P read from TMEM, B = V as MN-major shared memory);
//   warps 4-7     softmax warpgroup of half A: thread r owns TMEM lane r = one query row; reads S
//                 with tcgen05.ld, keeps max / sum in registers, writes P (bf16) over S with
//                 tcgen05.st, rescales O in TMEM only when the row max grew by more than 2^8;
//   warps 8-11    the same for half B;
//   warps 12-15   output warpgroup: takes a finished O out of TMEM, scales it by 1 / row sum and
//                 sends it out as bf16 through TMA stores (plain stores where a box would overhang
//                 the sequence), so the softmax warpgroups never stop for output.
//   warps 2-3     send the step's K and V tiles on to the paged cache where the call asks for it (t2_store_tile);
//   (setmaxnreg: warpgroup 0 -> 80, softmax -> 184, output -> 64 registers.)
// TMEM: S_A [0,128)  S_B [128,256)  O_A [256,384)  O_B [384,512).  Every mbarrier wait is bounded.
#include "../../include/b200_attn.h"
#include "kernels.cuh"
#include "tcgen05.cuh"

#include <type_traits>

namespace b200 {
extern std::atomic<long long> g_launches;

constexpr int kT2Kv = 128;
constexpr int kT2Sub = 128 * 128;            // one 64-column sub-tile of a 128-row tile (bytes)
constexpr int kT2Tile = 2 * kT2Sub;          // 128 rows x 128 dims bf16 = 32 KiB
constexpr int kT2Threads = 512;   // warpgroup 0: TMA producer, MMA issuer, two store warps (idle without the store); 1, 2: softmax; 3: output
constexpr int kT2Ring = 2;                   // K ring depth and V ring depth
constexpr int kT2Items = 4;                  // item descriptors in flight
constexpr int kT2MaxSeqSmem = 1024;          // sequences whose slot table fits in shared memory
// Sequences that are put in order of length: two threads each, so one round of the block.  Larger batches keep their own order.  What
// that costs, from batches of up to 256 measured both ways (sorted | the order of a shuffled batch): 64 of 100 .. 1024 tokens
// 34.7 | 41.6 us at 2/1 heads, 158 | 162 at 16/8; 256 of them 644 | 692 and, at 32/8, 1323 | 1319; 256 of 10 .. 120 at 2/1
// heads 20.7 | 18.3 (the sort itself takes 2.4 us).  With more than 256 prompts in a step an SM has several items of any
// length anyway.
constexpr int kT2MaxSort = kT2Threads / 2;
constexpr float kT2Rescale = 8.0f;

static __device__ int g_status_prefill_tc2 = 0;

static __device__ unsigned int g_prefill_ticket = 0;

// The kernel's bounded waits.  Six roles run through their loops at the same time and share the SM's instruction cache, so code
// size is time here.  Us for 256 prompts of 100 .. 1024 tokens with the store | without it, 256 of 10 .. 300 without it, in four launches
// after a rest (in 300 launches on end, at the power cap):
//   mbar_wait() (64-bit clock arithmetic and a spin counter at each of some thirty places), output and rescaling
//     loops unrolled, a mask by comparisons                                 803 | 657, 167  (885 | 766, 185)
//   these waits, those loops rolled, the mask from bits of one word         702 | 609, 146  (823 | 725, 170)
//   one output path instead of two, shifts for divisions by powers of two, table columns counted along and one copy
//     of the store's row loop: 64 KB of code for 78 with the store          653 | 598, 134  (770 | 713, 159)
// So the store in the launch costs 55 us; a launch of its own in front of the form without it 181 (782 for both, 884 on end).
//
// How long the hardware suspends a failed test is its own affair, so a count of tests is a limit but not one in time.  The time
// limit is the producer's, on the low word of the clock: it sets the abort flag, which every other wait looks at after a
// failed test.  That bounds them all: whatever hangs stops the ring that the producer waits for, and at the end the producer
// waits until every role has taken the end marker, which it does when it is through with all items.
constexpr int kT2WaitLimit = 1 << 22;
__device__ __forceinline__ bool t2_wait(uint64_t* bar, uint32_t parity, volatile int* abort_flag) {
#pragma unroll 1
  for (int n = 0; n < kT2WaitLimit; ++n) {
    if (mbar_try_wait(bar, parity)) return true;
    if (*abort_flag) return false;
  }
  *abort_flag = 1;
  return false;
}
__device__ __forceinline__ uint32_t t2_clock() {
  uint32_t c;
  asm volatile("mov.u32 %0, %%clock;" : "=r"(c));
  return c;
}
__device__ __forceinline__ bool t2_wait_timed(uint64_t* bar, uint32_t parity, volatile int* abort_flag) {
  const uint32_t t0 = t2_clock();
#pragma unroll 1
  while (!mbar_try_wait(bar, parity)) {
    if (*abort_flag) return false;
    if (t2_clock() - t0 > static_cast<uint32_t>(kSpinLimitCycles)) {
      *abort_flag = 1;
      return false;
    }
  }
  return true;
}
// On the S -> softmax -> PV chain: the second test does not come behind a look at the flag (long sequences lose 3 % to it).
__device__ __forceinline__ bool t2_wait_hot(uint64_t* bar, uint32_t parity, volatile int* abort_flag) {
  return mbar_try_wait(bar, parity) || t2_wait(bar, parity, abort_flag);
}

struct T2Item {
  int seq;        // -1: no more work
  int h;
  int q_row;      // global row of the block's first query token
  int tq0;        // that token's index within the sequence
  int Lq, Lk;
  int k_begin;    // dense K/V: first row of the sequence
  int n[2];       // K/V tiles each half needs (n[1] == 0: half B is empty)
};

// Output of one half of an item, run by the output warpgroup: a finished O row out of TMEM in chunks of 16 columns, scaled by
// 1 / row sum and as bf16 into staging boxes in shared memory (32 rows x 32 dims, 2 KiB, 64-byte swizzle; two per warp, used in
// turn).  Where all 32 rows of the warp are query rows the box leaves through a TMA store, with no global store instruction and no
// read-back; else row by row, from the same box.  The accumulator is released as soon as its last chunk is in registers.
__device__ __forceinline__ void t2_stage_chunk(const uint32_t (&ov)[16], unsigned char* box, int lane, int c, float inv) {
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    uint4 w;
    w.x = pack_bf16(__uint_as_float(ov[8 * i]) * inv, __uint_as_float(ov[8 * i + 1]) * inv);
    w.y = pack_bf16(__uint_as_float(ov[8 * i + 2]) * inv, __uint_as_float(ov[8 * i + 3]) * inv);
    w.z = pack_bf16(__uint_as_float(ov[8 * i + 4]) * inv, __uint_as_float(ov[8 * i + 5]) * inv);
    w.w = pack_bf16(__uint_as_float(ov[8 * i + 6]) * inv, __uint_as_float(ov[8 * i + 7]) * inv);
    *reinterpret_cast<uint4*>(box + lane * 64 + (((2 * c + i) ^ ((lane >> 1) & 3)) << 4)) = w;   // 64-byte swizzle
  }
}
// Before a box is written again: the store before the previous one has left it (plain stores are done with it already).
__device__ __forceinline__ void t2_open_box(bool tma, int lane) {
  if (tma && lane == 0) tma_store_wait_read_but_one();
  __syncwarp();
}
// `head0`, `tok0`: head and token of the warp's first tile row, `rows`: how many of its 32 are query rows.
__device__ __forceinline__ void t2_close_box(const PrefillParams& p, const CUtensorMap* map_o, const unsigned char* box, bool tma, int lane, int gs,
                                             int bx, int head0, int tok0, int rows) {
  if (tma) {
    fence_proxy_async_smem();
    __syncwarp();
    if (lane == 0) {
      tma_store_3d(map_o, box, bx * 32, head0, tok0);
      tma_store_commit();
    }
    return;
  }
  __syncwarp();
#pragma unroll 1
  for (int lr = lane >> 2; lr < rows; lr += 8) {
    const uint4 w = *reinterpret_cast<const uint4*>(box + lr * 64 + (((lane & 3) ^ ((lr >> 1) & 3)) << 4));
    reinterpret_cast<uint4*>(p.out + (static_cast<long long>(tok0 + (lr >> gs)) * p.H + head0 + (lr & ((1 << gs) - 1))) * 128)[bx * 4 + (lane & 3)] = w;
  }
  __syncwarp();
}
__device__ __forceinline__ void t2_output(const PrefillParams& p, const CUtensorMap* map_o, uint32_t tmem_o_lane, uint64_t* bar_o_free,
                                          unsigned char* stage, int lane, int gs, float inv, bool tma, int head0, int tok0, int rows) {
  // eight 16-column chunks, the TMEM load of the next one in flight while one is converted
  uint32_t a[16], b[16];
  tc::ld_32x32b_x16(tmem_o_lane, a);
#pragma unroll 1      // (code size: t2_wait)
  for (int bx = 0; bx < 4; ++bx) {
    unsigned char* box = stage + (bx & 1) * 2048;
    t2_open_box(tma, lane);
    tc::wait_ld();
    tc::ld_32x32b_x16(tmem_o_lane + bx * 32 + 16, b);
    t2_stage_chunk(a, box, lane, 0, inv);
    tc::wait_ld();
    if (bx == 3) {
      // the accumulator is in registers: the issuer may start the next item's PV
      tc::fence_before_sync();
      __syncwarp();
      if (lane == 0) mbar_arrive(bar_o_free);
    } else {
      tc::ld_32x32b_x16(tmem_o_lane + bx * 32 + 32, a);
    }
    t2_stage_chunk(b, box, lane, 1, inv);
    t2_close_box(p, map_o, box, tma, lane, gs, bx, head0, tok0, rows);
  }
}

// Output of an item whose keys the halves shared: the same rows lie in both accumulators, each relative to its own half's
// maximum; `wa` and `wb` bring them together (has_b false: there was one tile, half B has nothing).
__device__ __forceinline__ void t2_output_split(const PrefillParams& p, const CUtensorMap* map_o, uint32_t tmem_a, uint32_t tmem_b,
                                                bool has_b, uint64_t* bar_o_free, unsigned char* stage, int lane, int gs,
                                                float wa, float wb, bool tma, int head0, int tok0, int rows) {
#pragma unroll 1
  for (int cch = 0; cch < 8; ++cch) {
    unsigned char* box = stage + ((cch >> 1) & 1) * 2048;
    if (!(cch & 1)) t2_open_box(tma, lane);
    uint32_t a[16], b[16];
    tc::ld_32x32b_x16(tmem_a + cch * 16, a);
    if (has_b) tc::ld_32x32b_x16(tmem_b + cch * 16, b);
    tc::wait_ld();
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      const float o = __uint_as_float(a[i]) * wa;
      a[i] = __float_as_uint(has_b ? fmaf(__uint_as_float(b[i]), wb, o) : o);
    }
    if (cch == 7) {
      tc::fence_before_sync();
      __syncwarp();
      if (lane == 0) {
        mbar_arrive(&bar_o_free[0]);
        if (has_b) mbar_arrive(&bar_o_free[1]);
      }
    }
    t2_stage_chunk(a, box, lane, cch & 1, 1.f);
    if (cch & 1) t2_close_box(p, map_o, box, tma, lane, gs, cch >> 1, head0, tok0, rows);
  }
}

// The layer's cache store (nanovllm/layers/attention.py:10-40) on the side.  Attention over dense K and V does not read
// the cache, so the copy needs no launch of its own in front of it (193 us on 143872 tokens at 16/8 heads, 55 in this one), and every
// K and V tile passes through shared memory anyway: the item whose query block is the first to need a tile sends it on,
// warp 2 the K tiles and warp 3 the V tiles, as TMA stores of 32 rows where the slots run on (they do inside a block),
// else row by row.  Nothing is read from memory for it but the slots.
// t2_store_slots() looks the slots up before the tile has arrived: the slot of its first row if they run on, else -1.
__device__ __forceinline__ int t2_store_slots(const PrefillParams& p, int row0, int rows, int lane) {
  int s[4];
#pragma unroll
  for (int u = 0; u < 4; ++u) s[u] = u * 32 + lane < rows ? ld_s32(p.st_slots + row0 + u * 32 + lane) : 0;
  const int s0 = __shfl_sync(0xffffffffu, s[0], 0);
  bool run = s0 >= 0 && s0 + static_cast<long long>(rows) <= p.st_n_slots;
#pragma unroll
  for (int u = 0; u < 4; ++u) run = run && (u * 32 + lane >= rows || s[u] == s0 + u * 32 + lane);
  return __all_sync(0xffffffffu, run) ? s0 : -1;
}
__device__ __forceinline__ void t2_store_tile(const PrefillParams& p, const CUtensorMap* map, char* cache, const unsigned char* tile,
                                              int h, int row0, int rows, int s0, int lane) {
  const int boxes = s0 >= 0 ? rows >> 5 : 0;
  if (lane == 0 && boxes > 0) {
#pragma unroll 1
    for (int b = 0; b < boxes; ++b) {
      tma_store_3d(map, tile + b * 4096, 0, h, s0 + b * 32);
      tma_store_3d(map, tile + kT2Sub + b * 4096, 64, h, s0 + b * 32);
    }
    tma_store_commit();
  }
  const long long row_bytes = static_cast<long long>(p.Hkv) * 256;
#pragma unroll 1      // (short code: unrolled four times it costs the kernel 5 %, the hot loops fetch from the same cache)
  for (int e = boxes * 512 + lane; e < rows * 16; e += 32) {
    const int r = e >> 4, c = e & 15;
    const long long slot = s0 >= 0 ? s0 + r : ld_s32(p.st_slots + row0 + r);
    if (slot < 0 || slot >= p.st_n_slots) continue;
    *reinterpret_cast<uint4*>(cache + slot * row_bytes + h * 256 + c * 16) =
        *reinterpret_cast<const uint4*>(tile + (c >> 3) * kT2Sub + r * 128 + (((c & 7) ^ (r & 7)) << 4));
  }
  __syncwarp();
  if (lane == 0 && boxes > 0) tma_store_wait_read();
}

// Rows [row0, row1) that no query block loads (sequences without queries, rows outside cu_seqlens_k), all heads.
__device__ __forceinline__ void t2_store_rows(const PrefillParams& p, const char* src, long long stride, char* cache, int row0,
                                              int row1, int lane) {
  const int vecs = p.Hkv * 16;
#pragma unroll 1
  for (int r = row0; r < row1; ++r) {
    const long long slot = ld_s32(p.st_slots + r);
    if (slot < 0 || slot >= p.st_n_slots) continue;
#pragma unroll 1
    for (int v = lane; v < vecs; v += 32)
      reinterpret_cast<uint4*>(cache)[slot * vecs + v] = ld_row16(src + r * stride + v * 16);
  }
}

// Order of the query blocks: s_order has the batch's sequences by ascending number of keys, s_slot the first block of each in
// that order (and, at the end, the number of blocks).  Items are drawn from the back: longest sequence first and in it
// the last, longest block, so that the launch ends with short items whatever order the batch came in.  Two threads per
// sequence count what lies before it.  `scratch`: 8 bytes per sequence.
__device__ __forceinline__ void t2_order(const PrefillParams& p, int QB, int* s_slot, unsigned short* s_order, int2* scratch) {
  const int tid = threadIdx.x;
  if (tid < p.batch) {
    const int Lq = __ldg(p.cu_q + tid + 1) - __ldg(p.cu_q + tid);
    scratch[tid] = make_int2(Lq > 0 ? __ldg(p.cu_k + tid + 1) - __ldg(p.cu_k + tid) : 0, Lq > 0 ? (Lq + QB - 1) / QB : 0);
  }
  __syncthreads();
  const int i = tid >> 1;
  int rank = 0, first = 0;
  if (i < p.batch) {
    const int mine = scratch[i].x;
#pragma unroll 4
    for (int j = tid & 1; j < p.batch; j += 2) {
      const int2 o = scratch[j];
      const bool before = o.x < mine || (o.x == mine && j < i);
      rank += before;
      first += before ? o.y : 0;
    }
  }
  rank += __shfl_xor_sync(0xffffffffu, rank, 1);
  first += __shfl_xor_sync(0xffffffffu, first, 1);
  if (i < p.batch && !(tid & 1)) {
    s_order[rank] = static_cast<unsigned short>(i);
    s_slot[rank] = first;
    if (rank == p.batch - 1) s_slot[p.batch] = min(first + scratch[i].y, p.n_slots);
  }
}

// (kStore in the type, not in the arguments: the code of the store warps moves the hot loops of the others, worth 5 % to a
// launch that stores nothing.)
// kSplit: for launches with few items.  An item is one 128-row tile of queries, and its halves take the key tiles in turn
// (A the even, B the odd ones): the two chains S -> softmax -> PV that a CTA can keep going then work on the same rows, so
// a lone long item takes half as long.  The output warpgroup joins them.  The room of the second Q tile is a third K slot.
template <bool kStore, bool kSplit>
__global__ void __launch_bounds__(kT2Threads, 1)
prefill_attn_tc2_kernel(const PrefillParams p, const __grid_constant__ CUtensorMap map_q,
                        const __grid_constant__ CUtensorMap map_k, const __grid_constant__ CUtensorMap map_v,
                        const __grid_constant__ CUtensorMap map_o, const __grid_constant__ CUtensorMap map_kc,
                        const __grid_constant__ CUtensorMap map_vc) {
  extern __shared__ __align__(1024) unsigned char smem[];
  constexpr int kRingK = kSplit ? kT2Ring + 1 : kT2Ring;
  unsigned char* sQ = smem;                              // [2 (kSplit: 1)][32 KiB]
  unsigned char* sK = smem + (kSplit ? 1 : 2) * kT2Tile; // [kRingK][32 KiB]
  unsigned char* sV = sK + kRingK * kT2Tile;             // [kT2Ring][32 KiB]
  unsigned char* sStage = sV + kT2Ring * kT2Tile;       // [4 output warps][32 rows x 128 B] output staging
  int* s_slot = reinterpret_cast<int*>(sStage + 8 * 2048);       // [batch + 1] first slot of every sequence, in the order of
  unsigned short* s_order = reinterpret_cast<unsigned short*>(s_slot + p.batch + 1);             // [batch]
  __shared__ __align__(8) uint64_t bar_item_full[kT2Items], bar_item_empty[kT2Items];
  __shared__ __align__(8) uint64_t bar_q_full[2], bar_q_empty[2];
  __shared__ __align__(8) uint64_t bar_k_full[kRingK], bar_k_empty[kRingK], bar_v_full[kT2Ring], bar_v_empty[kT2Ring];
  __shared__ __align__(8) uint64_t bar_s_full[2], bar_p_full[2], bar_o_final[2], bar_o_free[2];
  __shared__ __align__(8) uint64_t bar_l_full[2], bar_l_empty[2];
  __shared__ float s_inv[2][128];                        // 1 / row sum of a finished half, softmax -> output warpgroup
  __shared__ float s_max[kSplit ? 2 : 1][128];           // kSplit: a half's row maximum (log2 units), its sum in s_inv
  __shared__ __align__(16) T2Item s_item[kT2Items];
  __shared__ uint32_t s_tmem_base;
  __shared__ int s_abort;

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  // (G divides 128: all of these are powers of two)
  const int G = p.G, gs = __ffs(p.G) - 1, qs_log = (kSplit ? 7 : 8) - gs, QT = 128 >> gs, QB = 1 << qs_log;
  const bool slot_in_smem = p.batch <= kT2MaxSeqSmem;

  if (tid == 0) {
    s_abort = 0;
    for (int i = 0; i < kT2Items; ++i) { mbar_init(&bar_item_full[i], 1); mbar_init(&bar_item_empty[i], kStore ? 15 : 13); }
    for (int i = 0; i < 2; ++i) {
      mbar_init(&bar_q_full[i], 1);
      mbar_init(&bar_q_empty[i], 1);
      mbar_init(&bar_s_full[i], 1);
      mbar_init(&bar_p_full[i], 4);
      mbar_init(&bar_o_final[i], 1);
      mbar_init(&bar_o_free[i], 4);
      mbar_init(&bar_l_full[i], 4);
      mbar_init(&bar_l_empty[i], 4);
    }
    for (int i = 0; i < kRingK; ++i) {
      mbar_init(&bar_k_full[i], 1);
      mbar_init(&bar_k_empty[i], kStore ? 2 : 1);
    }
    for (int i = 0; i < kT2Ring; ++i) {
      mbar_init(&bar_v_full[i], 1);
      mbar_init(&bar_v_empty[i], kStore ? 2 : 1);
    }
    mbar_fence_init();
  }
  // (cu_seqlens ahead of the wait below: no kernel that lets this one start early writes them)
  const bool sorted = p.batch <= kT2MaxSort;
  if (sorted) t2_order(p, QB, s_slot, s_order, reinterpret_cast<int2*>(sStage));
  // Launched with programmatic stream serialization: what is above overlaps the end of the kernel in front.  This kernel does
  // not let its successor start early (its waiting CTAs cost a prefill step 5 %: 166 against 175 us on 16298 tokens), and
  // TMEM is allocated behind the wait (in front of it: 2 % slower on every size, 786 against 769 us on cached prefixes).
  asm volatile("griddepcontrol.wait;" ::: "memory");
  if (slot_in_smem && !sorted)
    for (int i = tid; i <= p.batch; i += kT2Threads) {
      s_slot[i] = (__ldg(p.cu_q + i) >> qs_log) + i;
      if (i < p.batch) s_order[i] = static_cast<unsigned short>(i);
    }
  if (warp == 1) {
    tc::tmem_alloc(&s_tmem_base, 512);
    tc::tmem_relinquish();
  }
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  const uint32_t tmem = s_tmem_base;
  volatile int* abort_flag = &s_abort;

  // Registers move from the light warpgroup to the two softmax warpgroups, which hold a whole
  // 128-column S row (and later the O row) per thread.
  if (warp < 4) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 80;" ::: "memory");
  if (warp == 0) {
    // ================================ TMA producer ================================
    if (lane == 0) {
      tma_prefetch_desc(&map_q);
      tma_prefetch_desc(&map_k);
      tma_prefetch_desc(&map_v);
      const int n_slots = sorted ? s_slot[p.batch] : p.n_slots;
      const unsigned int n_items = static_cast<unsigned int>(n_slots) * p.Hkv;
      int n_pub = 0;            // items published
      int kt = 0, vt = 0;       // K / V tiles issued so far (ring positions)
      bool ok = true;
      while (ok) {
        // a ticket; each CTA draws until it fails, the last ticket of the launch resets the counter
        const unsigned int tk = atomicAdd(&g_prefill_ticket, 1u);
        if (tk == n_items + gridDim.x - 1) atomicExch(&g_prefill_ticket, 0u);
        // the descriptor is built in its ring slot; only what the loads need stays in registers
        const int is = n_pub % kT2Items;
        if (!t2_wait_timed(&bar_item_empty[is], ((n_pub / kT2Items) & 1) ^ 1, abort_flag)) { ok = false; break; }
        int seq = -1, h = 0, q_row = 0, k_begin = 0, n = 0;
        bool b_rows = false;                                            // half B holds query rows
        if (tk < n_items) {
          h = tk % p.Hkv;
          const int x = n_slots - 1 - static_cast<int>(tk / p.Hkv);     // reverse slot order: within a sequence the later, longer blocks come first
          int lo = 0, hi = p.batch;
          while (hi - lo > 1) {
            const int mid = (lo + hi) >> 1;
            const int f = slot_in_smem ? s_slot[mid] : (__ldg(p.cu_q + mid) >> qs_log) + mid;
            if (f <= x) lo = mid; else hi = mid;
          }
          const int qb = x - (slot_in_smem ? s_slot[lo] : (__ldg(p.cu_q + lo) >> qs_log) + lo);
          if (slot_in_smem) lo = s_order[lo];
          const int q_begin = __ldg(p.cu_q + lo);
          const int Lq = __ldg(p.cu_q + lo + 1) - q_begin;
          if (qb < 0 || qb * QB >= Lq) continue;                        // slot owns no query block
          k_begin = __ldg(p.cu_k + lo);
          const int Lk = __ldg(p.cu_k + lo + 1) - k_begin;
          const int shift = Lk - Lq;
          const int tq0 = qb * QB;
          const int nA = max(0, (min(Lk, shift + min(tq0 + QT, Lq)) + kT2Kv - 1) / kT2Kv);
          b_rows = !kSplit && tq0 + QT < Lq;
          const int nB = b_rows ? max(0, (min(Lk, shift + min(tq0 + QB, Lq)) + kT2Kv - 1) / kT2Kv) : 0;
          seq = lo;
          q_row = q_begin + tq0;
          n = max(nA, nB);
          s_item[is].h = h;
          s_item[is].q_row = q_row;
          s_item[is].tq0 = tq0;
          s_item[is].Lq = Lq;
          s_item[is].Lk = Lk;
          s_item[is].k_begin = k_begin;
          s_item[is].n[0] = kSplit ? (n + 1) >> 1 : nA;
          s_item[is].n[1] = kSplit ? n >> 1 : nB;
        }
        s_item[is].seq = seq;
        mbar_arrive(&bar_item_full[is]);                                // an item, or the end marker
        if (seq < 0) {
          t2_wait_timed(&bar_item_empty[is], (n_pub / kT2Items) & 1, abort_flag);     // every role has taken it
          break;
        }
        // The Q tiles can only be loaded once the previous item has let go of the buffers, which is when
        // they are needed: start them on their way into L2 now, with the item's first K/V tile.
        tma_prefetch_l2_3d(&map_q, 0, h * G, q_row);
        tma_prefetch_l2_3d(&map_q, 64, h * G, q_row);
        if (b_rows) {
          tma_prefetch_l2_3d(&map_q, 0, h * G, q_row + QT);
          tma_prefetch_l2_3d(&map_q, 64, h * G, q_row + QT);
        }
        // Q tiles (the buffers are free once every S MMA of the previous item has completed)
        const uint32_t qph = (n_pub & 1) ^ 1;
        for (int hx = 0; hx < 2; ++hx) {
          if (!t2_wait_timed(&bar_q_empty[hx], qph, abort_flag)) { ok = false; break; }
          if (hx == 1 && !b_rows) { mbar_arrive(&bar_q_full[1]); continue; }
          mbar_expect_tx(&bar_q_full[hx], kT2Tile);
          tma_load_3d(sQ + hx * kT2Tile, &map_q, &bar_q_full[hx], 0, h * G, q_row + hx * QT);
          tma_load_3d(sQ + hx * kT2Tile + kT2Sub, &map_q, &bar_q_full[hx], 64, h * G, q_row + hx * QT);
        }
        if (!ok) break;
        ++n_pub;
        // K and V tiles
        const int* bt_row = p.block_tables ? p.block_tables + seq * p.bt_row_stride : nullptr;
        // row of the next tile in turn (paged: the next block when one is through; blocks are multiples of 256 keys)
        int row_at = k_begin, left = bt_row ? 0 : 0x7fffffff, col = 0;
        auto next_row = [&]() -> int {
          if (left == 0) {
            const long long blk = col < p.bt_cols ? bt_row[col] : -1;
            ++col;
            left = p.block_size;
            row_at = blk >= 0 && blk < p.num_blocks ? static_cast<int>(blk * p.block_size) : -(1 << 30);      // (nowhere: zeros)
          }
          const int row = row_at;
          left -= kT2Kv;
          row_at += kT2Kv;
          return row;
        };
        auto load_k = [&](int row0) -> bool {
          const int ks = kt % kRingK;
          if (!t2_wait_timed(&bar_k_empty[ks], ((kt / kRingK) & 1) ^ 1, abort_flag)) return false;
          mbar_expect_tx(&bar_k_full[ks], kT2Tile);
          tma_load_3d(sK + ks * kT2Tile, &map_k, &bar_k_full[ks], 0, h, row0);
          tma_load_3d(sK + ks * kT2Tile + kT2Sub, &map_k, &bar_k_full[ks], 64, h, row0);
          ++kt;
          return true;
        };
        auto load_v = [&](int row0) -> bool {
          const int vs = vt % kT2Ring;
          if (!t2_wait_timed(&bar_v_empty[vs], ((vt / kT2Ring) & 1) ^ 1, abort_flag)) return false;
          mbar_expect_tx(&bar_v_full[vs], kT2Tile);
          tma_load_3d(sV + vs * kT2Tile, &map_v, &bar_v_full[vs], 0, h, row0);
          tma_load_3d(sV + vs * kT2Tile + kT2Sub, &map_v, &bar_v_full[vs], 64, h, row0);
          ++vt;
          return true;
        };
        if constexpr (kSplit) {
          // K two tiles ahead of V: the issuer needs K of step j + 2 in step j
          int row = 0, v0 = 0, v1 = 0;
#pragma unroll 1
          for (int j = 0; j < n + 2 && ok; ++j) {
            if (j < n) {
              row = next_row();
              ok = load_k(row);
            }
            if (ok && j >= 2) ok = load_v(v0);
            v0 = v1;
            v1 = row;
          }
        } else {
#pragma unroll 1
          for (int j = 0; j < n && ok; ++j) {
            const int row0 = next_row();
            ok = load_k(row0) && load_v(row0);
          }
        }
      }
    }
  } else if (warp == 1) {
    // ================================ MMA issuer ================================
    if (lane == 0) {
      constexpr uint32_t idesc_qk = tc::idesc_bf16_f32(128, 128, false, false);
      constexpr uint32_t idesc_pv = tc::idesc_bf16_f32(128, 128, false, true);
      constexpr uint32_t desc_hi = tc::smem_desc_sw128_hi(1024);
      const uint32_t q_lo = tc::smem_desc_sw128_lo(smem_u32(sQ), 16), k_lo = tc::smem_desc_sw128_lo(smem_u32(sK), 16);
      const uint32_t v_lo = tc::smem_desc_sw128_lo(smem_u32(sV), kT2Sub);
      int n_item = 0, kt = 0, vt = 0;
      int k_at = 0, k_ph = 0; // kSplit: place and phase in the K ring
      int np[2] = {0, 0};     // P tiles consumed per half (phase of bar_p_full)
      int no[2] = {0, 0};     // items whose O was read out per half (phase of bar_o_free)
      bool ok = true;
      auto issue_s = [&](int hx, int kslot) {
#pragma unroll
        for (int ks = 0; ks < 8; ++ks) {
          const uint32_t off = ((ks >> 2) * kT2Sub + (ks & 3) * 32) >> 4;
          tc::mma_ss_lo(tmem + hx * 128, q_lo + (kSplit ? 0 : hx) * (kT2Tile >> 4) + off, k_lo + kslot * (kT2Tile >> 4) + off, desc_hi,
                        idesc_qk, ks > 0);
        }
        tc::commit(&bar_s_full[hx]);
      };
      auto issue_pv = [&](int hx, int vslot, bool accumulate) {
#pragma unroll
        for (int ks = 0; ks < 8; ++ks)
          tc::mma_ts_lo(tmem + 256 + hx * 128, tmem + hx * 128 + ks * 8, v_lo + vslot * (kT2Tile >> 4) + ks * (2048 >> 4),
                        desc_hi, idesc_pv, accumulate || ks > 0);
      };
      while (ok) {
        const int is = n_item % kT2Items;
        if (!t2_wait(&bar_item_full[is], (n_item / kT2Items) & 1, abort_flag)) break;
        const int seq = s_item[is].seq, nA = s_item[is].n[0], nB = s_item[is].n[1], n = kSplit ? nA + nB : max(nA, nB);
        mbar_arrive(&bar_item_empty[is]);
        if (seq < 0) break;
        const uint32_t qph = n_item & 1;
        if (!t2_wait(&bar_q_full[0], qph, abort_flag) || !t2_wait(&bar_q_full[1], qph, abort_flag)) break;
        if constexpr (kSplit) {
          // the first S of either half, then PV of step j (half j & 1) and that half's next S; ring places and phases are
          // counted along, the half is a constant of the code: what this thread computes is tensor-core idle time
          auto next_k = [&]() { if (++k_at == kRingK) { k_at = 0; k_ph ^= 1; } };
          for (int j = 0; j < 2 && j < n && ok; ++j) {
            if (!t2_wait_hot(&bar_k_full[k_at], k_ph, abort_flag)) { ok = false; break; }
            tc::fence_after_sync();
            issue_s(j, k_at);
            tc::commit(&bar_k_empty[k_at]);
            next_k();
          }
          if (n <= 2) { tc::commit(&bar_q_empty[0]); tc::commit(&bar_q_empty[1]); }
          auto step = [&](auto half, int j) -> bool {
            constexpr int hx = decltype(half)::value;
            const int vslot = vt & 1;
            if (!t2_wait_hot(&bar_v_full[vslot], (vt >> 1) & 1, abort_flag)) return false;
            if (j + 2 < n && !t2_wait_hot(&bar_k_full[k_at], k_ph, abort_flag)) return false;
            if (j < 2 && !t2_wait_hot(&bar_o_free[hx], (no[hx] & 1) ^ 1, abort_flag)) return false;
            if (!t2_wait_hot(&bar_p_full[hx], np[hx] & 1, abort_flag)) return false;
            ++np[hx];
            tc::fence_after_sync();
            issue_pv(hx, vslot, j >= 2);
            tc::commit(&bar_v_empty[vslot]);
            ++vt;
            if (j + 2 >= n) {
              tc::commit(&bar_o_final[hx]);
              ++no[hx];
            } else {
              issue_s(hx, k_at);
              tc::commit(&bar_k_empty[k_at]);
              next_k();
              if (j + 3 >= n) { tc::commit(&bar_q_empty[0]); tc::commit(&bar_q_empty[1]); }   // the item's last S
            }
            return true;
          };
          static_assert(kT2Ring == 2, "V ring");
          for (int j = 0; j < n && ok; j += 2) {
            ok = step(std::integral_constant<int, 0>{}, j);
            if (ok && j + 1 < n) ok = step(std::integral_constant<int, 1>{}, j + 1);
          }
          ++n_item;
          continue;
        }
        // first K tile: S for both halves
        if (n > 0) {
          if (!t2_wait_hot(&bar_k_full[kt % kT2Ring], (kt / kT2Ring) & 1, abort_flag)) break;
          tc::fence_after_sync();
#pragma unroll 1      // (code size)
          for (int hx = 0; hx < 2; ++hx)
            if ((hx ? nB : nA) > 0) issue_s(hx, kt % kT2Ring);
          tc::commit(&bar_k_empty[kt % kT2Ring]);
          ++kt;
        }
        if (nA <= 1) tc::commit(&bar_q_empty[0]);
        if (nB <= 1) tc::commit(&bar_q_empty[1]);
        for (int j = 0; j < n && ok; ++j) {
          const int vslot = vt % kT2Ring;
          // V_j and the next K tile land long before the softmax is through: their barriers are tested
          // first, so that little but the issue itself stands between a half's P and its MMAs
          if (!t2_wait_hot(&bar_v_full[vslot], (vt / kT2Ring) & 1, abort_flag)) { ok = false; break; }
          if (j + 1 < n && !t2_wait_hot(&bar_k_full[kt % kT2Ring], (kt / kT2Ring) & 1, abort_flag)) { ok = false; break; }
          if (j == 0) {
            // the output warpgroup must have taken the previous item's O out of both accumulators
            if (nA > 0 && !t2_wait_hot(&bar_o_free[0], (no[0] & 1) ^ 1, abort_flag)) { ok = false; break; }
            if (nB > 0 && !t2_wait_hot(&bar_o_free[1], (no[1] & 1) ^ 1, abort_flag)) { ok = false; break; }
          }
          for (int hx = 0; hx < 2 && ok; ++hx) {
            const int nx = hx == 0 ? nA : nB;
            if (j >= nx) continue;
            // O_X += P_X V_j
            if (!t2_wait_hot(&bar_p_full[hx], np[hx] & 1, abort_flag)) { ok = false; break; }
            ++np[hx];
            tc::fence_after_sync();
            issue_pv(hx, vslot, j > 0);
            if (j == nx - 1) { tc::commit(&bar_o_final[hx]); ++no[hx]; }
            // S_X for the next K tile (its buffer is free: the PV above reads P before it runs)
            if (j + 1 < nx) {
              issue_s(hx, kt % kT2Ring);
              if (j + 2 >= nx) tc::commit(&bar_q_empty[hx]);   // that was the half's last S: its Q tile is free
            }
          }
          if (!ok) break;
          tc::commit(&bar_v_empty[vslot]);
          ++vt;
          if (j + 1 < n) { tc::commit(&bar_k_empty[kt % kT2Ring]); ++kt; }
        }
        ++n_item;
      }
    }
  } else if (kStore) {
    // ================================ cache store ================================
    const bool is_v = warp == 3;
    uint64_t* const full = is_v ? bar_v_full : bar_k_full;
    uint64_t* const empty = is_v ? bar_v_empty : bar_k_empty;     // (a tile's slot is free when this warp is through, too)
    const unsigned char* const ring = is_v ? sV : sK;
    const int depth = !kSplit || is_v ? kT2Ring : kRingK;
    const CUtensorMap* const map = is_v ? &map_vc : &map_kc;
    char* const cache = is_v ? p.st_v_cache : p.st_k_cache;
    int n_item = 0, kt = 0;
    bool ok = true;
    while (ok) {
      const int is = n_item % kT2Items;
      if (!t2_wait(&bar_item_full[is], (n_item / kT2Items) & 1, abort_flag)) break;
      const int seq = s_item[is].seq, h = s_item[is].h, tq0 = s_item[is].tq0, Lq = s_item[is].Lq, Lk = s_item[is].Lk;
      const int k_begin = s_item[is].k_begin, n = kSplit ? s_item[is].n[0] + s_item[is].n[1] : max(s_item[is].n[0], s_item[is].n[1]);
      __syncwarp();
      if (lane == 0) mbar_arrive(&bar_item_empty[is]);
      if (seq < 0) break;
      ++n_item;
      // The tiles this item stores: those whose first row lies in its query block; where queries and keys do not
      // start together, the sequence's last item, which loads all tiles, stores them all.
      const int j0 = Lq == Lk ? (tq0 + kT2Kv - 1) / kT2Kv : tq0 + QB >= Lq ? 0 : n;
      const int j1 = Lq == Lk ? min(n, (tq0 + QB + kT2Kv - 1) / kT2Kv) : n;
#pragma unroll 1
      for (int j = 0; j < n; ++j, ++kt) {
        const int slot = kt % depth;
        const bool mine = j >= j0 && j < j1;
        const int row0 = k_begin + j * kT2Kv, rows = min(min(kT2Kv, Lk - j * kT2Kv), p.st_tokens - row0);
        const int s0 = mine ? t2_store_slots(p, row0, rows, lane) : -1;
        if (!t2_wait(&full[slot], (kt / depth) & 1, abort_flag)) { ok = false; break; }
        if (mine) t2_store_tile(p, map, cache, ring + slot * kT2Tile, h, row0, rows, s0, lane);
        __syncwarp();
        if (lane == 0) mbar_arrive(&empty[slot]);
      }
    }
    if (ok) {
      const char* src = is_v ? p.st_v : p.st_k;
      const long long stride = is_v ? p.st_v_stride : p.st_k_stride;
      // (segment g: sequence g - 1; 0 and batch + 1: the rows in front of the first and behind the last)
#pragma unroll 1
      for (int g = blockIdx.x; g < p.batch + 2; g += gridDim.x) {
        const int r0 = g == 0 ? 0 : __ldg(p.cu_k + g - 1), r1 = g > p.batch ? p.st_tokens : min(__ldg(p.cu_k + g), p.st_tokens);
        if (g == 0 || g > p.batch || __ldg(p.cu_q + g - 1) == __ldg(p.cu_q + g)) t2_store_rows(p, src, stride, cache, r0, r1, lane);
      }
    }
  }
  } else if (warp < 12) {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 184;" ::: "memory");
    // ================================ softmax / epilogue ================================
    const int hx = (warp - 4) >> 2;                     // which half this warpgroup serves
    const int quarter = warp & 3;                       // TMEM lanes this warp may touch
    const int r = quarter * 32 + lane;                  // row of the (token, head) product
    const uint32_t lane_base = static_cast<uint32_t>(quarter * 32) << 16;
    const uint32_t tmem_s = tmem + hx * 128, tmem_o = tmem + 256 + hx * 128;
    const float c = p.scale_log2;
    int n_item = 0, ns = 0, vt_base = 0;
    bool ok = true;
    int n_fin = 0;                                      // halves handed to the output warpgroup

    while (ok) {
      const int is = n_item % kT2Items;
      if (!t2_wait(&bar_item_full[is], (n_item / kT2Items) & 1, abort_flag)) break;
      const T2Item it = s_item[is];
      __syncwarp();
      if (lane == 0) mbar_arrive(&bar_item_empty[is]);   // this warp has its copy
      if (it.seq < 0) break;
      ++n_item;
      const int nx = hx ? it.n[1] : it.n[0];
      const int n_all = kSplit ? it.n[0] + it.n[1] : max(it.n[0], it.n[1]);
      const int row_half = kSplit ? 0 : hx;               // which rows and ...
      const int shift = it.Lk - it.Lq;
      const int tok = it.tq0 + row_half * QT + (r >> gs);
      const bool row_ok = tok < it.Lq;
      const int kmax = row_ok ? shift + tok : -1;          // last visible key (inclusive)
      const int first_row_kmax = shift + it.tq0 + row_half * QT;
      float m_used = -INFINITY, l = 0.f;
      for (int j = 0; j < nx; ++j) {
        if (!t2_wait_hot(&bar_s_full[hx], ns & 1, abort_flag)) { ok = false; break; }
        ++ns;
        tc::fence_after_sync();
        const int tile = kSplit ? 2 * j + hx : j;        // ... which key tiles this half works on
        const int key0 = tile * kT2Kv;
        const bool need_mask = key0 + kT2Kv - 1 > first_row_kmax;
        // the whole S row in registers: four TMEM loads in flight, one wait
        uint32_t sv[4][32];
#pragma unroll
        for (int cch = 0; cch < 4; ++cch) tc::ld_32x32b_x32(tmem_s + lane_base + cch * 32, sv[cch]);
        tc::wait_ld();
        if (need_mask) {
          const int nvalid = kmax - key0 + 1;           // columns of this row that may be seen
#pragma unroll
          for (int cch = 0; cch < 4; ++cch) {
            if (nvalid < (cch + 1) * 32) {
              const uint32_t keep = nvalid <= cch * 32 ? 0u : (1u << (nvalid - cch * 32)) - 1;              // a chunk that lies wholly below the diagonal costs nothing
#pragma unroll
              for (int i = 0; i < 32; ++i)
                if (!((keep >> i) & 1)) sv[cch][i] = 0xff800000u;   // -inf
            }
          }
        }
        // eight independent chains of 3-input max
        float mx0 = -INFINITY, mx1 = -INFINITY, mx2 = -INFINITY, mx3 = -INFINITY;
        float mx4 = -INFINITY, mx5 = -INFINITY, mx6 = -INFINITY, mx7 = -INFINITY;
#pragma unroll
        for (int cch = 0; cch < 4; ++cch) {
#pragma unroll
          for (int i = 0; i < 32; i += 16) {
            mx0 = fmax3(mx0, __uint_as_float(sv[cch][i]), __uint_as_float(sv[cch][i + 1]));
            mx1 = fmax3(mx1, __uint_as_float(sv[cch][i + 2]), __uint_as_float(sv[cch][i + 3]));
            mx2 = fmax3(mx2, __uint_as_float(sv[cch][i + 4]), __uint_as_float(sv[cch][i + 5]));
            mx3 = fmax3(mx3, __uint_as_float(sv[cch][i + 6]), __uint_as_float(sv[cch][i + 7]));
            mx4 = fmax3(mx4, __uint_as_float(sv[cch][i + 8]), __uint_as_float(sv[cch][i + 9]));
            mx5 = fmax3(mx5, __uint_as_float(sv[cch][i + 10]), __uint_as_float(sv[cch][i + 11]));
            mx6 = fmax3(mx6, __uint_as_float(sv[cch][i + 12]), __uint_as_float(sv[cch][i + 13]));
            mx7 = fmax3(mx7, __uint_as_float(sv[cch][i + 14]), __uint_as_float(sv[cch][i + 15]));
          }
        }
        const float mx = fmax3(fmax3(mx0, mx1, mx2), fmax3(mx3, mx4, mx5), fmaxf(mx6, mx7));
        const float m_new = fmaxf(m_used, mx);
        if (j == 0) {
          m_used = m_new;
        } else {
          const bool grow = (m_new - m_used) * c > kT2Rescale;
          if (__any_sync(0xffffffffu, grow)) {
            const float alpha = grow ? fast_exp2((m_used - m_new) * c) : 1.f;
            if (grow) { m_used = m_new; l *= alpha; }
#pragma unroll 1          // (code size: t2_wait)
            for (int cch = 0; cch < 8; ++cch) {
              uint32_t v[16];
              tc::ld_32x32b_x16(tmem_o + lane_base + cch * 16, v);
              tc::wait_ld();
#pragma unroll
              for (int i = 0; i < 16; ++i) v[i] = __float_as_uint(__uint_as_float(v[i]) * alpha);
              tc::st_32x32b_x16(tmem_o + lane_base + cch * 16, v);
            }
          }
        }
        // P = exp2(c * (s - m)) (masked entries are -inf -> 0), row sum, packed bf16 back over S
        const float mc = (m_used == -INFINITY ? 0.f : m_used) * c;
        // packed 2 x fp32 FMA and ADD: half the instructions of the scalar form
        const unsigned long long c2 = f32x2_pack(c, c), nmc2 = f32x2_pack(-mc, -mc);
        unsigned long long ls0 = 0ull, ls1 = 0ull, ls2 = 0ull, ls3 = 0ull;   // four independent (pair) sum chains
#pragma unroll
        for (int cch = 0; cch < 4; ++cch) {
          uint32_t pk[16];
#pragma unroll
          for (int i = 0; i < 16; i += 4) {
            float p0, p1, p2, p3, p4, p5, p6, p7;
            f32x2_unpack(f32x2_fma(f32x2_pack(__uint_as_float(sv[cch][2 * i]), __uint_as_float(sv[cch][2 * i + 1])), c2, nmc2), p0, p1);
            f32x2_unpack(f32x2_fma(f32x2_pack(__uint_as_float(sv[cch][2 * i + 2]), __uint_as_float(sv[cch][2 * i + 3])), c2, nmc2), p2, p3);
            f32x2_unpack(f32x2_fma(f32x2_pack(__uint_as_float(sv[cch][2 * i + 4]), __uint_as_float(sv[cch][2 * i + 5])), c2, nmc2), p4, p5);
            f32x2_unpack(f32x2_fma(f32x2_pack(__uint_as_float(sv[cch][2 * i + 6]), __uint_as_float(sv[cch][2 * i + 7])), c2, nmc2), p6, p7);
            p0 = fast_exp2(p0); p1 = fast_exp2(p1); p2 = fast_exp2(p2); p3 = fast_exp2(p3);
            p4 = fast_exp2(p4); p5 = fast_exp2(p5); p6 = fast_exp2(p6); p7 = fast_exp2(p7);
            ls0 = f32x2_add(ls0, f32x2_pack(p0, p1));
            ls1 = f32x2_add(ls1, f32x2_pack(p2, p3));
            ls2 = f32x2_add(ls2, f32x2_pack(p4, p5));
            ls3 = f32x2_add(ls3, f32x2_pack(p6, p7));
            pk[i] = pack_bf16(p0, p1);
            pk[i + 1] = pack_bf16(p2, p3);
            pk[i + 2] = pack_bf16(p4, p5);
            pk[i + 3] = pack_bf16(p6, p7);
          }
          tc::st_32x32b_x16(tmem_s + lane_base + cch * 16, pk);
        }
        float l0, l1, l2, l3;
        {
          float a0, a1;
          f32x2_unpack(f32x2_add(f32x2_add(ls0, ls1), f32x2_add(ls2, ls3)), a0, a1);
          l0 = a0; l1 = a1; l2 = 0.f; l3 = 0.f;
        }
        l += (l0 + l1) + (l2 + l3);
        tc::wait_st();
        if (key0 + kT2Kv > it.Lk) {
          // ragged last tile of the sequence: V rows past its end are foreign data; zero them so
          // that 0 * garbage cannot turn into NaN inside the tensor core
          const int vt = vt_base + tile;
          if (!t2_wait_hot(&bar_v_full[vt % kT2Ring], (vt / kT2Ring) & 1, abort_flag)) { ok = false; break; }
          // (Rows are 128 bytes and follow each other, so they are zeroed as one range, thread after thread: a row per
          // thread hits the same banks with every lane and took 2000 cycles.)
          unsigned char* vrow = sV + (vt % kT2Ring) * kT2Tile;
#pragma unroll 1
          for (int i = (it.Lk - key0) * 128 + r * 16; i < kT2Sub; i += 128 * 16) {
            *reinterpret_cast<uint4*>(vrow + i) = make_uint4(0, 0, 0, 0);
            *reinterpret_cast<uint4*>(vrow + kT2Sub + i) = make_uint4(0, 0, 0, 0);
          }
          fence_proxy_async_smem();
        }
        tc::fence_before_sync();
        __syncwarp();
        if (lane == 0) mbar_arrive(&bar_p_full[hx]);   // one arrival per warp
      }
      if (!ok) break;
      vt_base += n_all;
      if (nx > 0) {
        // the row's 1 / sum goes to the output warpgroup, which drains O while this one moves on
        if (!t2_wait(&bar_l_empty[hx], (n_fin & 1) ^ 1, abort_flag)) { ok = false; break; }
        if constexpr (kSplit) s_max[hx][r] = m_used == -INFINITY ? -INFINITY : m_used * c;
        s_inv[hx][r] = kSplit ? l : l > 0.f ? 1.f / l : 0.f;
        __syncwarp();
        if (lane == 0) mbar_arrive(&bar_l_full[hx]);
        ++n_fin;
      } else if (row_ok && (!kSplit || n_all == 0) && !(kSplit && hx)) {
        // no visible key at all (Lk < Lq rows): zeros, as the reference's attention library does
        uint4* dst = reinterpret_cast<uint4*>(p.out + (static_cast<long long>(it.q_row + row_half * QT + (r >> gs)) * p.H + it.h * G + (r & (G - 1))) * 128);
#pragma unroll
        for (int i = 0; i < 16; ++i) dst[i] = make_uint4(0, 0, 0, 0);
      }
    }
  } else {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 64;" ::: "memory");
    // ================================ output warpgroup ================================
    const int quarter = warp & 3;
    const int r = quarter * 32 + lane;
    const uint32_t lane_base = static_cast<uint32_t>(quarter * 32) << 16;
    int n_item = 0;
    int nf[2] = {0, 0};                                  // halves drained so far
    bool ok = true;
    while (ok) {
      const int is = n_item % kT2Items;
      if (!t2_wait(&bar_item_full[is], (n_item / kT2Items) & 1, abort_flag)) break;
      const int seq = s_item[is].seq, h = s_item[is].h, q_row = s_item[is].q_row, tq0 = s_item[is].tq0, Lq = s_item[is].Lq;
      const int nA = s_item[is].n[0], nB = s_item[is].n[1];
      __syncwarp();
      if (lane == 0) mbar_arrive(&bar_item_empty[is]);
      if (seq < 0) break;
      ++n_item;
      if constexpr (kSplit) {
        if (nA <= 0) continue;
        const bool has_b = nB > 0;
        float m[2] = {0.f, -INFINITY}, l[2] = {0.f, 0.f};
#pragma unroll
        for (int hx = 0; hx < 2; ++hx) {
          if (hx == 1 && !has_b) continue;
          if (!t2_wait(&bar_l_full[hx], nf[hx] & 1, abort_flag)) ok = false;
          m[hx] = s_max[hx][r];
          l[hx] = s_inv[hx][r];
          __syncwarp();
          if (lane == 0) mbar_arrive(&bar_l_empty[hx]);
          if (!t2_wait(&bar_o_final[hx], nf[hx] & 1, abort_flag)) ok = false;
          ++nf[hx];
        }
        if (!ok) break;
        tc::fence_after_sync();
        const float M = fmaxf(m[0], m[1]);
        float wa = M == -INFINITY ? 0.f : fast_exp2(m[0] - M), wb = M == -INFINITY ? 0.f : fast_exp2(m[1] - M);
        const float sum = l[0] * wa + l[1] * wb, inv = sum > 0.f ? 1.f / sum : 0.f;
        const int rows = min(32, (min(Lq - tq0, QT) << gs) - quarter * 32);
        const bool tma = p.out_tma && rows == 32;
        if (!tma) {
          if (lane == 0) tma_store_wait_read();
          __syncwarp();
        }
        t2_output_split(p, &map_o, tmem + 256 + lane_base, tmem + 384 + lane_base, has_b, bar_o_free, sStage + quarter * 4096, lane, gs,
                        wa * inv, wb * inv, tma, h * G + (G > 32 ? (quarter * 32) & (G - 1) : 0), q_row + (quarter * 32 >> gs), rows);
        continue;
      }
#pragma unroll 1
      for (int hx = 0; hx < 2; ++hx) {
        if ((hx == 0 ? nA : nB) <= 0) continue;
        const uint32_t ph = nf[hx] & 1;
        if (!t2_wait(&bar_l_full[hx], ph, abort_flag)) { ok = false; break; }
        const float inv = s_inv[hx][r];
        __syncwarp();
        if (lane == 0) mbar_arrive(&bar_l_empty[hx]);
        if (!t2_wait(&bar_o_final[hx], ph, abort_flag)) { ok = false; break; }
        tc::fence_after_sync();
        const int rows = min(32, (min(Lq - tq0 - hx * QT, QT) << gs) - quarter * 32);      // query rows among this warp's
        const bool tma = p.out_tma && rows == 32;
        if (!tma) {
          if (lane == 0) tma_store_wait_read();
          __syncwarp();
        }
        t2_output(p, &map_o, tmem + 256 + hx * 128 + lane_base, &bar_o_free[hx], sStage + quarter * 4096, lane, gs, inv, tma,
                  h * G + (G > 32 ? (quarter * 32) & (G - 1) : 0), q_row + hx * QT + (quarter * 32 >> gs), rows);
        ++nf[hx];
      }
    }
    if (lane == 0) tma_store_wait_read();                // the staging tile must outlive its last store
  }

  // ---- teardown: everyone meets, then the allocating warp frees TMEM ----
  tc::fence_before_sync();
  __syncthreads();
  if (warp == 1) {
    tc::fence_after_sync();
    tc::tmem_dealloc(tmem, 512);
  }
  if (tid == 0 && s_abort) atomicExch(&g_status_prefill_tc2, 1);
}


int read_status_prefill_tc2() {
  int v = 0;
  cudaMemcpyFromSymbol(&v, g_status_prefill_tc2, sizeof(int));
  return v;
}

// A launch that gave up on a wait never draws its last ticket, so the counter keeps a stale value that
// would make the next launch skip its first items: clear it together with the status word.
int reset_state_prefill_tc2() {
  const int zero = 0;
  const unsigned int uzero = 0;
  int rc = check_cuda(cudaMemcpyToSymbol(g_status_prefill_tc2, &zero, sizeof(int)), "device_status: clearing the tcgen05 status word");
  if (rc) return rc;
  return check_cuda(cudaMemcpyToSymbol(g_prefill_ticket, &uzero, sizeof(unsigned int)), "device_status: clearing the ticket counter");
}

int inject_timeout_prefill_tc2() {
  const int one = 1;
  const unsigned int stale = 7;
  int rc = check_cuda(cudaMemcpyToSymbol(g_status_prefill_tc2, &one, sizeof(int)), "inject_timeout: status word");
  if (rc) return rc;
  return check_cuda(cudaMemcpyToSymbol(g_prefill_ticket, &stale, sizeof(unsigned int)), "inject_timeout: ticket counter");
}

// Test hook: one thread waits on a barrier that nobody arrives on, with either of the library's waits.
static __device__ float g_wait_seconds[2];
static __global__ void wait_limit_kernel() {
  __shared__ __align__(8) uint64_t bar;
  __shared__ int s_abort;
  mbar_init(&bar, 1);
  mbar_fence_init();
#pragma unroll 1
  for (int i = 0; i < 2; ++i) {
    s_abort = 0;
    unsigned long long t0, t1;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t0)::"memory");
    const bool arrived = i == 0 ? mbar_wait(&bar, 0, &s_abort) : t2_wait_timed(&bar, 0, &s_abort);
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t1)::"memory");
    g_wait_seconds[i] = !arrived && *const_cast<volatile int*>(&s_abort) ? static_cast<float>(t1 - t0) * 1e-9f : -1.f;
  }
}
int test_wait_limits(float* seconds) {
  wait_limit_kernel<<<1, 1>>>();
  int rc = check_cuda(cudaGetLastError(), "test_wait_limits launch");
  if (rc) return rc;
  return check_cuda(cudaMemcpyFromSymbol(seconds, g_wait_seconds, sizeof(g_wait_seconds)), "test_wait_limits");
}

// Needs whole query heads groups in a 128-row tile.  The query-block slots are laid out for 2 * QT tokens, or QT with `split`.
int launch_prefill_tc2(PrefillParams p, bool split, const CUtensorMap& map_q, const CUtensorMap& map_k, const CUtensorMap& map_v,
                       const CUtensorMap& map_o, const CUtensorMap& map_kc, const CUtensorMap& map_vc, cudaStream_t stream) {
  p.n_slots = p.total_q / ((split ? 1 : 2) * p.QT) + p.batch;
  const size_t smem = static_cast<size_t>(2 + 2 * kT2Ring) * kT2Tile + 8 * 2048 +
                      (p.batch <= kT2MaxSeqSmem ? (p.batch + 1) * 6 : 4) + 64;
  static std::atomic<size_t> configured[4][kMaxDevices];
  const bool store = p.st_slots != nullptr;
  auto* const kernel = split ? (store ? prefill_attn_tc2_kernel<true, true> : prefill_attn_tc2_kernel<false, true>)
                             : (store ? prefill_attn_tc2_kernel<true, false> : prefill_attn_tc2_kernel<false, false>);
  const int rc = ensure_dynamic_smem(reinterpret_cast<const void*>(kernel), smem, configured[2 * split + store],
                                     "prefill_attn(tcgen05): cudaFuncSetAttribute");
  if (rc) return rc;
  const int grid = sm_count();
  if (grid <= 0) return set_error(kErrNoDriver, "prefill_attn: no CUDA device");
  if (static_cast<long long>(p.n_slots) * p.Hkv > 0x7fffffffLL) return set_error(kErrBadShape, "prefill_attn: too many query blocks");
  const cudaError_t le = launch_early(kernel, grid, kT2Threads, smem, stream, p, map_q, map_k, map_v, map_o, map_kc, map_vc);
  g_launches.fetch_add(1);
  return check_cuda(le != cudaSuccess ? le : cudaGetLastError(), "prefill_attn(tc2) launch");
}

}  // namespace b200
