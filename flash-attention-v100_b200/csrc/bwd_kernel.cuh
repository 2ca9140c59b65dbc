// Backward attention kernel for sm_100a: fused dK / dV / dQ.
//
// Replaces fused_mha_backward_kernel of the reference (kernel/fused_mha_kernel.cu:325-735):
// the same identities  P = exp(scale*S - lse),  dV = P^T dO,  dP = dO V^T,
// dS = P o (dP - D) * scale,  dQ = dS K,  dK = dS^T Q  (kernel/fused_mha_kernel.cu:453-458,
// 503-506), with dQ accumulated in fp32 instead of the reference's fp16 atomics (:543,693).
//
// A work item is one 128-row KV tile of one (batch, head) and the query tiles (128 rows) that can
// see it.  A CTA stays on its SM and takes item after item (cluster launch control; deterministic, a counter).
// Everything is computed TRANSPOSED so that the KV rows sit on the 128 tensor-memory lanes, which lets P^T feed the
// dV MMA straight from tensor memory:
//
//   S^T  = K  Q_i^T    (A = K  smem K-major,  B = Q_i  smem K-major)      -> TMEM [0,128)
//   dP^T = V  dO_i^T   (A = V  smem K-major,  B = dO_i smem K-major)      -> TMEM [128,256)
//   dV  += P^T dO_i    (A = P^T TMEM fp16 over S^T, B = dO_i smem MN-major)-> TMEM [256+D, ..)
//                      (P^T: each compute group's packed columns at the start of its own part of S^T)
//   dK  += dS^T Q_i    (A = dS^T smem K-major, B = Q_i smem MN-major)      -> TMEM [256, 256+D)
//   dQ_i = dS  K       (A = dS^T smem read MN-major, B = K smem MN-major)  -> TMEM [128,128+D)
//                      (aliases dP^T, which is dead once dS^T is in shared memory)
//
//   compute groups  two of four warps, four at D = 64: one thread per KV row, group g owns 128 / groups query
//                   columns of the tile: P^T = exp2(S^T*c - lse2) and dS^T = P^T o (dP^T - D)
//   dQ group        four warps, one thread per query row; tensor memory -> registers ->
//                   shared-memory staging -> TMA reduce-add into the fp32 dQ accumulator
//                   (bulk async adds: no per-thread atomics in the load/store pipeline); at the end of an
//                   item dV and dK the same way, as 16-bit stores
//   producer warp   TMA (K, V once; Q_i through a ring of two slots, four at D = 64, dO_i through one) and
//                   source of the items
//   MMA warp        the whole warp runs the loop, one elected lane issues
//
// The per-row statistics come from the workspace the preprocess kernel fills, negated (they are
// added): lse2 = lse * log2(e) (+inf on padding rows) and delta = rowsum(dO o O) (0 on padding rows),
// both padded to a multiple of 128 rows per (batch, head); a tile's 2 x 128 values come in with Q_i.
//
// What bounds it at D = 128: the SM's port towards L2, and the power cap.  Per query tile there are 2560 clk of MMA
// and 64 KB of fp32 reduce-adds, which take 3000 clk through the port (about 20 bytes/clk; it is active 81 % of the
// time at Z8 H32 N2048 causal, the tensor pipe 62 %), in a period of 3700 to 3900.  At D = 64 (port 43 %, tensor
// pipe 31 %) it is a chain: P^T, wait, dS^T, wait.
// The end of an item costs extra: 4000 clk of loads that come in late, and 64 KB of dK and dV through the same port.
// Hence the first S^T of the next item is issued behind the last dQ and dK, for its K comes late, and dK and dV are
// written by the dQ group, which is idle there.  Against S^T ahead of them, dK and dV written by the compute groups
// behind P^T, a prefetch of K, V and dO towards L2, and at D = 64 eight compute warps of 64 columns instead of
// sixteen of 32, all together, whole backward, us: Z64 H16 N512 D64 bf16 363 -> 323, Z4 H16 N1024 D64 causal 51 -> 46,
// Z2 H16 N8192 D64 causal 914 -> 860, Z8 H32 N2016 D128 bf16 without a mask 1481 -> 1432, causal 954 -> 904, D96
// 838 -> 760.  The warps alone: Z2 H16 N8192 D64 causal 909 -> 888, Z64 H16 N512 345 -> 342.  With the prefetch again:
// D = 64 no difference, D = 96 and 128 0 to 4 % slower (it shares the unit with the loads it is meant to help).
// The instruction cache decides more than it seems: with MMA loops and write-outs unrolled the same kernel fetched
// 1.7 times the instructions from behind the first-level cache and ran 5-18 % SLOWER than one CTA per item, rolled up
// 5-10 % faster.  Hence the loops below.  At D = 128 shorter periods alone (sixteen compute warps there, too: -10 %) do
// not shorten the time, the clock falls instead: the power cap.
#pragma once
#include <cuda.h>
#include <math_constants.h>

#include <type_traits>

#include "aux_kernels.cuh"
#include "ptx.cuh"

namespace fmha {

struct BwdKernelParams {
  const float* neg_lse2;  // fp32 (Z*H, seqlen_q_pad)
  const void* neg_delta;  // (Z*H, seqlen_q_pad): fp32 with bf16 tensors, else fp16
  float* dk_accum;      // optional fp32 (Z, seqlen_k, H, D) contiguous: tm_dk then describes it
  float* dv_accum;      // optional
  long long accum_batch_stride;  // elements between batch entries of dk_accum / dv_accum
  int accum_overwrite;  // 1: dK / dV REPLACE what dk_accum / dv_accum hold (FMHA_BWD_ACCUM_OVERWRITE)
  int heads, seqlen_q, seqlen_k, seqlen_q_pad;
  int num_kv_blocks;    // ceil(seqlen_k / 128)
  int num_heads_total;  // batch * heads
  int head_group;       // heads whose CTAs are interleaved in the grid (>= 1)
  int q_tile_begin;     // query tiles before this one take no part (FmhaBwdParams.q_row_begin / 128)
  int deal;             // 1: every block has the one item of its index; 0: cluster launch control (dq_order: neither)
  uint16_t *dk, *dv;    // 16-bit outputs (element strides), for KV tiles that no query sees
  Strides3 dk_strides, dv_strides;
  float scale, scale_log2;
  int causal, causal_shift;
  int* status;
  // Deterministic dQ (not NULL): one word per (batch*head, query tile), zero at launch.  The
  // CTAs that add into a query tile's dQ take turns (bwd_turn): a CTA waits for the word to reach
  // its turn, adds, and once its adds have completed sets turn + 1.  The fp32 additions then
  // happen in one fixed order and dQ is the same bits on every run.
  // The first two of them are the halves of word 0, for word 1 counts the items that have been handed out (the
  // workspace has no other room, and its size is part of the ABI).
  unsigned* dq_order;
  int num_items;
  // optional per-batch lengths (right-padded batches), see FmhaBwdParams
  const int* seqused_q;
  const int* seqused_k;
  long long* timeline;  // debug builds (-DFMHA_TIMELINE) only
  int timeline_block;
};

template <int D, bool kBf16 = false, int DR = D>
struct BwdTraits {
  static constexpr int kBlock = 128;
  static constexpr int kBoxes = D / 64;
  static constexpr int kBoxBytes = 128 * 128;
  static constexpr int kTileBytes = kBoxes * kBoxBytes;  // a 128 x D fp16 tile
  static constexpr int kDsBytes = 2 * kBoxBytes;         // dS^T: 128 x 128 fp16
  // Tile slots.  K, V and dO are in slots 0-2 and change places from item to item (see the kernel);
  // the slots behind them take the query tiles in turn.  Where there is room for four (D = 64), a query tile's
  // load need not wait for dK of the tile two before: behind the reduce-adds of dQ, which go through the
  // same unit, it came too late for its S^T.  Whole backward, us, two slots / four: Z64 H16 N512 no mask, bf16
  // 379 / 353, Z4 H16 N1024 causal 55.6 / 53.4, Z2 H16 N8192 no mask, bf16 1680 / 1601.  (Room is left at D = 64 for a
  // second K and a second dO: Z64 H16 N512 no mask, bf16 334 -> 327, but Z2 H16 N8192 causal 875 -> 922.)
  static constexpr int kQSlots = D == 64 ? 4 : 2;
  static constexpr int kSlots = 3 + kQSlots;
  static constexpr int kStageBytes = 2 * 16384;          // dQ staging: 2 x (128 rows x 32 fp32)
  // statistics of one query tile: -lse2[128] (fp32), -delta[128] (fp32 with bf16 tensors, else fp16)
  static constexpr int kDeltaBytes = kBf16 ? 512 : 256;
  static constexpr int kStatBytes = 512 + kDeltaBytes;
  static constexpr int kItemStages = 4;                  // item ids published ahead

  // Warps: compute groups of four, the dQ group, {producer, MMA issuer, two that only take part in barriers}.
  static constexpr int kGroups = D == 64 ? 4 : 2;   // compute groups
  static constexpr int kCols = 128 / kGroups;       // query columns each owns
  static constexpr int kComputeWarps = 4 * kGroups;
  static constexpr int kProducerWarp = kComputeWarps + 4, kMmaWarp = kProducerWarp + 1;
  static constexpr int kThreads = 32 * (kComputeWarps + 8);
  // Registers per thread: of the launch, and after setmaxnreg
  static constexpr int kRegs = D == 64 ? 80 : 128;
  static constexpr int kRegsIssue = 80, kRegsCompute = D == 64 ? 72 : 128;
  static constexpr int kRegsDq = kRegs + (kRegs - kRegsIssue) + kGroups * (kRegs - kRegsCompute);
  static_assert(kThreads * kRegs <= 65536 && kRegsIssue <= kRegs && kRegsCompute <= kRegs && kRegsDq >= kRegs &&
                    kRegsIssue % 8 == 0 && kRegsCompute % 8 == 0 && kRegsDq % 8 == 0,
                "setmaxnreg.dec must not raise and .inc must not lower the registers of the launch");
  static constexpr int kTmemCols = 512;
  static constexpr int kColS = 0, kColDP = 128, kColDQ = 128, kColDK = 256, kColDV = 256 + D;
  static constexpr uint32_t kIdescST = umma_idesc_f16(128, 128, 0, 0, kBf16);  // S^T, dP^T
  static constexpr uint32_t kIdescDV = umma_idesc_f16(128, DR, 0, 1, kBf16);   // dV, dK
  static constexpr uint32_t kIdescDQ = umma_idesc_f16(128, DR, 1, 1, kBf16);   // dQ
};

// A work item: one KV tile of one (batch, head) and the query tiles that see it.  The producer warp
// works it out and publishes it in shared memory.
struct __align__(16) BwdItem {
  int id;       // -1: no more items
  int cnt;      // query tiles to walk (0: dK and dV of this KV tile are zeros)
  int i_begin;  // the first of them
  int kb;       // KV tile
  int z, h, zh;
  int sk;       // keys of the batch entry
};

// what the roles share beside the tiles, at the end of the dynamic shared memory
template <int D, bool kBf16>
struct __align__(16) BwdControl {
  using T = BwdTraits<D, kBf16>;
  uint8_t clc_word[16];  // the answer to the last request for an item
  BwdItem items[T::kItemStages];
  uint64_t bar_clc, bar_item_full[T::kItemStages], bar_item_empty[T::kItemStages];
  uint64_t bar_full[T::kSlots], bar_empty[T::kSlots];  // per tile slot
  uint64_t bar_s_full, bar_dp_full, bar_p_ready, bar_ds_ready, bar_dq_full, bar_dq_empty;
  uint64_t bar_acc_full;               // dK and dV of an item are complete
  uint64_t bar_dv_read, bar_dk_read;   // ... and have been read out of tensor memory
  uint32_t tmem_base;
  int abort_word;
  int skip_cta;
};

template <int D, bool kBf16>
constexpr int bwd_smem_bytes() {
  using T = BwdTraits<D, kBf16>;
  return T::kSlots * T::kTileBytes + T::kDsBytes + T::kStageBytes + T::kQSlots * T::kStatBytes +
         (int)sizeof(BwdControl<D, kBf16>);
}

// Heads are taken in groups of head_group; within a group the items are ordered by KV tile first
// (early KV tiles see the most query tiles under a causal mask and take longest), head second: the
// items in work at any time still belong to a handful of heads (their Q / dO tiles and dQ
// accumulators stay in L2), and what comes last, at the end of a group and of the grid, are the
// short ones.  head_group = 1: all items of a head in a row.
template <bool kDet>
__device__ __forceinline__ BwdItem bwd_item(const BwdKernelParams& p, int id) {
  BwdItem it;
  it.id = id;
  const int per_group = p.head_group * p.num_kv_blocks;
  const int group = id / per_group, within = id % per_group;
  const int heads_here = min(p.head_group, p.num_heads_total - group * p.head_group);
  it.zh = group * p.head_group + within % heads_here;
  it.kb = within / heads_here;
  if (kDet && p.causal) it.kb = p.num_kv_blocks - 1 - it.kb;  // see bwd_turn
  it.z = it.zh / p.heads;
  it.h = it.zh % p.heads;
  // the lengths that count for this batch entry: query tiles and keys beyond them are padding
  const int sq = p.seqused_q == nullptr ? p.seqlen_q : max(0, min(p.seqlen_q, __ldg(p.seqused_q + it.z)));
  it.sk = p.seqused_k == nullptr ? p.seqlen_k : max(0, min(p.seqlen_k, __ldg(p.seqused_k + it.z)));
  const int nq_tiles = (sq + 127) / 128;
  int i_begin = 0;
  if (p.causal) {
    // query row r sees key kv0 iff r + shift >= kv0
    const long long first_row = (long long)it.kb * 128 - p.causal_shift;
    i_begin = first_row <= 0 ? 0 : (int)min((long long)nq_tiles, first_row / 128);
  }
  it.i_begin = max(i_begin, p.q_tile_begin);
  // a KV tile that is all padding walks no query tile
  it.cnt = it.kb * 128 < it.sk ? max(0, nq_tiles - it.i_begin) : 0;
  return it;
}

// Deterministic dQ: the turn of an item's KV tile among those that add into a query tile.  An item only
// ever waits for items with lower indices.  A CTA draws every item, the first one too, from one counter (draw), and
// works through its items in the order in which it drew them.  So of the items that are not done the one with the
// lowest index waits for nobody, and is in work or drawn next, whatever the order in which blocks start.  (Half a
// word holds a turn modulo 2^16, which is enough: of the items drawn only a handful per CTA are not done.)
// Cluster launch control, by which the other mode takes items over, promises no order; an item per CTA, in the order
// of the block indices, relied on their being started in that order.  Whole backward, us, an item per CTA / by cluster
// launch control / drawn, bf16: Z2 H16 N2048 D128 causal 199 / 185 / 190 (the first draw, and which SMs get the first
// items), without a mask 313 / 297 / 292, Z8 H32 N2016 causal 1350 / 1224 / 1243, Z64 H16 N512 causal 618 / 608 / 545,
// D64 without a mask 558 / 500 / 468, Z1 H40 N640 without a mask 71 / 82 / 69; 126 shapes 1 / 1.055 / 1.073 times as
// fast.
// Without a mask: KV tile after KV tile, and the items of a head run staggered by one query tile each.
// Under a causal mask: from the diagonal downwards, and the items of a head are dispatched in that order.
// The item on the diagonal comes first to its query tile, the one below it a tile later, and so on: no item
// waits that has not been held up itself.  (In ascending order the item of KV tile kb had to wait for all kb
// before it when it came to its first query tile.  Whole backward, us, ascending / so: Z2 H16 N2048 D128 257 / 202,
// Z8 H32 N2048 D128 1757 / 1284, Z1 H8 N16384 D128 4289 / 2182, Z4 H16 N1024 D64 137 / 97.)
__device__ __forceinline__ int bwd_turn(const BwdKernelParams& p, const BwdItem& it, int tile) {
  if (!p.causal) return it.kb;
  const long long diagonal = ((long long)(tile + 1) * 128 + p.causal_shift - 1) / 128;  // last KV tile it sees
  return (int)min(diagonal, (long long)(it.sk - 1) / 128) - it.kb;
}

// DR <= D: elements per row of the tensors.  96 runs on the tiles of D = 128: the tile loads fill columns
// 96-127 with zeros, the MMAs leave them out (six steps instead of eight, N = 96 instead of 128), columns 96-127 of
// dQ, dK and dV do not exist (what the write-out reads there is clipped by the store), and the fp32 buffers have DR
// elements per row.  Z8 H32 N2048 D96 causal, fp16, forward and backward, the zeros multiplied too / left out: 1206 /
// 1165 us (the tensor cores spend little power on zeros, and it is the power cap that bounds both).
// kDet: deterministic dQ.  An instantiation of its own: the turns cost the other mode
// 1 to 3 % when they were a branch in the dQ group's loop.
template <int D, bool kBf16 = false, int DR = D, bool kDet = false>
__global__ void __launch_bounds__(BwdTraits<D, kBf16, DR>::kThreads, 1)
    fmha_bwd_kernel(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_k,
                    const __grid_constant__ CUtensorMap tm_v, const __grid_constant__ CUtensorMap tm_do,
                    const __grid_constant__ CUtensorMap tm_dk, const __grid_constant__ CUtensorMap tm_dv,
                    const __grid_constant__ CUtensorMap tm_dqacc, const BwdKernelParams p) {
  using T = BwdTraits<D, kBf16, DR>;
  // (no static shared memory: the tiles need every byte, and 1024-byte alignment)
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  const uint32_t smem_base = smem_u32(smem_raw);
  const uint32_t ds_smem = smem_base + T::kSlots * T::kTileBytes;   // dS^T
  const uint32_t stg_smem = ds_smem + T::kDsBytes;                  // staging of dQ, dK and dV, 2 x 16 KB
  const uint32_t stat_smem = stg_smem + T::kStageBytes;             // statistics, one block per query slot
  auto& sh = *reinterpret_cast<BwdControl<D, kBf16>*>(smem_raw + T::kSlots * T::kTileBytes + T::kDsBytes +
                                                      T::kStageBytes + T::kQSlots * T::kStatBytes);
  volatile int* const abort_word = &sh.abort_word;

  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0);  // warp-uniform for the compiler, too
  const int lane = threadIdx.x & 31;

  auto draw = [&]() -> unsigned { return atomicAdd(p.dq_order + 1, 1u); };
  // the first item (drawn ahead of the set-up: the answer takes a while)
  unsigned first_id = blockIdx.x;
  if (kDet && threadIdx.x == T::kProducerWarp * 32) first_id = draw();

  if (threadIdx.x == 0) {
    sh.skip_cta = (p.status != nullptr && *reinterpret_cast<volatile int*>(p.status) != 0) ? 1 : 0;
    sh.abort_word = 0;
  }
  __syncthreads();
  if (sh.skip_cta) return;

  // one tile into its slot; a query tile brings its lse2 and delta along
  auto send = [&](int slot, const CUtensorMap* tm, const BwdItem& it, int row, bool is_q) {
    if (elect_one()) {
      const uint32_t bar = smem_u32(&sh.bar_full[slot]);
      mbar_arrive_expect_tx(bar, T::kTileBytes + (is_q ? T::kStatBytes : 0));
#pragma unroll
      for (int b = 0; b < T::kBoxes; ++b)
        tma_load_4d(smem_base + slot * T::kTileBytes + b * T::kBoxBytes, tm, bar, b * 64, row, it.h, it.z);
      if (is_q) {
        const uint32_t st = stat_smem + (slot - 3) * T::kStatBytes;
        const size_t at = (size_t)it.zh * p.seqlen_q_pad + row;
        bulk_load(st, p.neg_lse2 + at, 512, bar);
        bulk_load(st + 512, static_cast<const char*>(p.neg_delta) + at * (T::kDeltaBytes / 128), T::kDeltaBytes, bar);
      }
    }
    __syncwarp();
  };

  // The producer warp sets the barriers up itself and sends the first tiles of its first item off at
  // once, before the CTA-wide barrier below that waits for the tensor-memory allocation.
  if (warp == T::kProducerWarp) {
    if (lane == 0) {
      mbar_init(smem_u32(&sh.bar_clc), 1);
      for (int s = 0; s < T::kItemStages; ++s) {
        mbar_init(smem_u32(&sh.bar_item_full[s]), 1);
        mbar_init(smem_u32(&sh.bar_item_empty[s]), 5 + T::kComputeWarps);  // MMA warp, four dQ warps
      }
      for (int s = 0; s < T::kSlots; ++s) {
        mbar_init(smem_u32(&sh.bar_full[s]), 1);
        mbar_init(smem_u32(&sh.bar_empty[s]), 1);
      }
      mbar_init(smem_u32(&sh.bar_s_full), 1);
      mbar_init(smem_u32(&sh.bar_dp_full), 1);
      mbar_init(smem_u32(&sh.bar_p_ready), T::kComputeWarps);  // one arrival per warp
      mbar_init(smem_u32(&sh.bar_ds_ready), T::kComputeWarps);
      mbar_init(smem_u32(&sh.bar_dq_full), 1);
      mbar_init(smem_u32(&sh.bar_dq_empty), 4);
      mbar_init(smem_u32(&sh.bar_acc_full), 1);
      mbar_init(smem_u32(&sh.bar_dv_read), 4);
      mbar_init(smem_u32(&sh.bar_dk_read), 4);
      fence_barrier_init();
    }
    __syncwarp();
    first_id = __shfl_sync(0xffffffffu, first_id, 0);
    BwdItem it;
    it.cnt = 0;
    if (first_id < (unsigned)p.num_items) it = bwd_item<kDet>(p, first_id);
    if (it.cnt > 0) {
      const int row0 = it.i_begin * T::kBlock;
      send(3, &tm_q, it, row0, true);
      send(0, &tm_k, it, it.kb * T::kBlock, false);
      send(1, &tm_v, it, it.kb * T::kBlock, false);
      send(2, &tm_do, it, row0, false);
    }
  }
  if (warp == T::kMmaWarp) {
    tmem_alloc(smem_u32(&sh.tmem_base), T::kTmemCols);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = __shfl_sync(0xffffffffu, sh.tmem_base, 0);

  // The next item published by the producer warp (every consuming warp keeps its own count); id = -1
  // when there is none, and when a wait ran out.
  uint32_t item_cnt = 0;
  auto take_item = [&]() -> BwdItem {
    const uint32_t s = item_cnt % T::kItemStages;
    BwdItem it;
    if (mbar_wait_warp(smem_u32(&sh.bar_item_full[s]), (item_cnt / T::kItemStages) & 1, abort_word, 16)) {
      it = sh.items[s];
      it.id = __shfl_sync(0xffffffffu, it.id, 0);  // warp-uniform for the compiler
      it.cnt = __shfl_sync(0xffffffffu, it.cnt, 0);
    } else {
      it.id = -1;
      it.cnt = 0;
    }
    __syncwarp();
    if (lane == 0) mbar_arrive(smem_u32(&sh.bar_item_empty[s]));
    ++item_cnt;
    return it;
  };

  // Register budget: the producer / MMA warpgroup and, at D = 64, the
  // compute warpgroups hand part of their share to the dQ warpgroup, which must hold a whole
  // dQ row per thread to drain tensor memory in one go (the next dP^T waits for
  // those columns).  Each setmaxnreg sits at the top of its warpgroup's own branch: the
  // compiler budgets registers per region only when the instruction dominates the region.
  if (warp >= T::kProducerWarp) {
    reg_dealloc<T::kRegsIssue>();
    // Slots of the running item's K, V and dO.  At the end of an item they fall free in the order
    // V (after the last dP^T), dO (after the last dV), K (after the last dQ), and the next item
    // needs K first, V and dO a while later: it takes them over in that order.
    int slot_k = 0, slot_v = 1, slot_do = 2;
    auto next_slots = [&]() {
      const int k = slot_k;
      slot_k = slot_v;
      slot_v = slot_do;
      slot_do = k;
    };
    if (warp == T::kProducerWarp) {
      // =========================== TMA producer, item source ===========================
      bool ok = true;
      uint32_t published = 0, asked = 0;
      bool pending = false;  // a request is out
      [[maybe_unused]] unsigned drawn = 0;
      auto ask = [&]() {
        if constexpr (kDet) {
          if (!pending && lane == 0) drawn = draw();
          pending = true;
          return;
        }
        if (p.deal || pending) return;
        if (elect_one()) {
          fence_proxy_async_smem();  // the last answer has been read
          mbar_arrive_expect_tx(smem_u32(&sh.bar_clc), 16);
          clc_request(smem_u32(sh.clc_word), smem_u32(&sh.bar_clc));
        }
        __syncwarp();
        pending = true;
      };
      // a KV tile without query tiles: zeros.  They are written here, so that only
      // items with query tiles to walk are published
      auto write_zeros = [&](const BwdItem& it) {
        const int rows = min(T::kBlock, p.seqlen_k - it.kb * T::kBlock);
        for (int which = 0; which < 2; ++which) {
          float* accum = which ? p.dk_accum : p.dv_accum;
          const uint4 zero = make_uint4(0, 0, 0, 0);
          if (accum != nullptr) {
            if (p.accum_overwrite == 0) continue;
            float* dst = accum + (size_t)it.z * p.accum_batch_stride +
                         ((size_t)it.kb * T::kBlock * p.heads + it.h) * DR;
            for (int i = lane; i < rows * (DR / 4); i += 32)
              *reinterpret_cast<uint4*>(dst + (size_t)(i / (DR / 4)) * p.heads * DR + (i % (DR / 4)) * 4) = zero;
          } else {
            const Strides3& s = which ? p.dk_strides : p.dv_strides;
            uint16_t* dst = (which ? p.dk : p.dv) + it.z * s.batch + (long long)it.kb * T::kBlock * s.row + it.h * s.head;
            for (int i = lane; i < rows * (DR / 8); i += 32)
              *reinterpret_cast<uint4*>(dst + (i / (DR / 8)) * s.row + (i % (DR / 8)) * 8) = zero;
          }
        }
      };

      // finds the next item with query tiles to walk and publishes it
      int id = -1;
      bool first = true;  // the block's own item comes first
      auto next_item = [&]() -> BwdItem {
        BwdItem it;
        for (;; first = false) {
          if (first) {
            id = first_id < (unsigned)p.num_items ? (int)first_id : -1;
          } else if (kDet) {
            ask();
            pending = false;
            id = drawn < (unsigned)p.num_items ? (int)drawn : -1;
          } else if (p.deal) {
            id = -1;
          } else {
            ask();
            ok = mbar_wait_warp(smem_u32(&sh.bar_clc), asked & 1, abort_word, 17);
            ++asked;
            pending = false;
            id = ok ? clc_answer(smem_u32(sh.clc_word)) : -1;
          }
          id = __shfl_sync(0xffffffffu, id, 0);
          it.id = -1;
          it.cnt = 0;
          if (id < 0) break;
          it = bwd_item<kDet>(p, id);
          it.cnt = __shfl_sync(0xffffffffu, it.cnt, 0);
          if (it.cnt > 0) break;
          ask();
          write_zeros(it);
        }
        const uint32_t s = published % T::kItemStages, round = published / T::kItemStages;
        if (round > 0 && !mbar_wait_warp(smem_u32(&sh.bar_item_empty[s]), (round - 1) & 1, abort_word, 18)) ok = false;
        if (ok && lane == 0) {
          sh.items[s] = it;
          mbar_arrive(smem_u32(&sh.bar_item_full[s]));
        }
        __syncwarp();
        ++published;
        if (!ok) it.id = -1;
        return it;
      };
      uint32_t used = 0;  // bit s: loads into slot s so far, modulo 2
      auto load = [&](int slot, const CUtensorMap* tm, const BwdItem& it, int row, bool is_q) {
        ok = ok && mbar_wait_warp(smem_u32(&sh.bar_empty[slot]), ((used >> slot) & 1) ^ 1, abort_word, 1);
        if (ok) send(slot, tm, it, row, is_q);
        used ^= 1u << slot;
      };
      uint32_t g = 0;  // query tiles so far, over all items
      // The answer to a request takes a microsecond, so it is asked for ahead of the item's last loads.  How far makes
      // little difference: two tiles ahead take 0.99 to 1.01 times as long as one, over 52 shapes at each D, and 1.02 at
      // Z4 H16 N1024 causal, where asking later balances better.  Deterministic, the items of a head end one after the
      // other, and the first to end has to be the first to ask: not ahead (two ahead / one / none, us: Z64 H16 N512 D128
      // bf16 causal 592 / 529 / 517, Z1 H40 N640 without a mask 75.5 / 68.0 / 67.8; 126 shapes 1.018 / 1.003 / 1).
      constexpr int kAskAhead = kDet ? 0 : T::kQSlots > 2 ? 1 : 2;
      while (ok) {
        const BwdItem it = next_item();
        if (it.id < 0) break;
        const int row0 = it.i_begin * T::kBlock, kv0 = it.kb * T::kBlock;
        if (first) {
          used = 0xf;  // sent off during the set-up
          first = false;
        } else {
          if (published > 1) next_slots();
          // in the order in which the slots fall free
          load(3 + g % T::kQSlots, &tm_q, it, row0, true);
          load(slot_k, &tm_k, it, kv0, false);
          load(slot_v, &tm_v, it, kv0, false);
          load(slot_do, &tm_do, it, row0, false);
        }
        ++g;
        if (it.cnt <= kAskAhead) ask();
#pragma unroll 1
        for (int n = 1; ok && n < it.cnt; ++n, ++g) {
          const int row = (it.i_begin + n) * T::kBlock;
          if (n >= it.cnt - kAskAhead) ask();
          load(3 + g % T::kQSlots, &tm_q, it, row, true);
          load(slot_do, &tm_do, it, row, false);
        }
      }
    } else if (warp == T::kMmaWarp) {
      // =========================== MMA issuer (converged warp) ===========================
      // D (+)= A B with A and B in shared memory, the contraction in blocks of 64.  Loops, not straight
      // code: what the roles of the CTA execute has to fit the instruction cache together.
      auto issue_ss = [&](int blocks, uint32_t d_col, uint32_t a_lo, uint32_t a_block, uint32_t a_step, uint32_t b_lo,
                          uint32_t b_block, uint32_t b_step, uint32_t idesc, uint32_t accumulate) {
#pragma unroll 1
        for (int b = 0; b < blocks; ++b) {
#pragma unroll
          for (int i = 0; i < 4; ++i)
            umma_ss_elect(tmem_base + d_col, a_lo + i * a_step, b_lo + i * b_step, idesc, i > 0 ? 1u : accumulate);
          a_lo += a_block;
          b_lo += b_block;
          accumulate = 1u;
        }
      };
      // steps of 16 along the contraction and blocks of 64, in descriptor units
      constexpr uint32_t kStepK = 32 >> 4, kBlockK = T::kBoxBytes >> 4;  // K-major operand
      constexpr uint32_t kStepMn = 2048 >> 4, kBlockMn = 4 * kStepMn;    // MN-major operand
      // C[128 x 128] = A[128 x DR] B[128 x DR]^T, both K-major
      auto issue_kmajor = [&](uint32_t d_col, uint32_t a_addr, uint32_t b_addr) {
        uint32_t a_lo = umma_desc_lo(a_addr, kLboKMajor), b_lo = umma_desc_lo(b_addr, kLboKMajor);
        if constexpr (DR % 64 == 0) {
          issue_ss(T::kBoxes, d_col, a_lo, kBlockK, kStepK, b_lo, kBlockK, kStepK, T::kIdescST, 0u);
        } else {  // 96: six steps, two at a time, the last two in the second box
#pragma unroll 1
          for (int b = 0; b < DR / 32; ++b) {
#pragma unroll
            for (int i = 0; i < 2; ++i)
              umma_ss_elect(tmem_base + d_col, a_lo + i * kStepK, b_lo + i * kStepK, T::kIdescST, b + i > 0 ? 1u : 0u);
            const uint32_t step = b == 0 ? 2 * kStepK : kBlockK - 2 * kStepK;
            a_lo += step;
            b_lo += step;
          }
        }
      };
      auto slot_addr = [&](int slot) { return smem_base + slot * T::kTileBytes; };
      uint32_t filled = 0;  // bit s: fills of slot s waited for so far, modulo 2
      auto wait_full = [&](int slot, int who) {
        const bool got = mbar_wait_warp(smem_u32(&sh.bar_full[slot]), (filled >> slot) & 1, abort_word, who);
        filled ^= 1u << slot;
        return got;
      };
      const uint32_t ds_lo_k = umma_desc_lo(ds_smem, kLboKMajor);    // dS^T as K-major A (dK)
      const uint32_t ds_lo_mn = umma_desc_lo(ds_smem, kLboMnMajor);  // dS^T read as MN-major A (dQ)

      uint32_t g = 0;  // query tiles so far, over all items
      bool ok = true;
#pragma unroll 1
      for (uint32_t item_no = 0; ok; ++item_no) {
        // S^T of the item's first query tile.  It comes behind dQ and dK of the item before: K and Q come late more
        // often than not, and what is left of the item before would wait for them.
        const BwdItem cur = take_item();
        if (cur.id < 0) break;
        if (item_no > 0) next_slots();
        if (!wait_full(slot_k, 3) || !wait_full(3 + g % T::kQSlots, 4)) break;
        tc_fence_after();
        issue_kmajor(T::kColS, slot_addr(slot_k), slot_addr(3 + g % T::kQSlots));
        umma_commit_elect(smem_u32(&sh.bar_s_full));
#pragma unroll 1
        for (int n = 0; ok && n < cur.cnt; ++n, ++g) {
          const bool last = n == cur.cnt - 1;
          // ---- dP^T of this query tile (its columns hold dQ of the one before until the dQ group read it)
          FMHA_TL(2, g, 0);
          ok = (n > 0 || wait_full(slot_v, 5)) && wait_full(slot_do, 9) &&
               (g == 0 || mbar_wait_warp(smem_u32(&sh.bar_dq_empty), (g - 1) & 1, abort_word, 10));
          if (!ok) break;
          tc_fence_after();
          FMHA_TL(2, g, 1);
          issue_kmajor(T::kColDP, slot_addr(slot_v), slot_addr(slot_do));
          umma_commit_elect(smem_u32(&sh.bar_dp_full));
          if (last) umma_commit_elect(smem_u32(&sh.bar_empty[slot_v]));
          // ---- dV += P^T dO_i; the first one overwrites the last item's dV
          FMHA_TL(2, g, 2);
          ok = (n > 0 || item_no == 0 ||
                mbar_wait_warp(smem_u32(&sh.bar_dv_read), (item_no - 1) & 1, abort_word, 19)) &&
               mbar_wait_warp(smem_u32(&sh.bar_p_ready), g & 1, abort_word, 6);
          if (!ok) break;
          tc_fence_after();
          FMHA_TL(2, g, 3);
          const uint32_t do_lo_mn = umma_desc_lo(slot_addr(slot_do), kLboMnMajor);  // dO as MN-major B
#pragma unroll 1
          for (int b = 0; b < 2; ++b)
#pragma unroll
            for (int i = 0; i < 4; ++i)
              umma_ts_elect(tmem_base + T::kColDV,
                            tmem_base + T::kColS + b * 64 + (T::kGroups == 2 ? i * 8 : (i >> 1) * 32 + (i & 1) * 8),
                            do_lo_mn + b * kBlockMn + i * kStepMn, T::kIdescDV, (n > 0 || b > 0 || i > 0) ? 1u : 0u);
          umma_commit_elect(smem_u32(&sh.bar_empty[slot_do]));
          // ---- S^T of the item's next query tile (the S region is free once dV has read P^T)
          if (!last) {
            if (!(ok = wait_full(3 + (g + 1) % T::kQSlots, 7))) break;
            tc_fence_after();
            issue_kmajor(T::kColS, slot_addr(slot_k), slot_addr(3 + (g + 1) % T::kQSlots));
            umma_commit_elect(smem_u32(&sh.bar_s_full));
          }
          // ---- dQ_i = dS K first (its read-out is on the critical path), then dK += dS^T Q_i
          FMHA_TL(2, g, 4);
          if (!(ok = mbar_wait_warp(smem_u32(&sh.bar_ds_ready), g & 1, abort_word, 8))) break;
          tc_fence_after();
          FMHA_TL(2, g, 5);
          const uint32_t k_lo_mn = umma_desc_lo(slot_addr(slot_k), kLboMnMajor);  // K as MN-major B
          issue_ss(2, T::kColDQ, ds_lo_mn, kBlockMn, kStepMn, k_lo_mn, kBlockMn, kStepMn, T::kIdescDQ, 0u);
          umma_commit_elect(smem_u32(&sh.bar_dq_full));
          if (last) umma_commit_elect(smem_u32(&sh.bar_empty[slot_k]));
          if (n == 0 && item_no > 0) {
            if (!(ok = mbar_wait_warp(smem_u32(&sh.bar_dk_read), (item_no - 1) & 1, abort_word, 20))) break;
            tc_fence_after();
          }
          const uint32_t q_lo_mn = umma_desc_lo(slot_addr(3 + g % T::kQSlots), kLboMnMajor);
          issue_ss(2, T::kColDK, ds_lo_k, kBlockK, kStepK, q_lo_mn, kBlockMn, kStepMn, T::kIdescDV, n > 0 ? 1u : 0u);
          umma_commit_elect(smem_u32(&sh.bar_empty[3 + g % T::kQSlots]));  // Q_i, and dS^T, have been read
          if (last) umma_commit_elect(smem_u32(&sh.bar_acc_full));
          FMHA_TL(2, g, 6);
        }
      }
    }
  } else {
    const int quad = warp & 3;
    const int r = quad * 32 + lane;  // TMEM lane of this thread
    const uint32_t lane_addr = uint32_t(quad * 32) << 16;

    if (warp < T::kComputeWarps) {
      // =========================== compute groups: P^T, dS^T ===========================
      reg_dealloc<T::kRegsCompute>();
      const int cg = warp >> 2;           // query columns [cg * kCols, (cg + 1) * kCols) are this group's
      const uint64_t c2 = pack2f(p.scale_log2, p.scale_log2);
      const uint32_t tS = tmem_base + lane_addr + T::kColS + cg * T::kCols;
      // P^T (packed columns) goes over the start of this group's own part of S^T, which only
      // this group reads: no ordering between the groups is needed
      const uint32_t tP = tS;
      const uint32_t tDP = tmem_base + lane_addr + T::kColDP + cg * T::kCols;
      // this thread's 128-byte row of dS^T
      const uint32_t row_addr = ds_smem + (cg * T::kCols / 64) * T::kBoxBytes + r * 128;
      const int chunk0 = (cg * T::kCols % 64) / 8;  // this group's first 16-byte chunk of it
      const bool tl = (threadIdx.x == 0);
      uint32_t g = 0;
      for (;;) {
        const BwdItem it = take_item();
        if (it.id < 0) break;
        const int kvi = it.kb * T::kBlock + r;  // key of this thread
#pragma unroll 1
        for (int n = 0; n < it.cnt; ++n, ++g) {
          const int qbase = (it.i_begin + n) * T::kBlock;
          const uint32_t sb = stat_smem + g % T::kQSlots * T::kStatBytes;  // -lse2 at 0, -delta at 512

          // first visible query column of this thread's kCols (>= kCols: none)
          int first_visible = 0;
          if (kvi >= it.sk) {
            first_visible = T::kBlock;
          } else if (p.causal) {
            const long long fv = (long long)kvi - p.causal_shift - qbase;
            first_visible = fv <= 0 ? 0 : (int)min(fv, (long long)T::kBlock);
          }
          const int fvh = first_visible - cg * T::kCols;

          uint32_t pp[T::kCols / 2];  // P^T of this row and group, 16-bit pairs
          if (tl) FMHA_TL(0, g, 0);
          // on a time-out: keep going, every later wait returns at once
          mbar_wait(smem_u32(&sh.bar_full[3 + g % T::kQSlots]), g / T::kQSlots & 1, abort_word, 21);  // the statistics
          mbar_wait(smem_u32(&sh.bar_s_full), g & 1, abort_word, 11);
          tc_fence_after();
          if (tl) FMHA_TL(0, g, 1);
          {
            uint32_t s[T::kCols / 32][32];
#pragma unroll
            for (int cc = 0; cc < T::kCols / 32; ++cc) tmem_ld32(tS + cc * 32, s[cc]);
            tmem_wait_ld();
#pragma unroll
            for (int cc = 0; cc < T::kCols / 32; ++cc)
#pragma unroll
              for (int i = 0; i < 32; i += 4) {
                const float4 nl = lds128(sb + (cg * T::kCols + cc * 32 + i) * 4);
                uint32_t x[4];
                unpack2(fma2(pack2(s[cc][i + 0], s[cc][i + 1]), c2, pack2f(nl.x, nl.y)), x[0], x[1]);
                unpack2(fma2(pack2(s[cc][i + 2], s[cc][i + 3]), c2, pack2f(nl.z, nl.w)), x[2], x[3]);
                // (in fp32 for either type: a pair in fp16 takes the MUFU unit as long as two of these, and a
                // 16-bit argument costs P two to three digits)
#pragma unroll
                for (int k = 0; k < 2; ++k)
                  pp[cc * 16 + (i >> 1) + k] =
                      pack16x2<kBf16>(fast_exp2(__uint_as_float(x[2 * k])), fast_exp2(__uint_as_float(x[2 * k + 1])));
              }
            if (fvh > 0) {
#pragma unroll
              for (int j = 0; j < T::kCols / 2; ++j) {  // pair j = columns 2j, 2j+1 of this group's
                if (2 * j + 1 < fvh) pp[j] = 0u;
                else if (2 * j < fvh) pp[j] &= 0xffff0000u;
              }
            }
          }
          if constexpr (T::kCols == 64) tmem_st32(tP, pp);
          else tmem_st16(tP, pp);
          tmem_wait_st();
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(smem_u32(&sh.bar_p_ready));
          if (tl) FMHA_TL(0, g, 2);
          mbar_wait(smem_u32(&sh.bar_dp_full), g & 1, abort_word, 12);
          if (tl) FMHA_TL(0, g, 3);
          // dS^T of the previous tile has been read: its dQ and dK MMAs were issued before this dP^T, and the
          // commit that told of it covers them.
          tc_fence_after();
          if (tl) FMHA_TL(0, g, 4);
          {
            uint32_t dp[T::kCols / 32][32];
#pragma unroll
            for (int cc = 0; cc < T::kCols / 32; ++cc) tmem_ld32(tDP + cc * 32, dp[cc]);
            tmem_wait_ld();
#pragma unroll
            for (int cc = 0; cc < T::kCols / 32; ++cc)
#pragma unroll
              for (int k8 = 0; k8 < 4; ++k8) {  // 8 columns = one 16-byte chunk
                uint32_t w[4];
                // -delta of this chunk's 8 query columns: fp16 pairs, with bf16 (8 mantissa bits) pairs of fp32
                const uint32_t at = sb + 512 + (cg * T::kCols + cc * 32 + k8 * 8) * (kBf16 ? 4 : 2);
                const float4 a = lds128(at), b = kBf16 ? lds128(at + 16) : a;
                [[maybe_unused]] const uint64_t nd[4] = {pack2f(a.x, a.y), pack2f(a.z, a.w), pack2f(b.x, b.y),
                                                         pack2f(b.z, b.w)};
                [[maybe_unused]] const uint32_t nd16[4] = {__float_as_uint(a.x), __float_as_uint(a.y),
                                                           __float_as_uint(a.z), __float_as_uint(a.w)};
#pragma unroll
                for (int q2 = 0; q2 < 4; ++q2) {
                  const int i = k8 * 8 + q2 * 2;     // column within this 32-column block
                  const int j = cc * 16 + (i >> 1);  // its fp16 pair
                  if constexpr (kBf16) {
                    uint32_t lo, hi;
                    unpack2(mul2(pack2f(bf16_lo(pp[j]), bf16_hi(pp[j])), add2(pack2(dp[cc][i], dp[cc][i + 1]), nd[q2])),
                            lo, hi);
                    w[q2] = pack_bf16x2(__uint_as_float(lo), __uint_as_float(hi));
                  } else {
                    // P dP - P D, not P (dP - D): the difference may be beyond fp16 where P times it is not, and
                    // 0 times infinity would be NaN.  (In fp32, as above, the whole backward at D = 64 takes 3 to 8 %
                    // longer: Z64 H16 N512 causal 265 us, so; 277 in fp32.)
                    w[q2] = fma_half2(pp[j], pack_half2(__uint_as_float(dp[cc][i]), __uint_as_float(dp[cc][i + 1])),
                                      mul_half2(pp[j], nd16[q2]));
                  }
                }
                const int ch = chunk0 + cc * 4 + k8;  // chunk of this thread's 128-byte row
                sts128(row_addr + ((ch ^ (r & 7)) << 4), w[0], w[1], w[2], w[3]);
              }
          }
          fence_proxy_async_smem();
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(smem_u32(&sh.bar_ds_ready));
          if (tl) FMHA_TL(0, g, 5);
        }
      }
    } else {
      // =========================== dQ group: dQ; dV, dK ===========================
      reg_alloc<T::kRegsDq>();
      const uint32_t tDQ = tmem_base + lane_addr + T::kColDQ;
      const bool tl = (r == 0);
      constexpr int kChunks = DR / 32;  // 32-column chunks of a dQ row
      // an odd number of chunks per tile breaks the alternation of the two staging buffers by
      // chunk index: count the chunks staged so far instead
      [[maybe_unused]] uint32_t chunk_no = 0;
      uint32_t g = 0, drained = 0;
      for (;;) {
        const BwdItem it = take_item();
        if (it.id < 0) break;
#pragma unroll 1
        for (int n = 0; n < it.cnt; ++n, ++g) {
          const int tile = it.i_begin + n;
          if (tl) FMHA_TL(1, g, 0);
          // on a time-out keep going (like the compute groups): every later wait returns at once,
          // and all 128 threads still meet at the named barriers
          mbar_wait(smem_u32(&sh.bar_dq_full), g & 1, abort_word, 14);
          tc_fence_after();
          if (tl) FMHA_TL(1, g, 1);
          // The whole dQ row goes to registers first so that the dQ columns are released to the
          // next dP^T as early as possible; then 32-column chunks go out through shared memory.
          uint32_t acc[kChunks][32];
#pragma unroll
          for (int cc = 0; cc < kChunks; ++cc) tmem_ld32(tDQ + cc * 32, acc[cc]);
          tmem_wait_ld();
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(smem_u32(&sh.bar_dq_empty));
          if (tl) FMHA_TL(1, g, 2);
          unsigned* order_word = nullptr;
          uint32_t order_shift = 0, order_mask = 0xffffffffu;
          unsigned turn = 0;
          if constexpr (kDet) {
            const size_t at = (size_t)it.zh * (p.seqlen_q_pad / T::kBlock) + tile;
            order_word = p.dq_order + (at == 1 ? 0 : at);
            order_shift = at == 1 ? 16 : 0;
            order_mask = at < 2 ? 0xffffu : 0xffffffffu;
            turn = bwd_turn(p, it, tile);
          }
#pragma unroll
          for (int cc = 0; cc < kChunks; ++cc) {
            // One reduce-add per 32-column chunk for the whole 128-row tile (16 KB): few large
            // bulk operations instead of many small ones.  The buffer was last used two
            // reduce-adds ago: at most one group may still be reading.
            uint32_t stg_buf;
            if constexpr (kChunks % 2 == 0) {
              stg_buf = stg_smem + (cc & 1) * 16384;
            } else {
              stg_buf = stg_smem + (chunk_no & 1u) * 16384;
              ++chunk_no;
            }
            if (r == 0) tma_wait_group_read<1>();
            named_bar_sync(2, 128);
            const uint32_t buf_row = stg_buf + r * 128;
#pragma unroll
            for (int k4 = 0; k4 < 8; ++k4)
              sts128(buf_row + ((k4 ^ (r & 7)) << 4), acc[cc][k4 * 4 + 0], acc[cc][k4 * 4 + 1],
                     acc[cc][k4 * 4 + 2], acc[cc][k4 * 4 + 3]);
            fence_proxy_async_smem();
            named_bar_sync(2, 128);
            if (r == 0) {
              if (kDet && cc == 0) {
                // those whose turn comes before have added their share of this query tile
                global_flag_wait(order_word, order_shift, order_mask, turn, &sh.abort_word, p.status, 22);
                fence_proxy_async_all();
              }
              tma_reduce_add_4d(&tm_dqacc, stg_buf, cc * 32, tile * T::kBlock, it.h, it.z);
              tma_commit_group();
              if (kDet && cc == kChunks - 1) {
                tma_wait_group<0>();  // the adds have been performed, not just read from shared memory
                fence_proxy_async_all();
                __threadfence();
                // (a half's carry is not the other half's)
                const bool wraps = order_mask == 0xffffu && order_shift == 0 && (turn & 0xffffu) == 0xffffu;
                global_flag_release(order_word, wraps ? 1u - 65536u : 1u << order_shift);
              }
            }
          }
          if (tl) FMHA_TL(1, g, 3);
        }
        // dV and dK of the item: tensor memory -> 16 bit -> TMA stores through the staging buffers; or (ring attention)
        // 32 columns of fp32 at a time, reduce-added to what is there or, with accum_overwrite, in its place.  (With
        // loads and stores of a row per thread, eight warps behind the next P^T / these four / so, whole backward, us,
        // bf16, adding: Z8 H16 N512 D128 120 / 130 / 81, D64 69 / 74 / 47, Z1 H32 N4096 D128 causal 479 / 500 / 383;
        // in its place: 98 / 92 / 78, 57 / 52 / 46, 439 / 424 / 390.  Through the staging buffers, but by loads and
        // stores of whole lines, which keep one fused multiply-add: 127, 67, 484.)  (This group does it
        // because it has time to until the next item's first dQ.  Written by the compute groups they hold up the next
        // item's P^T and dS^T: the SM's port towards L2, at 20 bytes/clk, has the last dQ to send, too.)
        mbar_wait(smem_u32(&sh.bar_acc_full), drained & 1, abort_word, 15);
        ++drained;
        tc_fence_after();
#pragma unroll 1
        for (int i = 0; i < 2; ++i) {
          const bool is_dk = i == 1;
          const uint32_t tAcc = tmem_base + lane_addr + (is_dk ? T::kColDK : T::kColDV);
          const float mul = is_dk ? p.scale : 1.f;
          float* accum = is_dk ? p.dk_accum : p.dv_accum;
          uint32_t acc[kChunks][32];
#pragma unroll
          for (int cc = 0; cc < kChunks; ++cc) tmem_ld32(tAcc + cc * 32, acc[cc]);
          tmem_wait_ld();
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(smem_u32(is_dk ? &sh.bar_dk_read : &sh.bar_dv_read));
          if (accum != nullptr) {
            // a padding key has no result: nothing is added to its row, and what replaces it is zero
            const bool have = it.kb * T::kBlock + r < it.sk;
            const float none = p.accum_overwrite != 0 ? 0.f : -0.f;
#pragma unroll
            for (int cc = 0; cc < kChunks; ++cc) {
              uint32_t stg_buf;
              if constexpr (kChunks % 2 == 0) {
                stg_buf = stg_smem + (cc & 1) * 16384;
              } else {
                stg_buf = stg_smem + (chunk_no & 1u) * 16384;
                ++chunk_no;
              }
              if (r == 0) tma_wait_group_read<1>();
              named_bar_sync(2, 128);
#pragma unroll
              for (int k4 = 0; k4 < 8; ++k4) {
                uint32_t w[4];
#pragma unroll
                for (int k = 0; k < 4; ++k)
                  w[k] = __float_as_uint(have ? __uint_as_float(acc[cc][k4 * 4 + k]) * mul : none);
                sts128(stg_buf + r * 128 + ((k4 ^ (r & 7)) << 4), w[0], w[1], w[2], w[3]);
              }
              fence_proxy_async_smem();
              named_bar_sync(2, 128);
              if (r == 0) {
                const CUtensorMap* tm = is_dk ? &tm_dk : &tm_dv;
                if (p.accum_overwrite != 0) tma_store_4d(tm, stg_buf, cc * 32, it.kb * T::kBlock, it.h, it.z);
                else tma_reduce_add_4d(tm, stg_buf, cc * 32, it.kb * T::kBlock, it.h, it.z);
                tma_commit_group();
              }
            }
            continue;
          }
#pragma unroll
          for (int b = 0; b < T::kBoxes; ++b) {  // 64 columns (128 bytes) of each row
            uint32_t stg_buf;
            if constexpr (kChunks % 2 == 0) {
              stg_buf = stg_smem + ((T::kBoxes == 1 ? i : b) & 1) * 16384;
            } else {
              stg_buf = stg_smem + (chunk_no & 1u) * 16384;
              ++chunk_no;
            }
            // At D = 64 an item leaves one box each of dV and dK.  If one of them is in fp32 (two boxes), the other
            // breaks the alternation of the buffers: then nothing may be reading before it, nor behind it.
            const bool alone = T::kBoxes == 1 && (p.dk_accum == nullptr) != (p.dv_accum == nullptr);
            if (r == 0) {
              if (alone) tma_wait_group_read<0>();
              else tma_wait_group_read<1>();
            }
            named_bar_sync(2, 128);
#pragma unroll
            for (int ch = 0; ch < (DR - b * 64 < 64 ? 4 : 8); ++ch) {
              const uint32_t* a = &acc[b * 2 + ch / 4][ch % 4 * 8];
              uint32_t w[4];
#pragma unroll
              for (int k = 0; k < 4; ++k)
                w[k] = pack16x2<kBf16>(__uint_as_float(a[2 * k]) * mul, __uint_as_float(a[2 * k + 1]) * mul);
              sts128(stg_buf + r * 128 + ((ch ^ (r & 7)) << 4), w[0], w[1], w[2], w[3]);
            }
            fence_proxy_async_smem();
            named_bar_sync(2, 128);
            if (r == 0) {
              tma_store_4d(is_dk ? &tm_dk : &tm_dv, stg_buf, b * 64, it.kb * T::kBlock, it.h, it.z);
              tma_commit_group();
              if (alone) tma_wait_group_read<0>();
            }
          }
        }
      }
      if (r == 0) tma_wait_group<0>();
    }
  }

  // ---- teardown
  tc_fence_before();
  __syncthreads();
  if (sh.abort_word != 0) {
    if (threadIdx.x == 0 && p.status != nullptr) atomicCAS(p.status, 0, sh.abort_word);
    // let copies that may still be in flight land before the shared memory is released
    for (int i = 0; i < 64; ++i) __nanosleep(1000);
  }
  if (warp == T::kMmaWarp) {
    tc_fence_after();
    tmem_dealloc(tmem_base, T::kTmemCols);
  }
}

}  // namespace fmha
