// Forward attention kernel for sm_100a: O = softmax(scale * Q K^T [+ mask]) V, LSE.
//
// Replaces fused_mha_forward_kernel of the reference (kernel/fused_mha_kernel.cu:20-323):
// same mathematics (online softmax over KV tiles, running max / sum, O rescale), none of its
// structure.  A work item is 256 query rows (two 128-row tiles) of one (batch, head), processed
// against the KV sequence (or a chunk of it) in 128-row tiles, one per ROUND:
//
//   warp 8      TMA producer for K and V through a ring of shared-memory slots of one tile (full /
//               empty mbarriers per slot); it is also the one that takes the next item
//   warp 10     TMA producer for the two Q tiles of an item, as soon as the previous item's
//               last S = Q K^T has released them
//   warp 9      MMA issuer.  A round is two turns, one per query tile t: O_t += P_t(j) V(j) (P_t
//               read from tensor memory, in two halves of 64 keys), S_t(j+1) = Q_t K(j+1)^T
//               (128 x 128).  The whole warp runs the loop so that descriptors stay in uniform
//               registers; one elected lane issues.
//   warps 0-3   softmax of query tile 0: one thread per row, a whole 128-column row of S_0(j) in
//               registers, online exp2 softmax, P_0(j) written back over S_0(j) as fp16 in two
//               halves (each released to the MMA warp as soon as it is there), lazy O_0 rescale,
//               epilogue
//   warps 4-7   the same for query tile 1
//
// What bounds it at D = 128: shared memory, then power.  Per round the tensor pipe needs 2048 clk, and
// its operands with the TMA writes are 256 KB, which at 128 bytes/clk is 2048 clk as well; a round takes
// 2850 clk with the exponentials left out and 3250 with them (1500-1700 clk per group).  At D = 64
// it is the softmax groups.  What made it faster than S tiles of 64 keys, double buffered, with two
// issuing warps (us, that form -> this one, sustained, in turn in one process; D = 128, Z=8, H=32, N=2048 without
// a mask, bf16 636 -> 531, causal, bf16 345 -> 312, Z=1, H=16, N=16384 without a mask, fp16 2608 -> 1918, causal, bf16
// 1175 -> 1055; D = 64, Z=2, H=16, N=8192 without a mask, fp16 1005 -> 759):
//   - S tiles of 128 keys read Q from shared memory half as often;
//   - the turns come in a fixed order, which keeps the two softmax groups half a round apart: while
//     one group's exponentials run, the tensor pipe works for the other;
//   - the code is small: the roles of a CTA share one instruction cache, and at 200 KB of code the MMA
//     warp waited for instructions (2850 clk of a round became 4000).  Control flow of the issuing
//     warps is made warp-uniform for the compiler, slow paths are rolled loops;
//   - no row maximum in the ordinary round (see the softmax groups; what has to be watched instead, so
//     that no score is too large for it, costs 1 %), and the epilogue of an item waits for nothing;
//   - 1/8 of the exponentials are a polynomial on the FMA pipe (see kFwdPolyPairs).
//
// While the groups run an item's epilogue the producers and the MMA warp already work on the next
// item, so that the load latency at the head of an item and the store at its tail are hidden.
//
// Element type: fp16 (the reference's only type, kernel/fused_mha_api.cpp:25-29) or bf16
// (kBf16): the tensor cores take either by two bits of the instruction descriptor; P and O are
// then rounded to bf16 instead of fp16, everything in between stays fp32.
//
// Tensor memory (512 columns): S_t [t * 128, + 128); O_0 [256, 256 + D), O_1 [256 + D, 256 + 2 D);
// P_t aliases the first 64 columns of S_t (two fp16 per 32-bit column).
//
// Shared memory: rows of 64 fp16 (128 bytes) in the TMA / UMMA 128-byte swizzle.  A 128 x D
// tile is D/64 boxes of 128 x 64, box b at byte offset b * 16384.  Per softmax group one box
// stages the output for the TMA store, 64 columns at a time.
//
// Work distribution: the grid has one block per item, heaviest first; a running CTA takes over
// further blocks through cluster launch control, i.e. the hardware balances the load.  A caller
// that wants SMs left free (sm_margin) gets a smaller grid with the items dealt round robin.
#pragma once
#include <cuda.h>
#include <math_constants.h>

#include <type_traits>

#include "aux_kernels.cuh"
#include "ptx.cuh"

namespace fmha {

struct FwdKernelParams {
  float* lse;
  int heads, seqlen_q, seqlen_k;
  int num_q_blocks;     // ceil(seqlen_q / 256)
  int num_heads_total;  // batch * heads
  int head_group;       // heads whose items are interleaved (>= 1)
  int items_per_head;   // query blocks, or chunks of them
  int num_items;
  int deal;             // 1: items are dealt round robin to the blocks; 0: cluster launch control
  int chunk_tiles;      // KV tiles of 128 an item covers at most
  float scale_log2;     // |scale| * log2(e)
  int negate;           // scale < 0: the tensor cores form -Q K^T, so that a row's maximum is a maximum
  int causal, causal_shift;
  int* status;
  // optional per-batch lengths (right-padded batches): rows >= seqused_q[z] and keys >=
  // seqused_k[z] are padding, skipped tile-wise and masked inside partial tiles
  const int* seqused_q;
  const int* seqused_k;
  // query blocks cut in several chunks: fp32 partial outputs (chunk, Z*H, seqlen_q, row_elems),
  // each normalised by its own row sum, and their log-sum-exp (chunk, Z*H, seqlen_q)
  float* o_part;
  float* lse_part;
  int row_elems;        // elements per row of the tensors (head_dim)
};

// Pairs out of every 8 whose exponential is a polynomial on the FMA pipe (the rest use MUFU).  None / 1 / 2
// (3 at D = 64), us: D = 128, Z=8, H=32, N=2048 without a mask 551 / 537 / -, Z=1, H=16, N=16384 causal
// 1136 / 1108 / -; D = 64, Z=2, H=16, N=8192 without a mask 799 / 783 / 784 (806), Z=64, H=16, N=512
// 126.7 / 124.2 / 127.7 (131.8); no difference between none and 1 at D = 128, N = 2048 causal.
constexpr int kFwdPolyPairs = 1;

// DR <= D: elements per row of the tensors.  96 runs on the tiles of 128: the second box of a tile load holds 32
// columns and zeros, which the MMAs leave out.
template <int D, bool kBf16 = false, int DR = D, bool kPair = false>
struct FwdTraits {
  static constexpr int kBlockM = 128;  // rows per query tile
  static constexpr int kTilesM = 2;    // query tiles per work item
  static constexpr int kBlockN = 128;  // rows per KV tile
  static constexpr int kBoxes = D / 64;
  static constexpr int kBoxBytes = 128 * 128;  // 128 rows x 128 bytes
  static constexpr int kTileBytes = kBoxes * kBoxBytes;
  // A paired item (see the kernel) has one query tile in shared memory and no output to stage: room for six K
  // or V tiles at D = 128, three per chunk.  64 queries x 8192 keys, 64 heads, bf16, two per chunk / three: 65.1 / 61.1
  // us (K and V alone take 41 at the rate of a copy).
  static constexpr int kQTiles = kPair ? 1 : kTilesM;
  // ring slots of one K or V tile
  static constexpr int kStages = (D == 128 ? 4 : 8) + (kPair ? (D == 128 ? 2 : 4) : 0);
  static constexpr int kItemStages = 4;  // item ids published ahead
  static constexpr int kThreads = 384;   // softmax 0, softmax 1, {K/V, MMA, Q, idle} warps
  // Q tiles, K/V ring, one 64-column output box per softmax group
  static constexpr int kSmemBytes =
      1024 + (kQTiles + kStages) * kTileBytes + (kPair ? 0 : kTilesM * kBoxBytes);
  static constexpr int kTmemCols = 512;
  static constexpr uint32_t kIdescQK = umma_idesc_f16(128, kBlockN, 0, 0, kBf16);
  static constexpr uint32_t kIdescPV = umma_idesc_f16(128, DR, 0, 1, kBf16);
};

constexpr int kFwdRegsIssue = 88;                                 // warps 8-11
constexpr int kFwdRegsSoftmax = 168 + (168 - kFwdRegsIssue) / 2;  // warps 0-7: 208
static_assert(kFwdRegsIssue <= 168 && kFwdRegsSoftmax >= 168 && kFwdRegsSoftmax % 8 == 0,
              "setmaxnreg.dec must not raise and .inc must not lower the 168 registers of the launch");

// lazy rescale: the exponentials of 64 keys of a row may add up to 2^10 before O is rescaled to a
// new reference (P has to stay far from the 65504 of fp16; O and the row sum are fp32)
constexpr float kRescaleSum = 1024.0f;

// A work item: 256 query rows from q0 of head zh = z * heads + h, KV tiles [kv_first, kv_first + n_t)
// for its query tile t (n_t = 0: the tile sees nothing of this chunk).  A paired item (see the kernel) has
// the same 128 rows twice, and its tile 1 the next chunk of the keys.  The producer warp works it out and
// publishes it in shared memory.
struct __align__(16) FwdItem {
  int id;      // -1: no more items
  int n0, n1;  // KV tiles of the two query tiles
  int q0;
  int z, h, zh;
  int kv_first;
  int sq, sk;  // lengths of the batch entry
  int chunk;   // index of the (first) chunk among those of its query block, -1: the block is not cut
  int pad;
};

// the lengths that count for batch entry z: the tensors' own, or the caller's per-batch ones
__device__ __forceinline__ void fwd_lengths(const FwdKernelParams& p, int z, int& sq, int& sk) {
  sq = p.seqused_q == nullptr ? p.seqlen_q : max(0, min(p.seqlen_q, __ldg(p.seqused_q + z)));
  sk = p.seqused_k == nullptr ? p.seqlen_k : max(0, min(p.seqlen_k, __ldg(p.seqused_k + z)));
}

// KV tiles the query rows up to r_last see, of nk_total
__host__ __device__ __forceinline__ int fwd_visible_tiles(bool causal, int shift, int r_last, int nk_total) {
  if (!causal) return nk_total;
  const long long lim = (long long)r_last + shift;
  if (lim < 0) return 0;
  return lim / 128 + 1 < nk_total ? (int)(lim / 128 + 1) : nk_total;
}
// chunks of a query block, by the tensors' own lengths (also on the host, where the per-batch
// lengths are not known)
__host__ __device__ __forceinline__ int fwd_chunks(bool causal, int shift, int qb, int seqlen_q, int nk_total,
                                                   int chunk_tiles) {
  const int r_last = (qb * 256 + 255 < seqlen_q - 1) ? qb * 256 + 255 : seqlen_q - 1;
  const int n = fwd_visible_tiles(causal, shift, r_last, nk_total);
  return n <= chunk_tiles ? 1 : (n + chunk_tiles - 1) / chunk_tiles;
}

// Items in groups of head_group heads (their K and V share the L2); in a group the last query
// blocks first (under a causal mask the heaviest), heads innermost.
template <bool kPair>
__device__ __forceinline__ FwdItem fwd_item(const FwdKernelParams& p, int id) {
  FwdItem it;
  it.id = id;
  it.pad = 0;
  const int per_group = p.head_group * p.items_per_head;
  const int group = id / per_group, within = id % per_group;
  const int heads_here = min(p.head_group, p.num_heads_total - group * p.head_group);
  int u = within / heads_here;
  it.zh = group * p.head_group + within % heads_here;
  it.z = it.zh / p.heads;
  it.h = it.zh % p.heads;
  int qb = p.num_q_blocks - 1;
  it.chunk = -1;
  it.kv_first = 0;
  int most = 0x7fffffff;
  if (kPair) {
    it.chunk = 2 * u;
    it.kv_first = it.chunk * p.chunk_tiles;
    most = p.chunk_tiles;
  } else if (p.o_part == nullptr) {
    qb -= u;
  } else {
    for (;; --qb) {
      const int chunks =
          fwd_chunks(p.causal != 0, p.causal_shift, qb, p.seqlen_q, (p.seqlen_k + 127) / 128, p.chunk_tiles);
      if (u < chunks || qb == 0) {
        if (chunks > 1) {
          it.chunk = u;
          it.kv_first = u * p.chunk_tiles;
          most = p.chunk_tiles;
        }
        break;
      }
      u -= chunks;
    }
  }
  it.q0 = qb * 256;
  fwd_lengths(p, it.z, it.sq, it.sk);
  const int nk_total = (it.sk + 127) / 128;
  auto tiles = [&](int r0, int first) {
    if (r0 >= it.sq) return 0;
    const int n = fwd_visible_tiles(p.causal != 0, p.causal_shift, min(r0 + 127, it.sq - 1), nk_total);
    return max(0, min(most, n - first));
  };
  it.n0 = tiles(it.q0, it.kv_first);
  it.n1 = kPair ? tiles(it.q0, it.kv_first + most) : tiles(it.q0 + 128, it.kv_first);
  return it;
}

// kPair: no more than 128 query rows.  Both query tiles are these rows, each against a chunk of the keys of its
// own, and both chunks leave partial results.  K and V of tile t come through a ring of their own, half of the
// slots.  (With one query tile, cut or not, a CTA takes 1.9 us per KV tile: MMA, softmax and MMA one after the
// other, and half of the SM idle.  64 queries x 8192 keys, 64 heads, bf16, us: D = 128 74 -> 64, D = 64 64 -> 46.)
template <int D, bool kBf16 = false, bool kPair = false, int DR = D>
__global__ void __launch_bounds__(384, 1)
    fmha_fwd_kernel(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_k,
                    const __grid_constant__ CUtensorMap tm_v, const __grid_constant__ CUtensorMap tm_o,
                    const FwdKernelParams p) {
  using T = FwdTraits<D, kBf16, DR, kPair>;
  extern __shared__ uint8_t smem_raw[];
  __shared__ __align__(16) uint8_t clc_word[16];
  __shared__ uint64_t bar_clc;                        // the answer to the last request is in clc_word
  __shared__ FwdItem items[T::kItemStages];           // items of this CTA
  __shared__ uint64_t bar_item_full[T::kItemStages], bar_item_empty[T::kItemStages];
  __shared__ uint64_t bar_q_full[2];   // Q_t of the current item has landed
  __shared__ uint64_t bar_q_free[2];   // the last S_t = Q_t K^T of the item is done: Q_t reusable
  __shared__ uint64_t bar_kv_full[T::kStages];
  __shared__ uint64_t bar_kv_empty[T::kStages];
  __shared__ uint64_t bar_s_full[2];     // S_t(j) is there, and so is the result of O_t += of round j - 1
  __shared__ uint64_t bar_p_full[2][2];  // [tile][half]: P_t for 64 keys is there
  __shared__ uint64_t bar_pv_half[2];    // O_t += of the first 64 keys of the round has completed
  __shared__ uint64_t bar_o_full[2];
  __shared__ uint64_t bar_o_read[2];   // the softmax group has O_t in registers: O_t reusable
  __shared__ uint32_t tmem_base_slot;
  __shared__ int abort_word;
  __shared__ int skip_cta;

  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0);  // warp-uniform for the compiler, too
  const int lane = threadIdx.x & 31;

  // a status word already set by an earlier launch / CTA means: drain the grid quickly
  if (threadIdx.x == 0) {
    skip_cta = (p.status != nullptr && *reinterpret_cast<volatile int*>(p.status) != 0) ? 1 : 0;
    abort_word = 0;
  }
  __syncthreads();
  if (skip_cta) return;

  const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  const uint32_t q_smem = smem_base;                                    // 2 query tiles (kPair: one)
  const uint32_t ring_smem = smem_base + T::kQTiles * T::kTileBytes;    // K/V ring
  const uint32_t ostage_smem = ring_smem + T::kStages * T::kTileBytes;  // 2 output boxes (kPair: none)
  constexpr uint32_t kRingSlots = T::kStages / 2;  // kPair: of each tile's ring

  // ---- set-up: barriers (thread 0), tensor memory (warp 9)
  if (threadIdx.x == 0) {
    mbar_init(smem_u32(&bar_clc), 1);
    for (int s = 0; s < T::kItemStages; ++s) {
      mbar_init(smem_u32(&bar_item_full[s]), 1);
      mbar_init(smem_u32(&bar_item_empty[s]), 10);  // MMA warp, Q warp, eight softmax warps
    }
    for (int s = 0; s < T::kStages; ++s) {
      mbar_init(smem_u32(&bar_kv_full[s]), 1);
      mbar_init(smem_u32(&bar_kv_empty[s]), 1);
    }
    for (int t = 0; t < 2; ++t) {
      mbar_init(smem_u32(&bar_q_full[t]), 1);
      mbar_init(smem_u32(&bar_q_free[t]), 1);
      mbar_init(smem_u32(&bar_s_full[t]), 1);
      // one arrival per softmax warp: 128 arrivals on one word are 128 serialised atomics.  A warp
      // cannot arrive twice in one phase: it needs the next S_t in between, which is only issued
      // once all four warps' P_t has been consumed.
      mbar_init(smem_u32(&bar_p_full[t][0]), 4);
      mbar_init(smem_u32(&bar_p_full[t][1]), 4);
      mbar_init(smem_u32(&bar_pv_half[t]), 1);
      mbar_init(smem_u32(&bar_o_full[t]), 1);
      mbar_init(smem_u32(&bar_o_read[t]), 4);
    }
    fence_barrier_init();
  }
  if (warp == 9) {
    tmem_alloc(smem_u32(&tmem_base_slot), T::kTmemCols);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = __shfl_sync(0xffffffffu, tmem_base_slot, 0);

  // The next item published by the producer warp (every consuming warp keeps its own count); id = -1
  // when there is none, and when a wait ran out.
  uint32_t item_cnt = 0;
  auto take_item = [&]() -> FwdItem {
    const uint32_t s = item_cnt % T::kItemStages;
    FwdItem it;
    if (mbar_wait_warp(smem_u32(&bar_item_full[s]), (item_cnt / T::kItemStages) & 1, &abort_word, 12)) {
      it = items[s];
      // what decides over branches is made warp-uniform for the compiler: only in control flow that
      // it knows to be uniform can it keep addresses and MMA descriptors in uniform registers
      it.id = __shfl_sync(0xffffffffu, it.id, 0);
      it.n0 = __shfl_sync(0xffffffffu, it.n0, 0);
      it.n1 = __shfl_sync(0xffffffffu, it.n1, 0);
    } else {
      it.id = -1;
      it.n0 = it.n1 = 0;
    }
    __syncwarp();
    if (lane == 0) mbar_arrive(smem_u32(&bar_item_empty[s]));
    ++item_cnt;
    return it;
  };

  // Register budget: 384 threads leave 168 per thread.  The producer / MMA warpgroup hands part
  // of its share to the softmax warpgroups, whose threads hold a 128-column row of S.  Each
  // setmaxnreg sits at the top of its warpgroup's own branch.
  if (warp >= 8) {
    reg_dealloc<kFwdRegsIssue>();
    if (warp == 8) {
      // =========================== K/V producer, item source (converged warp) ==========
      if (elect_one()) {
        tma_prefetch_desc(&tm_q);
        tma_prefetch_desc(&tm_k);
        tma_prefetch_desc(&tm_v);
      }
      __syncwarp();
      bool ok = true;
      uint32_t published = 0, asked = 0;
      // Asking for a block is separate from taking it: the answer takes a microsecond, and asking as
      // late as possible is what lets the CTA that is done first have the block.
      bool pending = false;
      auto ask = [&]() {
        if (p.deal || pending) return;
        if (elect_one()) {
          fence_proxy_async_smem();  // the last answer has been read
          mbar_arrive_expect_tx(smem_u32(&bar_clc), 16);
          clc_request(smem_u32(clc_word), smem_u32(&bar_clc));
        }
        __syncwarp();
        pending = true;
      };
      // finds the next item and publishes it
      int id = -1;
      auto next_item = [&]() -> FwdItem {
        if (published == 0) {
          id = blockIdx.x;
        } else if (p.deal) {
          id = p.num_items - id > (int)gridDim.x ? id + (int)gridDim.x : -1;
        } else {
          ask();
          ok = mbar_wait_warp(smem_u32(&bar_clc), asked & 1, &abort_word, 14);
          ++asked;
          pending = false;
          id = ok ? clc_answer(smem_u32(clc_word)) : -1;
        }
        id = __shfl_sync(0xffffffffu, id, 0);
        FwdItem it;
        it.id = -1;
        it.n0 = it.n1 = 0;
        if (id >= 0) it = fwd_item<kPair>(p, id);
        it.n0 = __shfl_sync(0xffffffffu, it.n0, 0);
        it.n1 = __shfl_sync(0xffffffffu, it.n1, 0);
        const uint32_t s = published % T::kItemStages, round = published / T::kItemStages;
        if (round > 0 && !mbar_wait_warp(smem_u32(&bar_item_empty[s]), (round - 1) & 1, &abort_word, 13)) ok = false;
        if (ok && lane == 0) {
          items[s] = it;
          mbar_arrive(smem_u32(&bar_item_full[s]));
        }
        __syncwarp();
        ++published;
        if (!ok) it.id = -1;
        return it;
      };
      uint32_t slot = 0, phase = 1;  // the next ring slot, parity of its last release (none yet: passes)
      uint32_t loaded[2] = {0, 0};   // kPair: tiles that went through each ring
      auto load = [&](const CUtensorMap* tm, const FwdItem& it, int tile, int ring) {
        if constexpr (kPair) {
          const uint32_t n = ring ? loaded[1]++ : loaded[0]++;
          slot = ring * kRingSlots + n % kRingSlots;
          phase = n / kRingSlots % 2 ^ 1;
        }
        if (!(ok = mbar_wait_warp(smem_u32(&bar_kv_empty[slot]), phase, &abort_word, 2))) return;
        if (elect_one()) {
          const uint32_t fbar = smem_u32(&bar_kv_full[slot]);
          mbar_arrive_expect_tx(fbar, T::kTileBytes);
#pragma unroll
          for (int b = 0; b < T::kBoxes; ++b)
            tma_load_4d(ring_smem + slot * T::kTileBytes + b * T::kBoxBytes, tm, fbar, b * 64,
                        (it.kv_first + tile) * T::kBlockN, it.h, it.z);
        }
        __syncwarp();
        if (!kPair && ++slot == T::kStages) {
          slot = 0;
          phase ^= 1u;
        }
      };
      // K(0) V(0) K(1) V(1) ... of one item after the other (kPair: of its tiles in turn; tile 0 has no fewer)
      while (ok) {
        const FwdItem it = next_item();
        if (it.id < 0) break;
        const int n = max(it.n0, it.n1);
#pragma unroll 1
        for (int i = 0; ok && i < 2 * n; ++i) {
          if (i >= 2 * n - 5) ask();
          load((i & 1) ? &tm_v : &tm_k, it, i >> 1, 0);
          if (kPair && ok && (i >> 1) < it.n1) load((i & 1) ? &tm_v : &tm_k, it, p.chunk_tiles + (i >> 1), 1);
        }
      }
    } else if (warp == 10) {
      // =========================== Q producer ===========================
      // its own warp, so that waiting for the Q buffers of the running item never holds back
      // the K/V prefetch of the next one
      uint32_t phase = 0;  // bit t: Q_t tiles loaded so far, modulo 2 (phase of the Q barriers)
      uint32_t used = 0;   // bit t: Q_t has been loaded before
      bool ok = true;
      while (ok) {
        const FwdItem it = take_item();
        if (it.id < 0) break;
        if constexpr (kPair) {
          // one tile for both: free once the last S of either of the item before is done
          if (it.n0 == 0) continue;
          for (int t = 0; ok && t < 2; ++t)
            if ((used >> t) & 1) ok = mbar_wait_warp(smem_u32(&bar_q_free[t]), ((phase >> t) & 1) ^ 1, &abort_word, 1);
          if (!ok) break;
          if (elect_one()) {
            const uint32_t qbar = smem_u32(&bar_q_full[0]);
            mbar_arrive_expect_tx(qbar, T::kTileBytes);
#pragma unroll
            for (int b = 0; b < T::kBoxes; ++b)
              tma_load_4d(q_smem + b * T::kBoxBytes, &tm_q, qbar, b * 64, it.q0, it.h, it.z);
          }
          __syncwarp();
          const uint32_t both = it.n1 > 0 ? 3u : 1u;
          phase ^= both;
          used |= both;
        } else {
#pragma unroll 1
          for (int t = 0; t < T::kTilesM; ++t) {
            if ((t == 0 ? it.n0 : it.n1) == 0) continue;
            const int row = it.q0 + t * T::kBlockM;
            if ((used >> t) & 1) {
              // cold from HBM this takes microseconds: start towards L2 before waiting for the buffer
              if (elect_one())
#pragma unroll
                for (int b = 0; b < T::kBoxes; ++b) tma_prefetch_l2_4d(&tm_q, b * 64, row, it.h, it.z);
              __syncwarp();
              if (!mbar_wait_warp(smem_u32(&bar_q_free[t]), ((phase >> t) & 1) ^ 1, &abort_word, 1)) {
                ok = false;
                break;
              }
            }
            if (elect_one()) {
              const uint32_t qbar = smem_u32(&bar_q_full[t]);
              mbar_arrive_expect_tx(qbar, T::kTileBytes);
#pragma unroll
              for (int b = 0; b < T::kBoxes; ++b)
                tma_load_4d(q_smem + t * T::kTileBytes + b * T::kBoxBytes, &tm_q, qbar, b * 64, row, it.h, it.z);
            }
            __syncwarp();
            phase ^= 1u << t;
            used |= 1u << t;
          }
        }
      }
    } else if (warp == 9) {
      // =========================== MMA issuer (converged warp, elected issue) ===================
      // All 32 lanes run the loop so that addresses and descriptors live in uniform registers;
      // a loop run by one lane only makes every operand a per-thread value that has to be moved
      // to a uniform register before each tcgen05.mma, and the issue rate falls below the
      // tensor pipe's 64 cycles per 128x128x16 MMA.
      const uint32_t q_lo0 = umma_desc_lo(q_smem, kLboKMajor);
      const uint32_t idesc_qk = T::kIdescQK | (p.negate ? kIdescNegateA : 0u);
      uint32_t slot = 0, slot_phase = 0;
      uint32_t phase_q = 0;  // bit t: parity of the next q_full[t]
      uint32_t phase_p = 0;  // bit t: parity of the next p_full[t]
      uint32_t phase_o = 0;  // bit t: parity of the next o_read[t], of the first one already waited for
      uint32_t used_o = 0;   // bit t: O_t has been written before
      auto slot_wait = [&]() {
        return mbar_wait_warp(smem_u32(&bar_kv_full[slot]), slot_phase, &abort_word, 4);
      };
      auto slot_next = [&]() {
        umma_commit_elect(smem_u32(&bar_kv_empty[slot]));
        if (++slot == T::kStages) {
          slot = 0;
          slot_phase ^= 1u;
        }
      };
      uint32_t taken[2] = {0, 0};  // kPair: tiles that came through each ring
      [[maybe_unused]] auto ring_next = [&](int t) {
        const uint32_t n = t ? taken[1]++ : taken[0]++;
        slot = t * kRingSlots + n % kRingSlots;
        slot_phase = n / kRingSlots % 2;
      };
      FwdItem cur = take_item();
      int j = -1;
      bool ok = true;
      // One pass per round: V(j) of cur (j = -1: none) and K(j+1), which after the last round is K(0) of
      // the item behind it (nxt).
      while (ok && cur.id >= 0) {
        const int n = max(cur.n0, cur.n1);
        if (n == 0) {
          cur = take_item();
          continue;
        }
        const bool last = j == n - 1;
        FwdItem nxt = cur;
        if (last) nxt = take_item();
        const bool has_k = !last || max(nxt.n0, nxt.n1) > 0;
        const int jk = last ? 0 : j + 1;
        // V(j) sits in the current slot, K(jk) in the one behind it
        const uint32_t v_addr = ring_smem + slot * T::kTileBytes;
        const uint32_t k_slot = j < 0 ? slot : (slot + 1 == T::kStages ? 0 : slot + 1);
        const uint32_t k_addr = ring_smem + k_slot * T::kTileBytes;
        const uint32_t k_phase = k_slot < slot ? slot_phase ^ 1u : slot_phase;
        if (!kPair && j >= 0 && !(ok = slot_wait())) break;
#pragma unroll 1
        for (int t = 0; t < 2; ++t) {
          const int nt = t == 0 ? cur.n0 : cur.n1;
          if (j >= 0 && j < nt) {
            // ---- O_t (+)= P_t V(j), as the two halves of P_t come in
            // the first O_t += of an item overwrites O_t: the previous item's epilogue must have
            // read it out of tensor memory
            if (j == 0) {
              if ((used_o >> t) & 1) {
                ok = mbar_wait_warp(smem_u32(&bar_o_read[t]), (phase_o >> t) & 1, &abort_word, 7);
                phase_o ^= 1u << t;
              }
              used_o |= 1u << t;
            }
            if (kPair) {
              ring_next(t);
              if (!(ok = slot_wait())) break;
            }
            const uint32_t v_lo = umma_desc_lo(kPair ? ring_smem + slot * T::kTileBytes : v_addr, kLboMnMajor);
            const uint32_t d = tmem_base + 256 + t * D, a = tmem_base + t * 128;
#pragma unroll
            for (int half = 0; half < 2; ++half) {
              ok = ok && mbar_wait_warp(smem_u32(&bar_p_full[t][half]), (phase_p >> t) & 1, &abort_word, 6);
              tc_fence_after();
#pragma unroll
              for (int ks = half * 4; ks < half * 4 + 4; ++ks)
                umma_ts_elect(d, a + ks * 8, v_lo + ((ks * 2048) >> 4), T::kIdescPV, (j > 0 || ks > 0) ? 1u : 0u);
              // told to the softmax group, for the rare case that it has to rescale in mid-round
              if (half == 0) umma_commit_elect(smem_u32(&bar_pv_half[t]));
            }
            phase_p ^= 1u << t;
            if (j == nt - 1) umma_commit_elect(smem_u32(&bar_o_full[t]));
            if (kPair) umma_commit_elect(smem_u32(&bar_kv_empty[slot]));
            if (!ok) break;
          }
          if (!kPair && t == 1 && j >= 0) slot_next();
          // ---- S_t = Q_t K^T of the round after, which may be the first of the next item
          if (!kPair && t == 0 && has_k &&
              !(ok = mbar_wait_warp(smem_u32(&bar_kv_full[k_slot]), k_phase, &abort_word, 5)))
            break;
          const int nk = t == 0 ? nxt.n0 : nxt.n1;
          if (jk < nk) {
            if (kPair) {
              ring_next(t);
              if (!(ok = slot_wait())) break;
            }
            if (jk == 0 && (!kPair || t == 0)) {
              ok = mbar_wait_warp(smem_u32(&bar_q_full[t]), (phase_q >> t) & 1, &abort_word, 3);
              phase_q ^= 1u << t;
              if (!ok) break;
            }
            tc_fence_after();
            const uint32_t a_lo = q_lo0 + (kPair ? 0 : (t * T::kTileBytes) >> 4);
            const uint32_t b_lo = umma_desc_lo(kPair ? ring_smem + slot * T::kTileBytes : k_addr, kLboKMajor);
#pragma unroll
            for (int ks = 0; ks < DR / 16; ++ks) {
              const uint32_t off = ((ks >> 2) * T::kBoxBytes + (ks & 3) * 32) >> 4;
              umma_ss_elect(tmem_base + t * 128, a_lo + off, b_lo + off, idesc_qk, ks > 0 ? 1u : 0u);
            }
            umma_commit_elect(smem_u32(&bar_s_full[t]));
            if (kPair) umma_commit_elect(smem_u32(&bar_kv_empty[slot]));
            if (jk == nk - 1) umma_commit_elect(smem_u32(&bar_q_free[t]));
          }
        }
        if (!ok) break;
        if (!kPair && has_k) slot_next();
        ++j;
        if (last) {
          cur = nxt;
          j = has_k ? 0 : -1;
        }
      }
    }
  } else {
    // =========================== softmax / epilogue ===========================
    reg_alloc<kFwdRegsSoftmax>();
    const int t = warp >> 2;    // query tile of this warpgroup
    const int quad = warp & 3;  // TMEM lane quadrant of this warp
    const int row_in_tile = quad * 32 + lane;
    const uint32_t lane_addr = uint32_t(quad * 32) << 16;
    const uint32_t tS = tmem_base + lane_addr + t * 128;
    const uint32_t tO = tmem_base + lane_addr + 256 + t * D;
    const uint32_t o_stage = ostage_smem + t * T::kBoxBytes;
    const float c = p.scale_log2;
    uint32_t phase_s = 0, phase_o = 0;  // parities of the next s_full[t], o_full[t]
    bool stored = false;  // a TMA store of this group may still be reading the staging box

    // The epilogue of an item is done after the first round of the next one: its O_t is complete by
    // then (nothing to wait for), and what follows the read of O_t (normalising, staging, storing)
    // runs while the tensor pipe works on the second round.
    bool pending = false;
    FwdItem done;           // the item whose epilogue is pending
    float done_m = 0.f, done_l = 0.f;

    for (;;) {
      const FwdItem it = take_item();
      const int n = t == 0 ? it.n0 : it.n1;
      float m_ref = -CUDART_INF_F;  // reference score of the running softmax (raw, unscaled)
      float neg_mc = 0.f;           // -m_ref * c, 0 while there is no reference
      float l = 0.f;                // running sum of exp2((s - m_ref) * c)
      int lim;                      // last visible column of this row in the round
      {
        const int row = it.q0 + (kPair ? 0 : t * T::kBlockM) + row_in_tile;
        long long last_key = p.causal ? (long long)row + p.causal_shift : (long long)it.sk - 1;
        last_key = min(last_key, (long long)it.sk - 1);
        if (row >= it.sq) last_key = -1;  // a padding row sees nothing: O = 0, LSE = -inf
        lim = (int)max(last_key, -1ll) - (it.kv_first + (kPair ? t * p.chunk_tiles : 0)) * T::kBlockN;
      }

      for (int j = 0; j < n || j == 0; ++j, lim -= T::kBlockN) {
        if (j < n) {
          // on a time-out keep going: every later wait returns at once, and all 128 threads of
          // the group still meet at the named barriers of the epilogue
          mbar_wait(smem_u32(&bar_s_full[t]), phase_s, &abort_word, 9);
          phase_s ^= 1u;
          tc_fence_after();
          uint32_t s[4][32];
#pragma unroll
          for (int cc = 0; cc < 4; ++cc) tmem_ld32(tS + cc * 32, s[cc]);
          tmem_wait_ld();
          if (lim < T::kBlockN - 1) {
#pragma unroll
            for (int cc = 0; cc < 4; ++cc)
#pragma unroll
              for (int i = 0; i < 32; ++i)
                if (cc * 32 + i > lim) s[cc][i] = __float_as_uint(-CUDART_INF_F);
          }
          // P of 64 keys -> tensor memory.  The reference m_ref stays what it was unless an exponential
          // comes out too large; what tells is their sum, which the row sum needs anyway (and for those
          // that are a polynomial, which wraps, their largest argument), so that in the ordinary case
          // no maximum of the scores is looked for at all.  (The first round has to look: it
          // has no reference yet.)
          auto half_round = [&](auto half_tag) {
            constexpr int half = decltype(half_tag)::value;
            const uint64_t c2 = pack2f(c, c), nm2 = pack2f(neg_mc, neg_mc);
            uint64_t la = pack2f(0.f, 0.f), lb = pack2f(0.f, 0.f);
            uint32_t pk[32];
            float top = 0.f;
#pragma unroll
            for (int ch = 0; ch < 2; ++ch) {
              const int cc = half * 2 + ch;
#pragma unroll
              for (int i = 0; i < 32; i += 2) {
                const uint64_t x2 = fma2(pack2(s[cc][i], s[cc][i + 1]), c2, nm2);
                uint64_t p2;
                // kFwdPolyPairs of every 8 pairs go through the FMA pipe instead of the MUFU unit
                if (((i >> 1) & 7) < kFwdPolyPairs) {
                  p2 = poly_exp2_pair(x2, top);
                } else {
                  uint32_t x0, x1;
                  unpack2(x2, x0, x1);
                  p2 = pack2f(fast_exp2(__uint_as_float(x0)), fast_exp2(__uint_as_float(x1)));
                }
                if (i & 2) lb = add2(lb, p2); else la = add2(la, p2);
                uint32_t p0, p1;
                unpack2(p2, p0, p1);
                pk[ch * 16 + (i >> 1)] = pack16x2<kBf16>(__uint_as_float(p0), __uint_as_float(p1));
              }
            }
            uint32_t a0, a1;
            unpack2(add2(la, lb), a0, a1);
            float sum = __uint_as_float(a0) + __uint_as_float(a1);
            // (a row that has not seen anything yet has no reference to compare with)
            const bool need = !(sum <= kRescaleSum) || !(top <= kPolyExp2Top) ||
                              (m_ref == -CUDART_INF_F && lim >= half * 64);
            if (!__any_sync(0xffffffffu, need)) {
              tmem_st32(tS + half * 32, pk);
            } else {
              // Rare: a new reference.  The scores of this half are still in tensor memory (P of the
              // half goes where columns before the ones read next were).
              // O_t += of the keys before is complete: that of the previous round because its MMAs
              // precede S_t(j), that of keys 0-63 of this round by a commit of its own.  The next
              // one is not issued before this warp has arrived on p_full.
              float m_new = m_ref;
#pragma unroll 1
              for (int ch = 0; ch < 2; ++ch) {
                uint32_t x[32];
                tmem_ld32(tS + half * 64 + ch * 32, x);
                tmem_wait_ld();
#pragma unroll
                for (int i = 0; i < 32; ++i)
                  if (half * 64 + ch * 32 + i <= lim) m_new = fmaxf(m_new, __uint_as_float(x[i]));
              }
              // In round 0 there is nothing to rescale: its reference is the maximum of all 128 keys, so
              // that m_new is m_ref (what leads here is a sum that is not finite, or no score but
              // -inf).  Nor may it wait for bar_pv_half: the first O_t += of an item follows
              // bar_o_read, on which this warp arrives in the epilogue behind this round.
              if (j > 0) {
                if (half == 1) mbar_wait(smem_u32(&bar_pv_half[t]), phase_s ^ 1u, &abort_word, 11);
                tc_fence_after();
                const float alpha = isinf(m_new) ? 1.f : fast_exp2((m_ref - m_new) * c);
                l *= alpha;
#pragma unroll 1
                for (int cc = 0; cc < DR / 16; ++cc) {
                  uint32_t o[16];
                  tmem_ld16(tO + cc * 16, o);
                  tmem_wait_ld();
#pragma unroll
                  for (int i = 0; i < 16; ++i) o[i] = __float_as_uint(__uint_as_float(o[i]) * alpha);
                  tmem_st16(tO + cc * 16, o);
                }
              }
              m_ref = m_new;
              neg_mc = isinf(m_ref) ? 0.f : -m_ref * c;
              sum = 0.f;
#pragma unroll 1
              for (int ch = 0; ch < 2; ++ch) {
                uint32_t x[32], h[16];
                tmem_ld32(tS + half * 64 + ch * 32, x);
                tmem_wait_ld();
#pragma unroll
                for (int i = 0; i < 32; i += 2) {
                  const int col = half * 64 + ch * 32 + i;
                  const float e0 = col <= lim ? fast_exp2(fmaf(__uint_as_float(x[i]), c, neg_mc)) : 0.f;
                  const float e1 = col + 1 <= lim ? fast_exp2(fmaf(__uint_as_float(x[i + 1]), c, neg_mc)) : 0.f;
                  sum += e0 + e1;
                  h[i >> 1] = pack16x2<kBf16>(e0, e1);
                }
                tmem_st16(tS + half * 32 + ch * 16, h);
              }
            }
            l += sum;
            tmem_wait_st();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(smem_u32(&bar_p_full[t][half]));
          };
          if (j == 0) {
            // over all 128 keys, so that half 1 never has to rescale in round 0 (see there)
            float mx[4];
#pragma unroll
            for (int cc = 0; cc < 4; ++cc) {
              mx[cc] = fmaxf(__uint_as_float(s[cc][0]), __uint_as_float(s[cc][1]));
#pragma unroll
              for (int i = 2; i < 32; i += 2)
                mx[cc] = max3(mx[cc], __uint_as_float(s[cc][i]), __uint_as_float(s[cc][i + 1]));
            }
            m_ref = fmaxf(max3(mx[0], mx[1], mx[2]), mx[3]);
            neg_mc = isinf(m_ref) ? 0.f : -m_ref * c;
          }
          half_round(std::integral_constant<int, 0>{});
          half_round(std::integral_constant<int, 1>{});
        }

        if (j > 0 || !pending) continue;
        // ---- epilogue of the item before: O_t / l -> registers (tensor memory released) -> 16 bit ->
        //      staging box -> TMA store; LSE.  A chunk of a query block leaves fp32 rows instead.
        pending = false;
        const int row = done.q0 + (kPair ? 0 : t * T::kBlockM) + row_in_tile;
        const int nd = t == 0 ? done.n0 : done.n1;
        const bool split = kPair || done.chunk >= 0;
        const int chunk = done.chunk + (kPair ? t : 0);
        // (a row sum that is NaN leaves NaN in both: an LSE of -inf means that the row sees nothing, and
        // whoever joins partial results leaves such a part out)
        const float inv_l = (done_l == 0.f) ? 0.f : 1.f / done_l;
        if (row < p.seqlen_q) {
          const float lse =
              (done_l == 0.f) ? -CUDART_INF_F : (done_m * c + log2f(done_l)) * 0.6931471805599453f;
          const size_t stat = (size_t)done.zh * p.seqlen_q + row;
          if (split) p.lse_part[(size_t)chunk * p.num_heads_total * p.seqlen_q + stat] = lse;
          else p.lse[stat] = lse;
        }
        if (nd > 0) {
          mbar_wait(smem_u32(&bar_o_full[t]), phase_o, &abort_word, 10);
          phase_o ^= 1u;
          tc_fence_after();
        }
        if (split) {
          if (nd == 0) continue;  // LSE = -inf: the combine kernel reads no row
          // (p.row_elems is DR.  Where it is left out here for good, the other code of the kernel comes out slower:
          // without a mask, Z1 H8 N8192 D64 210.9 -> 213.2 us, D96 230.1 -> 233.2, D128 0.2 %; not so for pairs.)
          const int row_elems = DR == D && !kPair ? p.row_elems : DR;
          float* dst = p.o_part + (((size_t)chunk * p.num_heads_total + done.zh) * p.seqlen_q + row) * row_elems;
#pragma unroll 1
          for (int cc = 0; cc < DR / 16; ++cc) {
            uint32_t o[16];
            tmem_ld16(tO + cc * 16, o);
            tmem_wait_ld();
            if (row < p.seqlen_q && ((kPair && DR == D) || cc * 16 < p.row_elems)) {
#pragma unroll
              for (int i = 0; i < 16; i += 4)
                *reinterpret_cast<float4*>(dst + cc * 16 + i) =
                    make_float4(__uint_as_float(o[i]) * inv_l, __uint_as_float(o[i + 1]) * inv_l,
                                __uint_as_float(o[i + 2]) * inv_l, __uint_as_float(o[i + 3]) * inv_l);
            }
          }
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(smem_u32(&bar_o_read[t]));
          continue;
        }
        uint32_t o[DR / 32][32];
        if (nd > 0) {
#pragma unroll
          for (int cc = 0; cc < DR / 32; ++cc) tmem_ld32(tO + cc * 32, o[cc]);
          tmem_wait_ld();
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(smem_u32(&bar_o_read[t]));
        } else {
#pragma unroll
          for (int cc = 0; cc < DR / 32; ++cc)
#pragma unroll
            for (int i = 0; i < 32; ++i) o[cc][i] = 0u;
        }
        // through this group's staging box and TMA stores, 64 columns at a time (per-thread stores of
        // whole rows are uncoalesced and clog the load/store pipe for everybody)
#pragma unroll
        for (int b = 0; b < T::kBoxes; ++b) {
          if (row_in_tile == 0 && stored) tma_wait_group_read<0>();  // the box's last store has been read
          named_bar_sync(1 + t, 128);
#pragma unroll
          for (int ch = 0; ch < (DR - b * 64 < 64 ? 4 : 8); ++ch) {  // 16-byte chunk (8 fp16) of this row
            const uint32_t* w = &o[b * 2 + (ch >> 2)][(ch & 3) * 8];
            uint32_t h4[4];
#pragma unroll
            for (int i = 0; i < 4; ++i)
              h4[i] = pack16x2<kBf16>(__uint_as_float(w[2 * i]) * inv_l, __uint_as_float(w[2 * i + 1]) * inv_l);
            sts128(o_stage + row_in_tile * 128 + ((ch ^ (row_in_tile & 7)) << 4), h4[0], h4[1], h4[2], h4[3]);
          }
          fence_proxy_async_smem();
          named_bar_sync(1 + t, 128);
          if (row_in_tile == 0) {
            tma_store_4d(&tm_o, o_stage, b * 64, done.q0 + t * T::kBlockM, done.h, done.z);
            tma_commit_group();
          }
          stored = true;
        }
      }
      if (it.id < 0) break;
      pending = kPair || it.q0 + t * T::kBlockM < p.seqlen_q;
      done = it;
      done_m = m_ref;
      done_l = l;
    }
    if (row_in_tile == 0) tma_wait_group<0>();
  }

  // ---- teardown
  tc_fence_before();
  __syncthreads();
  if (abort_word != 0) {
    if (threadIdx.x == 0 && p.status != nullptr) atomicCAS(p.status, 0, abort_word);
    // let copies that may still be in flight land before the shared memory is released
    for (int i = 0; i < 64; ++i) __nanosleep(1000);
  }
  if (warp == 9) {
    tc_fence_after();
    tmem_dealloc(tmem_base, T::kTmemCols);
  }
}

// Joins the chunks of the query blocks that were cut: one warp per row, rows from row_begin on.
// Every partial row is normalised; its weight is exp(lse_part - lse).
template <typename E>
__global__ void __launch_bounds__(256)
    fmha_fwd_combine_kernel(const FwdKernelParams p, E* __restrict__ o, long long so_batch, long long so_row,
                            long long so_head, int row_begin, long long total_rows) {
  grid_dependency_wait();
  const long long idx = (long long)blockIdx.x * 8 + (threadIdx.x >> 5);
  if (idx >= total_rows) return;
  const int lane = threadIdx.x & 31;
  const int rows = p.seqlen_q - row_begin;
  const int zh = (int)(idx / rows), row = row_begin + (int)(idx % rows);
  const int chunks = fwd_chunks(p.causal != 0, p.causal_shift, row / 256, p.seqlen_q, (p.seqlen_k + 127) / 128,
                                p.chunk_tiles);
  if (chunks <= 1) return;
  const size_t stat = (size_t)zh * p.seqlen_q + row, plane = (size_t)p.num_heads_total * p.seqlen_q;
  // a part that is NaN makes the row NaN
  float mx = -CUDART_INF_F;
  for (int c = lane; c < chunks; c += 32) mx = max_nan(mx, p.lse_part[c * plane + stat]);
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) mx = max_nan(mx, __shfl_xor_sync(0xffffffffu, mx, off));
  const float base = mx == -CUDART_INF_F ? 0.f : mx;
  float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
  float sum = 0.f;
  const int col = lane * 4;
  for (int c = 0; c < chunks; ++c) {
    const float lp = p.lse_part[c * plane + stat];
    if (lp == -CUDART_INF_F) continue;  // nothing visible in this chunk: its row was not written
    const float w = lp == base ? 1.f : expf(lp - base);  // (inf - inf would be NaN)
    sum += w;
    if (col < p.row_elems) {
      const float4 v = *reinterpret_cast<const float4*>(p.o_part + (c * plane + stat) * p.row_elems + col);
      acc.x += w * v.x, acc.y += w * v.y, acc.z += w * v.z, acc.w += w * v.w;
    }
  }
  const float inv = sum == 0.f ? 0.f : 1.f / sum;
  if (lane == 0) p.lse[stat] = sum == 0.f ? -CUDART_INF_F : base + logf(sum);
  if (col < p.row_elems) {
    constexpr bool kBf16 = std::is_same<E, __nv_bfloat16>::value;
    uint2 v;
    v.x = pack16x2<kBf16>(acc.x * inv, acc.y * inv);
    v.y = pack16x2<kBf16>(acc.z * inv, acc.w * inv);
    *reinterpret_cast<uint2*>(o + (zh / p.heads) * so_batch + row * so_row + (zh % p.heads) * so_head + col) = v;
  }
}

}  // namespace fmha
