// C-ABI launch layer of the B200 attention library (declared in include/fmha_b200.h).
//
// Replaces the host launchers of the reference (kernel/fused_mha_kernel.cu:891-916): validate
// plain-pointer parameters, build the TMA tensor maps, raise the dynamic shared-memory limit,
// launch, and return a status.  Nothing here allocates device memory or synchronises.
#include <cuda.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstdint>
#include <cstdlib>
#include <cstring>
#include <type_traits>

#include "../../include/fmha_b200.h"
#include "aux_kernels.cuh"
#include "bwd_kernel.cuh"
#include "fwd_kernel.cuh"
#include "peer_kernels.cuh"

namespace {

using EncodeTiledFn = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*,
                                   const cuuint64_t*, const cuuint64_t*, const cuuint32_t*,
                                   const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                   CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn get_encode_fn() {
  // resolved once; the pointer is process-wide and immutable afterwards
  static EncodeTiledFn fn = []() -> EncodeTiledFn {
    void* ptr = nullptr;
    cudaDriverEntryPointQueryResult qres;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &ptr, cudaEnableDefault, &qres) !=
            cudaSuccess ||
        qres != cudaDriverEntryPointSuccess)
      return nullptr;
    return reinterpret_cast<EncodeTiledFn>(ptr);
  }();
  return fn;
}

// 16-bit (Z, N, H, D) tensor with element strides -> 4-D map (D, N, H, Z), box 64 x 128 x 1
// x 1, 128-byte swizzle, zero fill outside the tensor
int make_tensor_map(CUtensorMap* map, const void* base, int Z, int N, int H, int D,
                    const FmhaStrides& s, bool bf16) {
  EncodeTiledFn encode = get_encode_fn();
  if (encode == nullptr) return FMHA_ERR_NO_DEVICE;
  // a stride of a size-1 dimension is never used for addressing; make it well-formed
  const int64_t row = (N > 1) ? s.row : (int64_t)H * D;
  const int64_t head = (H > 1) ? s.head : (int64_t)D;
  const int64_t batch = (Z > 1) ? s.batch : row * N;
  const cuuint64_t dims[4] = {(cuuint64_t)D, (cuuint64_t)N, (cuuint64_t)H, (cuuint64_t)Z};
  const cuuint64_t strides[3] = {(cuuint64_t)row * 2, (cuuint64_t)head * 2, (cuuint64_t)batch * 2};
  const cuuint32_t box[4] = {64, 128, 1, 1};
  const cuuint32_t estr[4] = {1, 1, 1, 1};
  const CUresult r = encode(map, bf16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16,
                            4, const_cast<void*>(base), dims,
                            strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                            CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? FMHA_OK : FMHA_ERR_TENSOR_MAP;
}

// fp32 dQ accumulator (Z, N, H, D) contiguous -> 4-D map, box 32 x 128 x 1 x 1 (a tile's 128 query
// rows x 32 columns = 128-byte rows), 128-byte swizzle; used by TMA reduce-add
int make_accum_map(CUtensorMap* map, float* base, int Z, int N, int H, int D, int64_t batch) {
  EncodeTiledFn encode = get_encode_fn();
  if (encode == nullptr) return FMHA_ERR_NO_DEVICE;
  const cuuint64_t dims[4] = {(cuuint64_t)D, (cuuint64_t)N, (cuuint64_t)H, (cuuint64_t)Z};
  if (Z == 1 || batch == 0) batch = (int64_t)N * H * D;
  const cuuint64_t strides[3] = {(cuuint64_t)H * D * 4, (cuuint64_t)D * 4, (cuuint64_t)batch * 4};
  const cuuint32_t box[4] = {32, 128, 1, 1};
  const cuuint32_t estr[4] = {1, 1, 1, 1};
  const CUresult r = encode(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, base, dims, strides, box, estr,
                            CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                            CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? FMHA_OK : FMHA_ERR_TENSOR_MAP;
}

// debug builds (-DFMHA_TIMELINE) set these through fmha_debug_set_timeline for the backward kernel;
// otherwise unused
long long* g_timeline = nullptr;
int g_timeline_block = 0;

constexpr int kMaxDevices = 64;

int current_device() {
  int dev = -1;
  return cudaGetDevice(&dev) == cudaSuccess && dev >= 0 && dev < kMaxDevices ? dev : -1;
}

// SMs of a device, asked once per device (the query costs as much host time as a tensor map)
int sm_count(int dev) {
  static std::atomic<int> cached[kMaxDevices];
  if (dev < 0) return 148;
  int n = cached[dev].load(std::memory_order_relaxed);
  if (n == 0) {
    if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0) return 148;
    cached[dev].store(n, std::memory_order_relaxed);
  }
  return n;
}

// Launches a kernel whose dynamic shared memory needs its limit raised, which is done once per kernel and
// device, and again where a launch is refused: the limit goes with the context when the host resets
// the device.
template <auto kKernel, typename... Args>
bool launch_with_smem(int dev, unsigned grid, unsigned threads, int bytes, cudaStream_t stream, const Args&... args) {
  static std::atomic<bool> raised[kMaxDevices];
  for (int attempt = 0; attempt < 2; ++attempt) {
    if (attempt > 0 || dev < 0 || !raised[dev].load(std::memory_order_acquire)) {
      if (cudaFuncSetAttribute(kKernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes) != cudaSuccess)
        return false;
      if (dev >= 0) raised[dev].store(true, std::memory_order_release);
    }
    kKernel<<<grid, threads, bytes, stream>>>(args...);
    if (cudaGetLastError() == cudaSuccess) return true;
  }
  return false;
}

bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }

int check_strides(const FmhaStrides& s, int N, int H, int Z) {
  if ((N > 1 && (s.row % 8 != 0 || s.row <= 0)) || (H > 1 && (s.head % 8 != 0 || s.head <= 0)) ||
      (Z > 1 && (s.batch % 8 != 0 || s.batch <= 0)))
    return FMHA_ERR_BAD_STRIDE;
  return FMHA_OK;
}

int check_common(int batch, int heads, int seqlen_q, int seqlen_k, int head_dim, float scale,
                 int dtype = FMHA_DTYPE_FP16) {
  if (dtype != FMHA_DTYPE_FP16 && dtype != FMHA_DTYPE_BF16) return FMHA_ERR_BAD_DTYPE;
  if (head_dim != 64 && head_dim != 96 && head_dim != 128) return FMHA_ERR_BAD_HEAD_DIM;
  if (batch <= 0 || heads <= 0 || seqlen_q <= 0 || seqlen_k <= 0) return FMHA_ERR_BAD_SHAPE;
  if (!std::isfinite(scale) || scale == 0.f) return FMHA_ERR_BAD_SHAPE;
  if ((long long)batch * heads * ((seqlen_q + 127) / 128 + 1) >= (1ll << 31) ||
      (long long)batch * heads * ((seqlen_k + 127) / 128 + 1) >= (1ll << 31))
    return FMHA_ERR_TOO_LARGE;
  return FMHA_OK;
}

// head_dim -> (D, DR) = (width the kernels run at, elements per row of the tensors):
// 64 -> (64, 64), 96 -> (128, 96), 128 -> (128, 128)
#define FMHA_DISPATCH_DIMS(head_dim, ...)       \
  if ((head_dim) == 128) {                      \
    constexpr int D = 128, DR = 128;            \
    __VA_ARGS__                                 \
  } else if ((head_dim) == 96) {                \
    constexpr int D = 128, DR = 96;             \
    __VA_ARGS__                                 \
  } else {                                      \
    constexpr int D = 64, DR = 64;              \
    __VA_ARGS__                                 \
  }

fmha::Strides3 to3(const FmhaStrides& s) { return fmha::Strides3{s.batch, s.row, s.head}; }

int round_up_128(int x) { return (x + 127) / 128 * 128; }

// Heads whose CTAs are interleaved in the backward grid (see the coordinates in bwd_kernel.cuh),
// for up to 32 KV tiles per head.  Measured on the fused kernel at Z=8, H=32, N=2048, D=128,
// alternating runs: causal 0.809 ms with one head at a time, 0.794 with groups of 4, 0.778 with 8,
// 0.771 with 16, 0.770 with 24, 0.769 with 32, 0.773 with 37 (the last CTAs of a group and of the
// grid being the short ones); without a mask, where all CTAs are equally long and only the L2
// matters, 1.351 ms with 8 against 1.37-1.40 with 16 to 37.  Longer sequences keep one head at a
// time: their grids are long, and many heads' query tiles would not share the L2.
// FMHA_BWD_HEAD_GROUP overrides (tuning experiments).
// Deterministic, without a mask: the items of a head run staggered by a query tile, and the more heads have their
// first KV tiles in work, the less of that is waiting: as many as fit the L2, up to 32, in even groups.  Whole
// backward, us, one head / 8 / 16 / 32 / this rule: D128 Z2 H16 N2048 433 / 346 / 326 / 311 / 311, Z3 H11 N2048 444 / 398 / 382 /
// 368 / 331 (two groups of 17 and 16), Z1 H8 N8192 1456 / 1117 / 1117 / 1117 / 1117, Z2 H9 N8192 2912 / 2402 / 2357 /
// 2184 / 2246, Z1 H5 N16384 2953 / 2715 / 2715 / 2715 / 2815; D64 Z16 H16 N512 187 / 178 / 168 / 157 / 157, Z2 H16
// N4096 1027 / 753 / 715 / 699 / 698.  Over 60 shapes (D = 64, 96, 128, N = 512 to 16384, 5 to 256 heads) 0.89 to 1.04 of the
// best of the four.  (The waiting is worth more here than the L2, so the limit is higher than the forward's 48 MB.)
int bwd_head_group(int num_kv_blocks, bool causal, bool deterministic, int num_heads, double bytes_per_head) {
  static const int forced = []() {
    const char* e = std::getenv("FMHA_BWD_HEAD_GROUP");
    return e != nullptr ? std::atoi(e) : 0;
  }();
  if (forced >= 1) return forced;
  if (deterministic && !causal) {
    const int most = (int)std::max(1.0, std::min(32.0, 104e6 / bytes_per_head));
    const int groups = (num_heads + most - 1) / most;
    return (num_heads + groups - 1) / groups;
  }
  if (num_kv_blocks > 32) return 1;
  return causal ? 16 : 8;
}

struct BwdWorkspace {
  float* dq_accum;
  float* lse2;
  float* delta;
  unsigned* dq_order;  // one word per (batch*head, query tile), two at least: FMHA_BWD_DETERMINISTIC
  size_t order_bytes;
  size_t bytes;
};

BwdWorkspace carve_workspace(void* ws, int Z, int H, int Nq, int D) {
  BwdWorkspace w;
  const size_t dq_bytes = (size_t)Z * Nq * H * D * sizeof(float);  // multiple of 256
  const size_t stat_bytes = (size_t)Z * H * round_up_128(Nq) * sizeof(float);
  char* base = static_cast<char*>(ws);
  w.dq_accum = reinterpret_cast<float*>(base);
  w.lse2 = reinterpret_cast<float*>(base + dq_bytes);
  w.delta = reinterpret_cast<float*>(base + dq_bytes + stat_bytes);
  w.dq_order = reinterpret_cast<unsigned*>(base + dq_bytes + 2 * stat_bytes);
  w.order_bytes = std::max((size_t)2, (size_t)Z * H * (round_up_128(Nq) / 128)) * sizeof(int);
  w.bytes = dq_bytes + 2 * stat_bytes + (w.order_bytes + 255) / 256 * 256;
  return w;
}

// ---------------------------------------------------------------------------------------
// How the forward's work is cut.  A query block (256 rows) is one item unless that leaves SMs
// idle: then its KV range is cut into chunks of chunk_tiles tiles, each an item of its own that
// leaves an fp32 partial result, and a second kernel joins them.
//
// Measured, uncut / as cut by plan_fwd (chunks), us, fp16, D = 128, the ordinary cut (pairs of chunks: below):
//   64 queries x 8192 keys     8 heads 115.0 / 25.8 (13)
//   256 queries x 4096 keys    8 heads 59.5 / 26.8 (8), 64: 61.7 / 53.4 (2)
//   causal, 1 head             N = 1024 24.2 / 22.7 (4), 4096 59.8 / 28.8 (8), 16384 214.5 / 113.7 (6)
//   causal, 4 heads            N = 1024 24.3 / 22.7 (4), 4096 60.9 / 43.2 (3)
// and what it leaves uncut, uncut / cut in two: 64 heads of 512 x
// 2048 37.0 / 67.7, causal 16 heads N = 4096 63.6 / 97.9, 4 heads N = 16384 227.9 / 261.5.  Over 150 shapes
// (D = 64 and 128, 1 to 296 heads) no ordinary cut of its was slower than none.  It is a rough estimate on
// the cautious side: where the items are just fewer than the SMs a cut that it does not make
// would be up to 1.4 times as fast (causal, 4 heads, N = 8192: 113.1 / 80.3), and under a mask fewer chunks
// than it makes up to 1.3 times (1 head, N = 16384: 113.7 in 6, 86.6 in 4).
// ---------------------------------------------------------------------------------------
struct FwdPlan {
  int chunk_tiles = 1 << 30;
  int max_chunks = 1;      // of any query block
  int items_per_head = 0;
  int first_cut_row = 0;   // rows from here on belong to cut query blocks
  size_t workspace = 0;    // bytes of the partial results
  bool pair = false;       // up to 128 query rows: an item is two chunks, both in work
};

FwdPlan plan_fwd(const FmhaFwdParams* p, int sms) {
  FwdPlan plan;
  const bool causal = p->causal != 0;
  const int nqb = (p->seqlen_q + 255) / 256, nk = (p->seqlen_k + 127) / 128;
  const double heads = (double)p->batch * p->heads;
  plan.items_per_head = nqb;
  // In units of one round (256 query rows x 128 keys; about 1.2 us with the whole chip at work, 1.9 us
  // with a few SMs): an item costs its rounds and half a round of its own.
  auto visible = [&](int qb) {
    return fmha::fwd_visible_tiles(causal, p->causal_shift, std::min(qb * 256 + 255, p->seqlen_q - 1), nk);
  };
  const int n_max = visible(nqb - 1);
  if (n_max < 4) return plan;
  const bool can_pair = p->seqlen_q <= 128 && n_max >= 16;  // (shorter: nothing to gain beyond the noise)
  if (heads * nqb > 8.0 * sms && !can_pair) return plan;  // enough items to balance
  auto cost = [&](int chunk, int& items) {  // makespan with chunks of `chunk` tiles
    double total = 0;
    items = 0;
    for (int qb = causal ? 0 : nqb - 1; qb < nqb; ++qb) {
      const int n = visible(qb), c = n <= chunk ? 1 : (n + chunk - 1) / chunk;
      items += c;
      total += n + 0.5 * c;
    }
    const int rep = causal ? 1 : nqb;
    items *= rep;
    total *= rep;
    const int longest = std::min(chunk, n_max);
    // equal items run in whole waves; unequal ones, longest first, fill the gaps
    const double waves = causal ? std::max(longest + 0.5, total * heads / sms + 0.5 * (longest < n_max ? longest : 2))
                                : std::ceil(items * heads / sms) * (longest + 0.5);
    return waves;
  };
  int items = 0;
  double best = 0.85 * cost(n_max, items);  // a cut has to be worth it: the estimate is rough
  // without a mask the work per SM is what it is unless SMs idle; under one, unless one block dominates
  for (int k = 2; heads * nqb <= 8.0 * sms && k <= 64 && n_max / k >= 2; ++k) {
    const int chunk = (n_max + k - 1) / k;
    const double t0 = cost(chunk, items);
    // the joining kernel: its launch, and the partial rows written and read (at about 4 TB/s)
    const double t = t0 + 2.5 + heads * items * 256.0 * p->head_dim * 8.0 / 4e12 / 1.2e-6;
    if (t < best) {
      best = t;
      plan.chunk_tiles = chunk;
      plan.items_per_head = items;
      plan.max_chunks = (n_max + chunk - 1) / chunk;
    }
    if (heads * items > 8.0 * sms) break;
  }
  if (can_pair) {
    // Few queries: an item with one query tile is a chain of MMA, softmax and MMA, and half of the SM idles.  Items of
    // two chunks, which idle less but leave partial rows, or the plan so far?  Estimates of each, in us: a fixed part
    // and one per chunk (the join); the rounds of the longest item, wave after wave, and K and V from HBM, of which the
    // longer one counts and the shorter one a little; the partial rows, more beyond 40 MB, which the L2 does not keep.
    // A round of one tile takes 1.5 to 1.7 us, of two chunks 1.8 to 2.1; rows that a tile does not have cost 0.1 to
    // 0.2, for they are masked.  Pairs have to be estimated 8 % faster than whole items, 4 % faster than the ordinary
    // cut.  Constants from 2918 shapes (D = 64, 96, 128, 1 to 128 rows, 1921 to 32768 keys, 8 to 1200 heads, bf16),
    // every way timed, searched on one half of them and as good on the other: 0.5 % slower than the best way on average,
    // by more than 3 % in 110 of them, 17 % at most (without pairs 22 % slower on average).  148 heads of 128 rows over
    // 4096 keys, D = 128: whole 59 us, one pair 73; 64 rows over 8192, 64 heads: whole 113, two pairs 54.
    // Padded batches: the lengths are not known here.  Taken as 0.56 of the whole on average, and waves and margins as
    // they were best for 1639 shapes with 8 entries of n/8 to n keys: 1.2 % slower than the best way on average, 22 %
    // at most (without pairs 27 % on average).
    const double wide = p->head_dim / 64.0;
    const bool full = p->seqlen_q == 128, padded = p->seqused_k != nullptr;
    const double one_tile = 1.37 + 0.19 * wide - (full ? 0.2 : 0.0);
    const double two_chunks = 1.52 + 0.32 * wide - (full ? 0.1 : 0.0);
    // items per head; of a padded batch, the part of their rounds that exists
    auto waves = [&](int items, double filled) {
      const double per_sm = heads * items / sms;
      if (!padded || per_sm <= 1) return std::ceil(per_sm);
      return std::max(1.0, per_sm * filled + 0.25 * std::ceil(per_sm * filled));
    };
    auto time = [&](double rounds_us, int chunks) {
      const double part = padded ? 0.56 : 1.0;
      const double kv_us = part * heads * n_max * 128 * p->head_dim * 4 / 7.1e6;
      const double parts_mb = part * heads * chunks * p->seqlen_q * p->head_dim * 8 / 1e6;
      const double x = rounds_us * rounds_us, y = kv_us * kv_us;
      return 6.0 + 0.27 * chunks + std::sqrt(std::sqrt(x * x + y * y)) + 0.34 * parts_mb +
             0.1 * std::max(0.0, parts_mb - 40);
    };
    const int chunks = plan.max_chunks;
    double most = chunks > 1 ? (padded ? 0.93 : 0.96) *
                                   time(waves(chunks, 0.58) * (one_tile * plan.chunk_tiles + 2.5), chunks)
                             : (padded ? 0.88 : 0.92) * (time(waves(1, 0.67) * (one_tile * n_max - 0.5), 0) - 0.5);
    for (int k = 1; k <= 32; ++k) {
      const int chunk = (n_max + 2 * k - 1) / (2 * k), n = (n_max + 2 * chunk - 1) / (2 * chunk);
      if (chunk < 4) break;
      const double t = time(waves(n, 0.58 + 0.27 / n) * (two_chunks * chunk + 1.3), 2 * n);
      if (t < most) {
        most = t;
        plan.pair = true;
        plan.chunk_tiles = chunk;
        plan.items_per_head = n;
        plan.max_chunks = 2 * n;
      }
    }
  }
  if (plan.max_chunks > 1) {
    int qb = 0;
    while (visible(qb) <= plan.chunk_tiles) ++qb;
    plan.first_cut_row = qb * 256;
    plan.workspace = (size_t)plan.max_chunks * p->batch * p->heads * p->seqlen_q * (p->head_dim + 1) * sizeof(float);
  }
  return plan;
}

// Heads whose items are interleaved in the forward's order, so that the last items are the short
// ones of a causal mask: as many as have their K and V in 48 of the 126 MB of L2.  One head at a time /
// 24 / 48 / 96 / 1000 MB, us, fp16: Z8 H32 N2048 D128 causal 371 / 328 / 328 / 343 / 377, without a mask 607 /
// 536 / 546 / 604 / 652, Z4 H32 N4096 causal 637 / 572 / 561 / 592 / 648, Z2 H32 N8192 without a mask 2038 /
// 1973 / 1988 / 2070 / 2161.
int fwd_head_group(const FmhaFwdParams* p) {
  const double kv_bytes = 4.0 * p->seqlen_k * p->head_dim;
  return (int)std::max(1.0, std::min((double)p->batch * p->heads, 48e6 / kv_bytes));
}

// D is the head dimension the tiles have; the tensors have DR <= D elements per row (96 runs on the tiles of
// 128: the tensor maps describe 96 columns, the loads fill the rest of a 128-wide tile with zeros, the MMAs leave it
// out and the stores clip it)
template <int D, bool kBf16, int DR = D>
int launch_fwd(const FmhaFwdParams* p, void* workspace, size_t workspace_bytes, cudaStream_t stream) {
  using T = fmha::FwdTraits<D, kBf16, DR>;
  using TPair = fmha::FwdTraits<D, kBf16, DR, true>;
  using E = typename std::conditional<kBf16, __nv_bfloat16, __half>::type;
  CUtensorMap tq, tk, tv, to;
  int rc;
  constexpr int Dr = DR;
  if ((rc = make_tensor_map(&tq, p->q, p->batch, p->seqlen_q, p->heads, Dr, p->q_strides, kBf16)))
    return rc;
  if ((rc = make_tensor_map(&tk, p->k, p->batch, p->seqlen_k, p->heads, Dr, p->k_strides, kBf16)))
    return rc;
  if ((rc = make_tensor_map(&tv, p->v, p->batch, p->seqlen_k, p->heads, Dr, p->v_strides, kBf16)))
    return rc;
  if ((rc = make_tensor_map(&to, p->o, p->batch, p->seqlen_q, p->heads, Dr, p->o_strides, kBf16)))
    return rc;
  const int dev = current_device();
  const int sms = std::max(1, sm_count(dev) - std::max(0, (int)p->sm_margin));
  FwdPlan plan;
  if (workspace != nullptr) plan = plan_fwd(p, sms);
  if (plan.workspace > workspace_bytes || plan.max_chunks <= 1) {
    plan = FwdPlan();
    plan.items_per_head = (p->seqlen_q + 255) / 256;
  }
  fmha::FwdKernelParams kp;
  kp.lse = p->lse;
  kp.heads = p->heads;
  kp.seqlen_q = p->seqlen_q;
  kp.seqlen_k = p->seqlen_k;
  kp.num_q_blocks = (p->seqlen_q + 255) / 256;
  kp.num_heads_total = p->batch * p->heads;
  kp.head_group = fwd_head_group(p);
  kp.items_per_head = plan.items_per_head;
  kp.num_items = plan.items_per_head * kp.num_heads_total;
  kp.chunk_tiles = plan.chunk_tiles;
  kp.scale_log2 = std::fabs(p->scale) * 1.4426950408889634f;
  kp.negate = p->scale < 0.f;
  kp.causal = p->causal ? 1 : 0;
  kp.causal_shift = p->causal_shift;
  kp.status = p->status;
  kp.seqused_q = p->seqused_q;
  kp.seqused_k = p->seqused_k;
  kp.row_elems = Dr;
  kp.o_part = nullptr;
  kp.lse_part = nullptr;
  if (plan.max_chunks > 1) {
    kp.o_part = static_cast<float*>(workspace);
    kp.lse_part = kp.o_part + (size_t)plan.max_chunks * kp.num_heads_total * p->seqlen_q * Dr;
  }
  // One block per item, taken over by running blocks; dealt out instead where every item has an SM
  // of its own (nothing to take over) or the caller wants SMs left free.
  kp.deal = kp.num_items <= sms || p->sm_margin > 0;
  const unsigned grid = kp.deal ? (unsigned)std::min(kp.num_items, sms) : (unsigned)kp.num_items;
  const bool launched =
      plan.pair ? launch_with_smem<fmha::fmha_fwd_kernel<D, kBf16, true, DR>>(dev, grid, TPair::kThreads, TPair::kSmemBytes,
                                                                              stream, tq, tk, tv, to, kp)
                : launch_with_smem<fmha::fmha_fwd_kernel<D, kBf16, false, DR>>(dev, grid, T::kThreads, T::kSmemBytes,
                                                                               stream, tq, tk, tv, to, kp);
  if (!launched) return FMHA_ERR_LAUNCH;
  if (plan.max_chunks > 1) {
    const long long rows = (long long)kp.num_heads_total * (p->seqlen_q - plan.first_cut_row);
    // Launched as soon as no block of the chunks is left to start or run, and not only when their writes are visible:
    // it waits for those itself.  64 queries x 8192 keys, 64 heads, D = 128, bf16, call after call 57.7 -> 55.6 us; 216
    // shapes 1.06 times as fast, in a captured graph no difference.  Not so the kernels of a backward: Z4 H16 N1024 D64
    // causal 49.3 -> 47.1 us on the GPU, but this launch takes the host half a microsecond longer, and small training
    // steps wait for the host (76.3 -> 77.7).
    cudaLaunchAttribute early;
    early.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    early.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t config = {};
    config.gridDim = dim3((unsigned)((rows + 7) / 8));
    config.blockDim = dim3(256);
    config.stream = stream;
    config.attrs = &early;
    config.numAttrs = 1;
    if (cudaLaunchKernelEx(&config, fmha::fmha_fwd_combine_kernel<E>, kp, static_cast<E*>(p->o),
                           (long long)p->o_strides.batch, (long long)p->o_strides.row, (long long)p->o_strides.head,
                           plan.first_cut_row, rows) != cudaSuccess) {
      (void)cudaGetLastError();
      return FMHA_ERR_LAUNCH;
    }
  }
  return FMHA_OK;
}

// D: the head dimension the kernels run at; DR <= D: what the tensors have (p->head_dim)
template <int D, bool kBf16, int DR = D>
int launch_bwd(const FmhaBwdParams* p, const BwdWorkspace& w, cudaStream_t stream) {
  using T = fmha::BwdTraits<D, kBf16>;
  using E = typename std::conditional<kBf16, __nv_bfloat16, __half>::type;
  const int Z = p->batch, H = p->heads, Nq = p->seqlen_q, Nk = p->seqlen_k;
  const int Nq_pad = round_up_128(Nq);
  constexpr int Dr = DR;
  // Where the call both zeroes and converts the accumulator, the conversion need not read the rows of padding
  // queries.  They are zeroed all the same, for later calls on this workspace, unless the caller has none in mind.
  const bool whole = !(p->flags & (FMHA_BWD_KEEP_WORKSPACE | FMHA_BWD_PREPROCESS_ONLY | FMHA_BWD_SKIP_DQ_CONVERT));
  const int zero_padding = whole && (p->flags & FMHA_BWD_DROP_WORKSPACE) ? 0 : 1;

  if (!(p->flags & FMHA_BWD_KEEP_WORKSPACE)) {
    const long long rows = (long long)Z * H * Nq_pad;
    constexpr int rows_per_block = 256 / (D / 8);
    const unsigned grid = (unsigned)((rows + rows_per_block - 1) / rows_per_block);
    fmha::fmha_bwd_preprocess_kernel<D, E, DR><<<grid, 256, 0, stream>>>(
        static_cast<const E*>(p->o), to3(p->o_strides), static_cast<const E*>(p->dout),
        to3(p->dout_strides), p->lse, w.dq_accum, w.lse2, w.delta, H, Nq, Nq_pad, rows, p->seqused_q, zero_padding);
    if (cudaGetLastError() != cudaSuccess) return FMHA_ERR_LAUNCH;
  }
  if (p->flags & FMHA_BWD_PREPROCESS_ONLY) return FMHA_OK;

  {
    CUtensorMap tq, tk, tv, tdo, tdk, tdv, tacc;
    int rc;
    if ((rc = make_accum_map(&tacc, w.dq_accum, Z, Nq, H, Dr, 0))) return rc;
    if ((rc = make_tensor_map(&tq, p->q, Z, Nq, H, Dr, p->q_strides, kBf16))) return rc;
    if ((rc = make_tensor_map(&tk, p->k, Z, Nk, H, Dr, p->k_strides, kBf16))) return rc;
    if ((rc = make_tensor_map(&tv, p->v, Z, Nk, H, Dr, p->v_strides, kBf16))) return rc;
    if ((rc = make_tensor_map(&tdo, p->dout, Z, Nq, H, Dr, p->dout_strides, kBf16))) return rc;
    // with fp32 accumulation the 16-bit outputs are not touched
    auto kv_out_map = [&](CUtensorMap* map, float* accum, void* out, const FmhaStrides& strides) {
      return accum != nullptr ? make_accum_map(map, accum, Z, Nk, H, Dr, p->accum_batch_stride)
                              : make_tensor_map(map, out, Z, Nk, H, Dr, strides, kBf16);
    };
    if ((rc = kv_out_map(&tdk, p->dk_accum, p->dk, p->dk_strides))) return rc;
    if ((rc = kv_out_map(&tdv, p->dv_accum, p->dv, p->dv_strides))) return rc;
    fmha::BwdKernelParams kp;
    kp.neg_lse2 = w.lse2;
    kp.neg_delta = w.delta;
    kp.dk_accum = p->dk_accum;
    kp.dv_accum = p->dv_accum;
    kp.accum_batch_stride =
        p->accum_batch_stride > 0 ? p->accum_batch_stride : (long long)Nk * H * Dr;
    kp.accum_overwrite = (p->flags & FMHA_BWD_ACCUM_OVERWRITE) ? 1 : 0;
    kp.heads = H;
    kp.seqlen_q = Nq;
    kp.seqlen_k = Nk;
    kp.seqlen_q_pad = Nq_pad;
    kp.num_kv_blocks = (Nk + 127) / 128;
    kp.num_heads_total = Z * H;
    // q, dout, dQ accumulator; k, v
    const double bytes_per_head = ((double)Nq * 8 + (double)Nk * 4) * Dr;
    kp.head_group = bwd_head_group(kp.num_kv_blocks, p->causal != 0, (p->flags & FMHA_BWD_DETERMINISTIC) != 0,
                                   kp.num_heads_total, bytes_per_head);
    kp.q_tile_begin = p->q_row_begin / 128;
    kp.dk = static_cast<uint16_t*>(p->dk);
    kp.dv = static_cast<uint16_t*>(p->dv);
    kp.dk_strides = to3(p->dk_strides);
    kp.dv_strides = to3(p->dv_strides);
    kp.scale = p->scale;
    kp.scale_log2 = p->scale * 1.4426950408889634f;
    kp.causal = p->causal ? 1 : 0;
    kp.causal_shift = p->causal_shift;
    kp.status = p->status;
    kp.seqused_q = p->seqused_q;
    kp.seqused_k = p->seqused_k;
    kp.dq_order = nullptr;
    if (p->flags & FMHA_BWD_DETERMINISTIC) {
      // a memset node, not an allocation; every call starts its own count at zero
      if (cudaMemsetAsync(w.dq_order, 0, w.order_bytes, stream) != cudaSuccess) return FMHA_ERR_LAUNCH;
      kp.dq_order = w.dq_order;
    }
    kp.num_items = kp.num_kv_blocks * H * Z;
    // One block per item, taken over by running blocks, unless every item has an SM of its own.  Deterministic: a block
    // per SM, which draw the items from a counter.
    const int dev = current_device();
    kp.deal = kp.num_items <= sm_count(dev);
    const unsigned grid = kp.dq_order != nullptr ? std::min(kp.num_items, sm_count(dev)) : kp.num_items;
    kp.timeline = g_timeline;
    kp.timeline_block = g_timeline_block;
    constexpr int smem = fmha::bwd_smem_bytes<D, kBf16>();
    const bool launched =
        kp.dq_order != nullptr
            ? launch_with_smem<fmha::fmha_bwd_kernel<D, kBf16, DR, true>>(dev, grid, T::kThreads, smem, stream, tq, tk, tv,
                                                                          tdo, tdk, tdv, tacc, kp)
            : launch_with_smem<fmha::fmha_bwd_kernel<D, kBf16, DR>>(dev, grid, T::kThreads, smem, stream, tq, tk, tv, tdo,
                                                                    tdk, tdv, tacc, kp);
    if (!launched) return FMHA_ERR_LAUNCH;
  }

  if (!(p->flags & FMHA_BWD_SKIP_DQ_CONVERT)) {
    const long long rows = (long long)Z * Nq * H;
    constexpr int rows_per_block = 256 / (D / 8);
    const unsigned grid = (unsigned)((rows + rows_per_block - 1) / rows_per_block);
    fmha::fmha_bwd_convert_dq_kernel<D, E, DR><<<grid, 256, 0, stream>>>(
        w.dq_accum, static_cast<E*>(p->dq), to3(p->dq_strides), H, Nq, p->scale, rows,
        whole ? p->seqused_q : nullptr);
    if (cudaGetLastError() != cudaSuccess) return FMHA_ERR_LAUNCH;
  }
  return FMHA_OK;
}

FmhaStrides dense_strides(int n, int head, int k) {
  FmhaStrides s;
  s.head = k;
  s.row = (int64_t)head * k;
  s.batch = (int64_t)n * head * k;
  return s;
}

// ---------------------------------------------------------------------------------------
// Built-in scratch for fmha_bwd_static_scratch: part of the device image, so it exists on every
// GPU that loads the library and costs no allocation call at run time.
// In HOST code the name below is only a handle for cudaGetSymbolAddress: it is not a device
// address and must never be handed to a kernel.
// ---------------------------------------------------------------------------------------
static __device__ __align__(256) unsigned char g_fmha_static_scratch[FMHA_STATIC_SCRATCH_BYTES];

std::atomic<void*> g_static_scratch_addr[kMaxDevices];  // per device, filled on first use

// Device address of the scratch area on the CURRENT device, or nullptr (rc set) on failure.
void* static_scratch_for_current_device(int* rc) {
  const int dev = current_device();
  if (dev < 0) {
    *rc = FMHA_ERR_NO_DEVICE;
    return nullptr;
  }
  void* ptr = g_static_scratch_addr[dev].load(std::memory_order_acquire);
  if (ptr == nullptr) {
    // once per device, with that device current; the address differs from device to device
    if (cudaGetSymbolAddress(&ptr, g_fmha_static_scratch) != cudaSuccess || ptr == nullptr) {
      (void)cudaGetLastError();
      *rc = FMHA_ERR_NO_DEVICE;
      return nullptr;
    }
    g_static_scratch_addr[dev].store(ptr, std::memory_order_release);
  }
  *rc = FMHA_OK;
  return ptr;
}

}  // namespace

extern "C" {

int fmha_fwd(const FmhaFwdParams* p, void* stream) { return fmha_fwd_with_workspace(p, nullptr, 0, stream); }

int fmha_fwd_with_workspace(const FmhaFwdParams* p, void* workspace, size_t workspace_bytes, void* stream) {
  if (p == nullptr || p->q == nullptr || p->k == nullptr || p->v == nullptr || p->o == nullptr ||
      p->lse == nullptr)
    return FMHA_ERR_NULL_POINTER;
  int rc = check_common(p->batch, p->heads, p->seqlen_q, p->seqlen_k, p->head_dim, p->scale, p->dtype);
  if (rc) return rc;
  if (!aligned16(p->q) || !aligned16(p->k) || !aligned16(p->v) || !aligned16(p->o) || !aligned16(workspace))
    return FMHA_ERR_BAD_ALIGNMENT;
  if ((rc = check_strides(p->q_strides, p->seqlen_q, p->heads, p->batch))) return rc;
  if ((rc = check_strides(p->k_strides, p->seqlen_k, p->heads, p->batch))) return rc;
  if ((rc = check_strides(p->v_strides, p->seqlen_k, p->heads, p->batch))) return rc;
  if ((rc = check_strides(p->o_strides, p->seqlen_q, p->heads, p->batch))) return rc;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  if (p->dtype == FMHA_DTYPE_BF16) {
    FMHA_DISPATCH_DIMS(p->head_dim, return launch_fwd<D, true, DR>(p, workspace, workspace_bytes, s);)
  } else {
    FMHA_DISPATCH_DIMS(p->head_dim, return launch_fwd<D, false, DR>(p, workspace, workspace_bytes, s);)
  }
}

size_t fmha_fwd_workspace_bytes(const FmhaFwdParams* p) {
  if (p == nullptr || check_common(p->batch, p->heads, p->seqlen_q, p->seqlen_k, p->head_dim, p->scale, p->dtype))
    return 0;
  return plan_fwd(p, std::max(1, sm_count(current_device()) - std::max(0, (int)p->sm_margin))).workspace;
}

size_t fmha_bwd_workspace_bytes(const FmhaBwdParams* p) {
  if (p == nullptr || p->batch <= 0 || p->heads <= 0 || p->seqlen_q <= 0 || p->head_dim <= 0)
    return 0;
  return carve_workspace(nullptr, p->batch, p->heads, p->seqlen_q, p->head_dim).bytes;
}

int fmha_bwd(const FmhaBwdParams* p, void* workspace, size_t workspace_bytes, void* stream) {
  if (p == nullptr || p->q == nullptr || p->k == nullptr || p->v == nullptr || p->dout == nullptr ||
      p->lse == nullptr)
    return FMHA_ERR_NULL_POINTER;
  const bool keep = (p->flags & FMHA_BWD_KEEP_WORKSPACE) != 0;
  const bool pre_only = (p->flags & FMHA_BWD_PREPROCESS_ONLY) != 0;
  const bool skip_convert = pre_only || (p->flags & FMHA_BWD_SKIP_DQ_CONVERT) != 0;
  if (keep && pre_only) return FMHA_ERR_WORKSPACE;
  if (!keep && p->o == nullptr) return FMHA_ERR_NULL_POINTER;
  if (!skip_convert && p->dq == nullptr) return FMHA_ERR_NULL_POINTER;
  if (p->dk_accum == nullptr && p->dk == nullptr) return FMHA_ERR_NULL_POINTER;
  if (p->dv_accum == nullptr && p->dv == nullptr) return FMHA_ERR_NULL_POINTER;
  int rc = check_common(p->batch, p->heads, p->seqlen_q, p->seqlen_k, p->head_dim, p->scale, p->dtype);
  if (rc) return rc;
  if (!aligned16(p->q) || !aligned16(p->k) || !aligned16(p->v) || !aligned16(p->dout) ||
      (!keep && !aligned16(p->o)) || (!skip_convert && !aligned16(p->dq)) ||
      (p->dk_accum == nullptr && !aligned16(p->dk)) || (p->dv_accum == nullptr && !aligned16(p->dv)) ||
      !aligned16(p->dk_accum) || !aligned16(p->dv_accum))
    return FMHA_ERR_BAD_ALIGNMENT;
  if ((rc = check_strides(p->q_strides, p->seqlen_q, p->heads, p->batch))) return rc;
  if ((rc = check_strides(p->k_strides, p->seqlen_k, p->heads, p->batch))) return rc;
  if ((rc = check_strides(p->v_strides, p->seqlen_k, p->heads, p->batch))) return rc;
  if ((rc = check_strides(p->dout_strides, p->seqlen_q, p->heads, p->batch))) return rc;
  if (!keep && (rc = check_strides(p->o_strides, p->seqlen_q, p->heads, p->batch))) return rc;
  if (!skip_convert && (rc = check_strides(p->dq_strides, p->seqlen_q, p->heads, p->batch)))
    return rc;
  if (p->dk_accum == nullptr && (rc = check_strides(p->dk_strides, p->seqlen_k, p->heads, p->batch)))
    return rc;
  if (p->dv_accum == nullptr && (rc = check_strides(p->dv_strides, p->seqlen_k, p->heads, p->batch)))
    return rc;
  if (p->q_row_begin < 0 || p->q_row_begin % 128 != 0 ||
      (p->q_row_begin != 0 && p->q_row_begin >= p->seqlen_q))
    return FMHA_ERR_BAD_SHAPE;
  if (p->dk_accum != nullptr || p->dv_accum != nullptr) {
    // the epilogue adds with 16-byte accesses at accum + z * stride: the stride must keep them
    // aligned, and batch entries must not overlap
    const int64_t st = p->accum_batch_stride;
    if (st < 0 || (st != 0 && (st % 4 != 0 || st < (int64_t)p->seqlen_k * p->heads * p->head_dim)))
      return FMHA_ERR_BAD_STRIDE;
  }
  const BwdWorkspace w = carve_workspace(workspace, p->batch, p->heads, p->seqlen_q, p->head_dim);
  if (workspace == nullptr || workspace_bytes < w.bytes) return FMHA_ERR_WORKSPACE;
  if (!aligned16(workspace)) return FMHA_ERR_BAD_ALIGNMENT;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  if (p->dtype == FMHA_DTYPE_BF16)
    return p->head_dim == 128 ? launch_bwd<128, true>(p, w, s)
           : p->head_dim == 96 ? launch_bwd<128, true, 96>(p, w, s)
                               : launch_bwd<64, true>(p, w, s);
  return p->head_dim == 128 ? launch_bwd<128, false>(p, w, s)
         : p->head_dim == 96 ? launch_bwd<128, false, 96>(p, w, s)
                             : launch_bwd<64, false>(p, w, s);
}

int fmha_bwd_static_scratch(const FmhaBwdParams* p, void* stream) {
  if (p == nullptr) return FMHA_ERR_NULL_POINTER;
  // the shared area cannot carry an accumulator over from an earlier call, nor hand an
  // unconverted fp32 dQ to a later one (the caller has no address for it)
  if (p->flags & (FMHA_BWD_KEEP_WORKSPACE | FMHA_BWD_PREPROCESS_ONLY | FMHA_BWD_SKIP_DQ_CONVERT))
    return FMHA_ERR_WORKSPACE;
  if (p->batch <= 0 || p->heads <= 0 || p->seqlen_q <= 0 || p->head_dim <= 0)
    return FMHA_ERR_BAD_SHAPE;
  const size_t need = fmha_bwd_workspace_bytes(p);
  if (need == 0 || need > (size_t)FMHA_STATIC_SCRATCH_BYTES) return FMHA_ERR_TOO_LARGE;
  int rc = FMHA_OK;
  void* scratch = static_scratch_for_current_device(&rc);
  if (scratch == nullptr) return rc;
  // same validation, kernels and launch order as the caller-workspace entry point
  FmhaBwdParams own = *p;
  own.flags |= FMHA_BWD_DROP_WORKSPACE;  // the caller never sees it
  return fmha_bwd(&own, scratch, (size_t)FMHA_STATIC_SCRATCH_BYTES, stream);
}

int fmha_bwd_convert_dq(const void* workspace, void* dq, FmhaStrides dq_strides, int32_t batch,
                        int32_t heads, int32_t seqlen_q, int32_t head_dim, float scale,
                        int32_t dtype, void* stream) {
  if (workspace == nullptr || dq == nullptr) return FMHA_ERR_NULL_POINTER;
  if (dtype != FMHA_DTYPE_FP16 && dtype != FMHA_DTYPE_BF16) return FMHA_ERR_BAD_DTYPE;
  if (head_dim != 64 && head_dim != 96 && head_dim != 128) return FMHA_ERR_BAD_HEAD_DIM;
  if (batch <= 0 || heads <= 0 || seqlen_q <= 0) return FMHA_ERR_BAD_SHAPE;
  if (!aligned16(workspace) || !aligned16(dq)) return FMHA_ERR_BAD_ALIGNMENT;
  int rc = check_strides(dq_strides, seqlen_q, heads, batch);
  if (rc) return rc;
  const long long rows = (long long)batch * seqlen_q * heads;
  const int rows_per_block = 256 / ((head_dim > 64 ? 128 : 64) / 8);  // 16 or 8 threads per row
  const unsigned grid = (unsigned)((rows + rows_per_block - 1) / rows_per_block);
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const float* acc = static_cast<const float*>(workspace);
  const fmha::Strides3 sd = to3(dq_strides);
  if (dtype == FMHA_DTYPE_BF16) {
    auto* out = static_cast<__nv_bfloat16*>(dq);
    FMHA_DISPATCH_DIMS(head_dim,
                       fmha::fmha_bwd_convert_dq_kernel<D, __nv_bfloat16, DR><<<grid, 256, 0, s>>>(
                           acc, out, sd, heads, seqlen_q, scale, rows, nullptr);)
  } else {
    auto* out = static_cast<__half*>(dq);
    FMHA_DISPATCH_DIMS(head_dim,
                       fmha::fmha_bwd_convert_dq_kernel<D, __half, DR><<<grid, 256, 0, s>>>(
                           acc, out, sd, heads, seqlen_q, scale, rows, nullptr);)
  }
  return cudaGetLastError() == cudaSuccess ? FMHA_OK : FMHA_ERR_LAUNCH;
}

int fmha_merge_rows(float* o_acc, float* lse_acc, const void* o_part, FmhaStrides o_part_strides,
                    const float* lse_part, void* o_out, int32_t batch, int32_t heads, int32_t rows,
                    int32_t acc_rows, int32_t row_offset, int32_t head_dim, int32_t dtype,
                    void* stream) {
  if (o_acc == nullptr || lse_acc == nullptr || o_part == nullptr || lse_part == nullptr)
    return FMHA_ERR_NULL_POINTER;
  if (dtype != FMHA_DTYPE_FP16 && dtype != FMHA_DTYPE_BF16) return FMHA_ERR_BAD_DTYPE;
  if (head_dim != 64 && head_dim != 96 && head_dim != 128) return FMHA_ERR_BAD_HEAD_DIM;
  if (batch <= 0 || heads <= 0 || rows <= 0 || row_offset < 0 ||
      (long long)row_offset + rows > (long long)acc_rows)
    return FMHA_ERR_BAD_SHAPE;
  if (!aligned16(o_acc) || !aligned16(o_part) || !aligned16(o_out)) return FMHA_ERR_BAD_ALIGNMENT;
  int rc = check_strides(o_part_strides, rows, heads, batch);
  if (rc) return rc;
  const long long total = (long long)batch * rows * heads;
  const int rows_per_block = 256 / ((head_dim > 64 ? 128 : 64) / 8);  // 16 or 8 threads per row
  const unsigned grid = (unsigned)((total + rows_per_block - 1) / rows_per_block);
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const fmha::Strides3 sp = to3(o_part_strides);
  if (dtype == FMHA_DTYPE_BF16) {
    auto* part = static_cast<const __nv_bfloat16*>(o_part);
    auto* out = static_cast<__nv_bfloat16*>(o_out);
    FMHA_DISPATCH_DIMS(head_dim,
                       fmha::fmha_merge_kernel<D, __nv_bfloat16, DR><<<grid, 256, 0, s>>>(
                           o_acc, lse_acc, part, sp, lse_part, out, heads, rows, acc_rows, row_offset, total);)
  } else {
    auto* part = static_cast<const __half*>(o_part);
    auto* out = static_cast<__half*>(o_out);
    FMHA_DISPATCH_DIMS(head_dim,
                       fmha::fmha_merge_kernel<D, __half, DR><<<grid, 256, 0, s>>>(
                           o_acc, lse_acc, part, sp, lse_part, out, heads, rows, acc_rows, row_offset, total);)
  }
  return cudaGetLastError() == cudaSuccess ? FMHA_OK : FMHA_ERR_LAUNCH;
}

int fmha_merge(float* o_acc, float* lse_acc, const void* o_part, FmhaStrides o_part_strides,
               const float* lse_part, void* o_out, int32_t batch, int32_t heads, int32_t rows,
               int32_t head_dim, int32_t dtype, void* stream) {
  return fmha_merge_rows(o_acc, lse_acc, o_part, o_part_strides, lse_part, o_out, batch, heads,
                         rows, rows, 0, head_dim, dtype, stream);
}

// ---------------------------------------------------------------------------------------
// multi-GPU plumbing
// ---------------------------------------------------------------------------------------
int fmha_ipc_export(const void* ptr, void* handle64, int64_t* offset) {
  if (ptr == nullptr || handle64 == nullptr || offset == nullptr) return FMHA_ERR_NULL_POINTER;
  static_assert(sizeof(cudaIpcMemHandle_t) == 64, "the header promises 64 bytes");
  using RangeFn = CUresult (*)(CUdeviceptr*, size_t*, CUdeviceptr);
  void* fn = nullptr;
  cudaDriverEntryPointQueryResult qres;
  if (cudaGetDriverEntryPoint("cuMemGetAddressRange", &fn, cudaEnableDefault, &qres) != cudaSuccess ||
      qres != cudaDriverEntryPointSuccess)
    return FMHA_ERR_NO_DEVICE;
  CUdeviceptr base = 0;
  size_t size = 0;
  if (reinterpret_cast<RangeFn>(fn)(&base, &size, reinterpret_cast<CUdeviceptr>(ptr)) != CUDA_SUCCESS)
    return FMHA_ERR_BAD_ALIGNMENT;
  cudaIpcMemHandle_t h;
  if (cudaIpcGetMemHandle(&h, reinterpret_cast<void*>(base)) != cudaSuccess) {
    (void)cudaGetLastError();
    return FMHA_ERR_LAUNCH;
  }
  std::memcpy(handle64, &h, sizeof(h));
  *offset = (int64_t)(reinterpret_cast<CUdeviceptr>(ptr) - base);
  return FMHA_OK;
}

int fmha_ipc_open(const void* handle64, int64_t offset, void** ptr) {
  if (handle64 == nullptr || ptr == nullptr) return FMHA_ERR_NULL_POINTER;
  cudaIpcMemHandle_t h;
  std::memcpy(&h, handle64, sizeof(h));
  void* base = nullptr;
  if (cudaIpcOpenMemHandle(&base, h, cudaIpcMemLazyEnablePeerAccess) != cudaSuccess) {
    (void)cudaGetLastError();
    return FMHA_ERR_LAUNCH;
  }
  *ptr = static_cast<char*>(base) + offset;
  return FMHA_OK;
}

int fmha_ipc_close(void* ptr, int64_t offset) {
  if (ptr == nullptr) return FMHA_ERR_NULL_POINTER;
  if (cudaIpcCloseMemHandle(static_cast<char*>(ptr) - offset) != cudaSuccess) {
    (void)cudaGetLastError();
    return FMHA_ERR_LAUNCH;
  }
  return FMHA_OK;
}

int fmha_peer_copy(void* dst, const void* src, size_t bytes, void* stream) {
  if (dst == nullptr || src == nullptr) return FMHA_ERR_NULL_POINTER;
  if (bytes == 0) return FMHA_OK;
  return cudaMemcpyAsync(dst, src, bytes, cudaMemcpyDefault, static_cast<cudaStream_t>(stream)) ==
                 cudaSuccess
             ? FMHA_OK
             : FMHA_ERR_LAUNCH;
}

int fmha_peer_copy_2d(void* dst, size_t dst_pitch, const void* src, size_t src_pitch,
                      size_t row_bytes, size_t rows, void* stream) {
  if (dst == nullptr || src == nullptr) return FMHA_ERR_NULL_POINTER;
  if (row_bytes == 0 || rows == 0) return FMHA_OK;
  if (row_bytes > dst_pitch || row_bytes > src_pitch) return FMHA_ERR_BAD_STRIDE;
  return cudaMemcpy2DAsync(dst, dst_pitch, src, src_pitch, row_bytes, rows, cudaMemcpyDefault,
                           static_cast<cudaStream_t>(stream)) == cudaSuccess
             ? FMHA_OK
             : FMHA_ERR_LAUNCH;
}

int fmha_counter_bump(int32_t* word, void* stream) {
  if (word == nullptr) return FMHA_ERR_NULL_POINTER;
  fmha::counter_bump_kernel<<<1, 1, 0, static_cast<cudaStream_t>(stream)>>>(word);
  return cudaGetLastError() == cudaSuccess ? FMHA_OK : FMHA_ERR_LAUNCH;
}

int fmha_peer_signal(int32_t* const* flags, int32_t n, const int32_t* value, void* stream) {
  if (flags == nullptr || value == nullptr) return FMHA_ERR_NULL_POINTER;
  if (n <= 0) return FMHA_OK;
  if (n > fmha::kMaxPeers) return FMHA_ERR_TOO_LARGE;
  fmha::PeerFlagList list;
  list.n = n;
  for (int i = 0; i < n; ++i) {
    if (flags[i] == nullptr) return FMHA_ERR_NULL_POINTER;
    list.ptr[i] = flags[i];
  }
  fmha::peer_signal_kernel<<<1, 32, 0, static_cast<cudaStream_t>(stream)>>>(list, value);
  return cudaGetLastError() == cudaSuccess ? FMHA_OK : FMHA_ERR_LAUNCH;
}

int fmha_peer_wait(const int32_t* const* flags, int32_t n, const int32_t* value, int32_t* status,
                   int32_t timeout_ms, void* stream) {
  if (flags == nullptr || value == nullptr) return FMHA_ERR_NULL_POINTER;
  if (n <= 0) return FMHA_OK;
  if (n > fmha::kMaxPeers) return FMHA_ERR_TOO_LARGE;
  if (timeout_ms <= 0 || timeout_ms > 60000) return FMHA_ERR_BAD_SHAPE;
  fmha::PeerFlagList list;
  list.n = n;
  for (int i = 0; i < n; ++i) {
    if (flags[i] == nullptr) return FMHA_ERR_NULL_POINTER;
    list.ptr[i] = const_cast<int*>(flags[i]);
  }
  fmha::peer_wait_kernel<<<1, 32, 0, static_cast<cudaStream_t>(stream)>>>(
      list, value, status, (unsigned long long)timeout_ms * 1000000ull);
  return cudaGetLastError() == cudaSuccess ? FMHA_OK : FMHA_ERR_LAUNCH;
}

int fmha_sum_partials(const float* const* parts, const int32_t* rows_per_part, int32_t n_parts,
                      void* out, FmhaStrides out_strides, int32_t batch, int32_t heads, int32_t rows,
                      int32_t head_dim, int32_t dtype, void* stream) {
  if (parts == nullptr || rows_per_part == nullptr || out == nullptr) return FMHA_ERR_NULL_POINTER;
  if (dtype != FMHA_DTYPE_FP16 && dtype != FMHA_DTYPE_BF16) return FMHA_ERR_BAD_DTYPE;
  if (head_dim != 64 && head_dim != 96 && head_dim != 128) return FMHA_ERR_BAD_HEAD_DIM;
  if (batch <= 0 || heads <= 0 || rows <= 0 || n_parts <= 0) return FMHA_ERR_BAD_SHAPE;
  if (n_parts > fmha::kMaxPeers) return FMHA_ERR_TOO_LARGE;
  if (!aligned16(out)) return FMHA_ERR_BAD_ALIGNMENT;
  int rc = check_strides(out_strides, rows, heads, batch);
  if (rc) return rc;
  fmha::PartList list;
  list.n = n_parts;
  for (int i = 0; i < n_parts; ++i) {
    if (parts[i] == nullptr) return FMHA_ERR_NULL_POINTER;
    if (!aligned16(parts[i])) return FMHA_ERR_BAD_ALIGNMENT;
    if (rows_per_part[i] < 0 || rows_per_part[i] > rows) return FMHA_ERR_BAD_SHAPE;
    list.ptr[i] = parts[i];
    list.rows[i] = rows_per_part[i];
  }
  const long long total = (long long)batch * rows * heads;
  const int rows_per_block = 256 / ((head_dim > 64 ? 128 : 64) / 8);  // 16 or 8 threads per row
  const unsigned grid = (unsigned)((total + rows_per_block - 1) / rows_per_block);
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const fmha::Strides3 so = to3(out_strides);
  if (dtype == FMHA_DTYPE_BF16) {
    auto* o = static_cast<__nv_bfloat16*>(out);
    FMHA_DISPATCH_DIMS(head_dim,
                       fmha::sum_partials_kernel<D, __nv_bfloat16, DR><<<grid, 256, 0, s>>>(
                           list, o, so, heads, rows, total);)
  } else {
    auto* o = static_cast<__half*>(out);
    FMHA_DISPATCH_DIMS(head_dim,
                       fmha::sum_partials_kernel<D, __half, DR><<<grid, 256, 0, s>>>(
                           list, o, so, heads, rows, total);)
  }
  return cudaGetLastError() == cudaSuccess ? FMHA_OK : FMHA_ERR_LAUNCH;
}

int fmha_merge_parts(const void* const* o_parts, const float* const* lse_parts,
                     const int32_t* row_offset, const int32_t* rows_per_part, int32_t n_parts,
                     void* o_out, float* lse_out, int32_t batch, int32_t heads, int32_t rows,
                     int32_t head_dim, int32_t dtype, void* stream) {
  if (o_parts == nullptr || lse_parts == nullptr || row_offset == nullptr || rows_per_part == nullptr ||
      o_out == nullptr || lse_out == nullptr)
    return FMHA_ERR_NULL_POINTER;
  if (dtype != FMHA_DTYPE_FP16 && dtype != FMHA_DTYPE_BF16) return FMHA_ERR_BAD_DTYPE;
  if (head_dim != 64 && head_dim != 96 && head_dim != 128) return FMHA_ERR_BAD_HEAD_DIM;
  if (batch <= 0 || heads <= 0 || rows <= 0 || n_parts <= 0) return FMHA_ERR_BAD_SHAPE;
  if (n_parts > fmha::kMaxPeers) return FMHA_ERR_TOO_LARGE;
  if (!aligned16(o_out)) return FMHA_ERR_BAD_ALIGNMENT;
  fmha::MergeList list;
  list.n = n_parts;
  for (int i = 0; i < n_parts; ++i) {
    if (o_parts[i] == nullptr || lse_parts[i] == nullptr) return FMHA_ERR_NULL_POINTER;
    if (!aligned16(o_parts[i])) return FMHA_ERR_BAD_ALIGNMENT;
    if (rows_per_part[i] <= 0 || row_offset[i] < 0 ||
        (long long)row_offset[i] + rows_per_part[i] > (long long)rows)
      return FMHA_ERR_BAD_SHAPE;
    list.o[i] = o_parts[i];
    list.lse[i] = lse_parts[i];
    list.row0[i] = row_offset[i];
    list.rows[i] = rows_per_part[i];
  }
  const long long total = (long long)batch * rows * heads;
  const int rows_per_block = 256 / ((head_dim > 64 ? 128 : 64) / 8);  // 16 or 8 threads per row
  const unsigned grid = (unsigned)((total + rows_per_block - 1) / rows_per_block);
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  if (dtype == FMHA_DTYPE_BF16) {
    auto* o = static_cast<__nv_bfloat16*>(o_out);
    FMHA_DISPATCH_DIMS(head_dim,
                       fmha::merge_parts_kernel<D, __nv_bfloat16, DR><<<grid, 256, 0, s>>>(
                           list, o, lse_out, heads, rows, total);)
  } else {
    auto* o = static_cast<__half*>(o_out);
    FMHA_DISPATCH_DIMS(head_dim,
                       fmha::merge_parts_kernel<D, __half, DR><<<grid, 256, 0, s>>>(
                           list, o, lse_out, heads, rows, total);)
  }
  return cudaGetLastError() == cudaSuccess ? FMHA_OK : FMHA_ERR_LAUNCH;
}

int fmha_b200_forward(const void* query_ptr, const void* key_ptr, const void* value_ptr,
                      void* output_ptr, void* lse_ptr, int batch, int head, int m, int n, int k,
                      float scale, int causal, void* stream) {
  FmhaFwdParams p;
  std::memset(&p, 0, sizeof(p));
  p.q = query_ptr;
  p.k = key_ptr;
  p.v = value_ptr;
  p.o = output_ptr;
  p.lse = static_cast<float*>(lse_ptr);
  p.q_strides = p.o_strides = dense_strides(m, head, k);
  p.k_strides = p.v_strides = dense_strides(n, head, k);
  p.batch = batch;
  p.heads = head;
  p.seqlen_q = m;
  p.seqlen_k = n;
  p.head_dim = k;
  p.scale = scale;
  p.causal = causal;
  return fmha_fwd(&p, stream);
}

int fmha_b200_backward(const void* query_ptr, const void* key_ptr, const void* value_ptr,
                       const void* output_ptr, const void* d_output_ptr, const void* lse_ptr,
                       void* d_query_ptr, void* d_key_ptr, void* d_value_ptr, void* workspace,
                       size_t workspace_bytes, int batch, int head, int m, int n, int k,
                       float scale, int causal, void* stream) {
  FmhaBwdParams p;
  std::memset(&p, 0, sizeof(p));
  p.q = query_ptr;
  p.k = key_ptr;
  p.v = value_ptr;
  p.o = output_ptr;
  p.dout = d_output_ptr;
  p.lse = static_cast<const float*>(lse_ptr);
  p.dq = d_query_ptr;
  p.dk = d_key_ptr;
  p.dv = d_value_ptr;
  p.q_strides = p.o_strides = p.dout_strides = p.dq_strides = dense_strides(m, head, k);
  p.k_strides = p.v_strides = p.dk_strides = p.dv_strides = dense_strides(n, head, k);
  p.batch = batch;
  p.heads = head;
  p.seqlen_q = m;
  p.seqlen_k = n;
  p.head_dim = k;
  p.scale = scale;
  p.causal = causal;
  return fmha_bwd(&p, workspace, workspace_bytes, stream);
}

const char* fmha_status_string(int status) {
  switch (status) {
    case FMHA_OK: return "ok";
    case FMHA_ERR_NULL_POINTER: return "a required pointer is NULL";
    case FMHA_ERR_BAD_HEAD_DIM: return "head_dim must be 64, 96 or 128";
    case FMHA_ERR_BAD_SHAPE: return "sizes must be positive and scale finite and non-zero";
    case FMHA_ERR_BAD_STRIDE: return "strides must be positive multiples of 8 elements";
    case FMHA_ERR_BAD_ALIGNMENT: return "pointers must be 16-byte aligned";
    case FMHA_ERR_WORKSPACE: return "backward workspace missing or too small";
    case FMHA_ERR_TENSOR_MAP: return "cuTensorMapEncodeTiled rejected a tensor";
    case FMHA_ERR_NO_DEVICE: return "CUDA driver entry point unavailable";
    case FMHA_ERR_LAUNCH: return "kernel launch failed";
    case FMHA_ERR_TOO_LARGE: return "a size exceeds the supported maximum";
    case FMHA_ERR_BAD_DTYPE: return "dtype must be FMHA_DTYPE_FP16 or FMHA_DTYPE_BF16";
    default: return "unknown status";
  }
}

const char* fmha_version(void) { return "0.3.0"; }

#ifdef FMHA_TIMELINE
// debug builds only: device buffer (>= 3 * 512 int64) and the CTA whose events are recorded
void fmha_debug_set_timeline(long long* buf, int block) {
  g_timeline = buf;
  g_timeline_block = block;
}
#endif

}  // extern "C"
