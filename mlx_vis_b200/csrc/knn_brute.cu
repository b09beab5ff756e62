// Exact brute-force kNN on B200 — replaces mlx_vis/_knn.py:47-88.
//
// 1. prep:   X (f32) -> two BF16 operands with row pitch ld = round_up(d + 3, 8):
//            A_i = [x~_i, 1, 1, 1, 0...] and B_j = [-2 x~_j, h1, h2, h3, 0...],
//            x~ = bf16(x) and h1 + h2 + h3 = |x~_j|^2 (float32 split into three
//            BF16 parts, relative error ~2^-27).  A_i . B_j is then the score
//            s_ij = |x~_j|^2 - 2 x~_i . x~_j, which orders row i's candidates by
//            distance (|x~_i|^2 is constant along the row).  The three extra K
//            columns live in padding the 64-wide K blocks carry anyway.
// 2. topk:   persistent tcgen05 kernel.  The n x n score matrix is cut into
//            tiles of 256 points (MMA N) by 256 query rows (a CTA pair on one TPC,
//            cluster of 2, tcgen05.mma.cta_group::2 with M = 256) or by 128 rows
//            (pairing switched off: one CTA, M = 128);
//            unit u (pair or CTA) owns the contiguous tile range
//            [u*T/G, (u+1)*T/G) in (row block, column tile) order.  In every CTA
//            warp 0 streams k-blocks with TMA (128-byte swizzle, zero fill past
//            n and d): its own 128 query rows and, in a pair, its half (128) of
//            the tile's points, so each CTA reads (128 + 128) x K per 128 x 256
//            outputs instead of (128 + 256) x K.  Warp 1 of the even CTA issues
//            the MMAs into one of two TMEM accumulators (2 x 256 columns, rows
//            split over the pair's TMEMs), warps 4-7 of each CTA read the
//            finished accumulator (one TMEM lane = one query row per thread) and
//            keep the row's best L scores.  When a unit leaves a row block it
//            writes the lists to cand[row][slot] (slot = which unit of that row
//            block).
// 3. rerank: one warp per row merges its slots, keeps the best L by
//            (score, index), recomputes those L distances exactly in FP32
//            (sum of (x_i - x_j)^2) and writes the k nearest by (distance, index).
// Lists of more than 128 candidates (L = k + extra > 128) go to knn_exact.cu.
#include <cuda_bf16.h>
#include <math.h>
#include <stdlib.h>

#include <mutex>
#include <vector>

#include "common.cuh"
#include "knn_exact.cuh"
#include "tc.cuh"

namespace umapb {
namespace knn {

constexpr int BM = 128;  // query rows per tile = TMEM lanes
constexpr int BN = 256;  // points per tile = MMA N
constexpr int BK = 64;   // BF16 elements per 128-byte swizzled row
constexpr int UK = 16;   // K of one tcgen05.mma kind::f16
constexpr int A_BYTES = BM * BK * 2;
// warp 0 TMA, warp 1 MMA, warp 2 TMEM owner, warp 3 release relay, warps 4-7 epilogue,
// then four warps per further list of 32
constexpr int THREADS = 256;

// Selection of the L best of a row, L <= 32 NL: the row's list is cut into NL sorted
// lists of 32 (score, column) pairs, each in the registers of one thread.  The epilogue
// thread of the row (the leader, list 0) appends hits (scores below the row's L-th best)
// to a private buffer in shared memory and merges it in batches of 16 by
// data-independent sorting networks, so the 32 rows of a warp merge in lockstep without
// divergence.  The 16 pairs that a merge pushes out of a list go through a shared-memory
// mailbox to the follower thread that holds the next 32, which merges them while the
// leader scans on; the last list yields the admission threshold.
// What bounds it: the epilogue warps' instruction latency, one warp per scheduler, for
// small d; the MMAs and their operands from L2 for d in the hundreds.  Sorted registers
// cost about 3 instructions per hit against 15 for reducing unsorted lists by
// bisection.  B200, tile kernel: 9999 x 50, k = 30 (two lists) 7842 -> 186 us (one
// thread inserting into a list in shared memory before); 20000 x 784, k = 100 (four
// lists) 58.6 -> 1.4 ms; 20000 x 784, k = 15 (one list, appends without a branch) 549 ->
// 497 us.
// PAIR: the CTA holds 128 of the tile's 256 points (its half of the pair's B).
template <int NL, bool PAIR>
struct Cfg {
  static_assert(NL >= 1 && NL <= 4, "lists of 32, at most 128 candidates");
  static constexpr int kThreads = THREADS + 128 * (NL - 1);
  static constexpr int kBBytes = (PAIR ? BN / 2 : BN) * BK * 2;
  static constexpr int kStageBytes = A_BYTES + kBBytes;
  static constexpr int kRowsPerBlock = PAIR ? 2 * BM : BM;
  static constexpr int kStages = PAIR ? (NL == 1 ? 5 : NL == 4 ? 3 : 4) : (NL == 1 ? 3 : 2);
  // merge once some row of the warp holds kMergeAt hits; a 32-column group then adds at
  // most 32 to the kMergeAt - 1 already pending
  static constexpr int kMergeAt = 16;
  static constexpr int kBuf = kMergeAt + 32;
  static constexpr int kMailBytes = BM * 16 * 8;  // one mailbox per link: 16 pairs for each row
  static constexpr int kListBytes = BM * kBuf * 8 + (NL - 1) * kMailBytes + BM * 4;  // ... and the thresholds
  static constexpr int kBarBytes = 512;
  static constexpr int kSmem = 1024 + kStages * kStageBytes + kListBytes + kBarBytes;
  static_assert(kSmem <= 227 * 1024, "shared memory of one CTA");
};

struct Plan {
  int64_t n, d, ld;
  int64_t m, r0;  // query rows [r0, r0 + m) against all n rows (m = n, r0 = 0: every row)
  int k, L, lists, num_kb, slots;  // lists: 32-entry lists per row
  bool pair;     // 256-row tiles on CTA pairs (cta_group::2)
  int rb_rows;   // query rows per row block: 256 (pair) or 128
  int64_t row_blocks, col_tiles, tiles, cols_pad;
  int64_t grid;  // work units: CTA pairs (pair) or CTAs
  size_t ws_bytes;
  // workspace layout
  int32_t* status;
  __nv_bfloat16* xa;  // A operand rows [x~, 1, 1, 1]
  __nv_bfloat16* xb;  // B operand rows [-2 x~, h1, h2, h3]
  float* cand_s;
  int32_t* cand_i;
  bool exact;       // k + extra > 128: the long-list path (knn_exact.cu)
  knnx::Plan xp;
};

__host__ __device__ inline int64_t first_cta(int64_t tile, int64_t tiles, int64_t grid) {
  // largest unit c with floor(c * tiles / grid) <= tile
  return ((tile + 1) * grid + tiles - 1) / tiles - 1;
}

// CTA pairs of the cluster launch that fit on the device at once (0: pairs
// unavailable); defined after the kernel.
static int64_t resident_pairs();

// Pairing is on unless the environment sets UMAPB_KNN_PAIR=0 (read per call).
static bool pairing_enabled() {
  const char* e = getenv("UMAPB_KNN_PAIR");
  return !(e && e[0] == '0' && e[1] == 0);
}

static int make_plan(int64_t n, int64_t d, int k, int extra, void* ws, Plan& p, int64_t r0 = 0,
                     int64_t m = -1, bool pair_ok = true) {
  if (m < 0) m = n;
  if (n < 2) return set_error(UMAPB_ERR_ARG, "knn_brute: need n >= 2 (got %lld)", (long long)n);
  if (r0 < 0 || m < 1 || r0 + m > n)
    return set_error(UMAPB_ERR_ARG, "knn_brute: query rows [%lld, %lld) outside [0, %lld)", (long long)r0,
                     (long long)(r0 + m), (long long)n);
  p.m = m;
  p.r0 = r0;
  if (d < 1) return set_error(UMAPB_ERR_ARG, "knn_brute: need d >= 1");
  if (k < 1 || k > n - 1) return set_error(UMAPB_ERR_ARG, "knn_brute: need 1 <= k <= n-1 (k=%d, n=%lld)", k, (long long)n);
  if (extra < 0) return set_error(UMAPB_ERR_ARG, "knn_brute: extra must be >= 0");
  if (n > (int64_t)1 << 30) return set_error(UMAPB_ERR_UNSUPPORTED, "knn_brute: n above 2^30");
  p.n = n;
  p.d = d;
  p.k = k;
  p.L = k + extra;
  if (p.L > n - 1) p.L = (int)(n - 1);
  if (p.L < k) p.L = k;
  p.exact = p.L > 128;
  if (p.exact) {  // exact distances for every pair, no candidate lists
    int s = knnx::plan(n, d, k, p.L, r0, m, ws, p.xp);
    p.ws_bytes = p.xp.bytes;
    p.status = p.xp.status;
    return s;
  }
  p.lists = (p.L + 31) / 32;
  // features + three norm columns, padded to whole 64-element K blocks so every
  // 128-byte TMA box row starts on a 128-byte boundary
  p.ld = (d + 3 + BK - 1) / BK * BK;
  p.num_kb = (int)ceil_div(p.ld, BK);
  int64_t g = 0;
  p.pair = false;
  if (pair_ok && pairing_enabled()) {
    g = resident_pairs();
    p.pair = g > 0;
  }
  if (!p.pair) g = num_sms();
  p.rb_rows = p.pair ? 2 * BM : BM;
  p.row_blocks = ceil_div(m, p.rb_rows);
  p.col_tiles = ceil_div(n, BN);
  p.cols_pad = p.col_tiles * BN;
  p.tiles = p.row_blocks * p.col_tiles;
  p.grid = g < p.tiles ? g : p.tiles;
  int64_t slots = 1;
  for (int64_t rb = 0; rb < p.row_blocks; ++rb) {
    int64_t a = first_cta(rb * p.col_tiles, p.tiles, p.grid);
    int64_t b = first_cta(rb * p.col_tiles + p.col_tiles - 1, p.tiles, p.grid);
    if (b - a + 1 > slots) slots = b - a + 1;
  }
  p.slots = (int)slots;
  Carver c(ws);
  p.status = c.take<int32_t>(64);
  p.xa = c.take<__nv_bfloat16>((size_t)n * p.ld, 1024);
  p.xb = c.take<__nv_bfloat16>((size_t)n * p.ld, 1024);
  p.cand_s = c.take<float>((size_t)m * p.slots * p.L);
  p.cand_i = c.take<int32_t>((size_t)m * p.slots * p.L);
  p.ws_bytes = c.bytes();
  return UMAPB_OK;
}

// ---- 1. prep: augmented BF16 operands (one warp per row) ---------------------
__global__ void prep_kernel(const float* __restrict__ X, int64_t n, int d, int ld, __nv_bfloat16* __restrict__ xa,
                            __nv_bfloat16* __restrict__ xb, int32_t* __restrict__ status) {
  if (blockIdx.x == 0 && threadIdx.x == 0) *status = 0;  // the call's status word, before the tile kernel
  const int64_t row = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (row >= n) return;
  const float* xr = X + row * d;
  __nv_bfloat16* ar = xa + row * ld;
  __nv_bfloat16* br = xb + row * ld;
  float acc = 0.f;
  for (int c = lane; c < d; c += 32) {
    const __nv_bfloat16 h = __float2bfloat16_rn(__ldg(xr + c));
    const float r = __bfloat162float(h);
    ar[c] = h;
    br[c] = __float2bfloat16_rn(-2.0f * r);  // exact: a power-of-two scaling
    acc = fmaf(r, r, acc);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
  // |x~|^2 = h1 + h2 + h3; each remainder is exact in float32
  const __nv_bfloat16 h1 = __float2bfloat16_rn(acc);
  const float r1 = acc - __bfloat162float(h1);
  const __nv_bfloat16 h2 = __float2bfloat16_rn(r1);
  const __nv_bfloat16 h3 = __float2bfloat16_rn(r1 - __bfloat162float(h2));
  const __nv_bfloat16 one = __float2bfloat16_rn(1.0f), zero = __float2bfloat16_rn(0.0f);
  for (int c = d + lane; c < ld; c += 32) {
    const int e = c - d;
    ar[c] = e < 3 ? one : zero;
    br[c] = e == 0 ? h1 : (e == 1 ? h2 : (e == 2 ? h3 : zero));
  }
}

// ---- sorting networks on (score, column) pairs held in registers -------------
__device__ __forceinline__ bool key_lt2(float a, int ia, float b, int ib) {
  return a < b || (a == b && ia < ib);
}

// Compare-exchange on the score alone: which of two equal scores survives at the
// 32nd slot does not change the result, because the exact rerank orders the
// surviving candidates by (distance, index).
__device__ __forceinline__ void cex(float& a, int& ia, float& b, int& ib, bool ascending) {
  const bool sw = ascending ? (b < a) : (a < b);
  const float ta = a, tb = b;
  const int xa = ia, xb = ib;
  a = sw ? tb : ta;
  b = sw ? ta : tb;
  ia = sw ? xb : xa;
  ib = sw ? xa : xb;
}

// ascending bitonic sort of 16 pairs
__device__ __forceinline__ void sort16(float (&v)[16], int (&x)[16]) {
#pragma unroll
  for (int size = 2; size <= 16; size <<= 1) {
#pragma unroll
    for (int stride = size >> 1; stride > 0; stride >>= 1) {
#pragma unroll
      for (int i = 0; i < 16; ++i) {
        const int j = i ^ stride;
        if (j > i) cex(v[i], x[i], v[j], x[j], (i & size) == 0);
      }
    }
  }
}

// ascending order of 16 pairs that form a bitonic sequence
__device__ __forceinline__ void clean16(float (&v)[16], int (&x)[16]) {
#pragma unroll
  for (int stride = 8; stride > 0; stride >>= 1) {
#pragma unroll
    for (int i = 0; i < 16; ++i)
      if ((i & stride) == 0) cex(v[i], x[i], v[i + stride], x[i + stride], true);
  }
}

// list (32, ascending) := smallest 32 of list U batch (16, ascending), ascending; the
// batch becomes the 16 largest, a bitonic sequence.
// [list, +inf x16, reversed batch] is bitonic; its half-cleaner keeps the 32
// smallest in the lower half, which a bitonic merge then sorts.
__device__ __forceinline__ void merge_32_16(float (&lv)[32], int (&li)[32], float (&bv)[16], int (&bx)[16]) {
#pragma unroll
  for (int i = 16; i < 32; ++i) cex(lv[i], li[i], bv[31 - i], bx[31 - i], true);
#pragma unroll
  for (int stride = 16; stride > 0; stride >>= 1) {
#pragma unroll
    for (int i = 0; i < 32; ++i) {
      if ((i & stride) == 0) cex(lv[i], li[i], lv[i + stride], li[i + stride], true);
    }
  }
}

__device__ __forceinline__ void reset_list(float (&lv)[32], int (&li)[32]) {
#pragma unroll
  for (int e = 0; e < 32; ++e) {
    lv[e] = INFINITY;
    li[e] = -1;
  }
}

// the list's entries [0, m) to the candidate arrays
__device__ __forceinline__ void store_list(const float (&lv)[32], const int (&li)[32], int m, float* cs, int32_t* ci) {
#pragma unroll
  for (int e = 0; e < 32; ++e) {
    if (e < m) {
      cs[e] = lv[e];
      ci[e] = li[e];
    }
  }
}

// entry p of the list (p a run-time value below 32)
__device__ __forceinline__ float list_at(const float (&lv)[32], int p) {
  float x = lv[31];
#pragma unroll
  for (int e = 0; e < 31; ++e) x = e == p ? lv[e] : x;
  return x;
}

// (score, column) pairs in shared memory, 8 bytes each
__device__ __forceinline__ void lds_pair(uint32_t at, float& s, int& x) {
  uint32_t u;
  asm volatile("ld.shared.v2.b32 {%0, %1}, [%2];" : "=r"(u), "=r"(x) : "r"(at) : "memory");
  s = __uint_as_float(u);
}
__device__ __forceinline__ void sts_pair(uint32_t at, float s, int x) {
  asm volatile("st.shared.v2.b32 [%0], {%1, %2};" ::"r"(at), "r"(__float_as_uint(s)), "r"(x) : "memory");
}

enum MailCmd : int { kMailMerge = 0, kMailFlush = 1, kMailExit = 2 };

// ---- 2. tcgen05 distance tiles + fused per-row top-L ------------------------
template <int NL, bool PAIR>
__global__ void __launch_bounds__(Cfg<NL, PAIR>::kThreads, 1)
    topk_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
                int n, int num_kb, int64_t col_tiles, int64_t tiles, int slots,
                int L, float* __restrict__ cand_s, int32_t* __restrict__ cand_i, int32_t* __restrict__ status,
                int m_rows, int r0) {
  using C = Cfg<NL, PAIR>;
  constexpr int STAGE_BYTES = C::kStageBytes;
  constexpr int RB = C::kRowsPerBlock;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* stages = smem;
  // pending hits [kBuf][BM] and mailboxes [NL - 1][16][BM], (score, column) pairs; the
  // rows' thresholds [BM]
  float* list_s = reinterpret_cast<float*>(smem + C::kStages * STAGE_BYTES);
  float* mail_s = list_s + 2 * C::kBuf * BM;
  volatile float* tau_s = mail_s + (NL - 1) * (C::kMailBytes / 4);
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + C::kStages * STAGE_BYTES + C::kListBytes);
  uint64_t* full = bars;
  uint64_t* empty = bars + C::kStages;
  uint64_t* tfull = bars + 2 * C::kStages;
  uint64_t* tempty = tfull + 2;
  uint64_t* relay = tempty + 2;  // pair, rank 1: its epilogue's releases, forwarded to rank 0
  uint64_t* mfull = relay + 2;              // [NL - 1][4]: mailbox of link l, lane quarter q, is full ...
  uint64_t* mempty = mfull + 4 * (NL - 1);  // ... has been read
  uint64_t* flushed = mempty + 4 * (NL - 1);  // [4]: the last list of the quarter is reset
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(flushed + 4);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  volatile int* mail_cmd = reinterpret_cast<volatile int*>(tmem_slot + 2);  // [NL - 1][4]
  static_assert((2 * 5 + 2 + 2 + 2 + 8 * 3 + 4) * 8 + (2 + 4 * 3) * 4 <= C::kBarBytes, "barrier area");

  if constexpr (PAIR) {
    uint32_t nrank;
    asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(nrank));
    if (nrank != 2) {  // cta_group::2 needs the cluster launch of two CTAs
      if (threadIdx.x == 0) atomicExch(status, (int32_t)kDevBadLaunch);
      return;
    }
  }
  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  // rank 0 of a pair issues the MMAs and owns the full / tempty barriers the
  // pair shares; rank 1 holds accumulator rows 128-255 of each tile
  const uint32_t rank = PAIR ? tc::cluster_ctarank() : 0u;
  const int64_t G = PAIR ? (int64_t)(gridDim.x >> 1) : (int64_t)gridDim.x;
  const int64_t cta = PAIR ? (int64_t)(blockIdx.x >> 1) : (int64_t)blockIdx.x;  // work unit
  const int64_t t_begin = cta * tiles / G;
  const int64_t t_end = (cta + 1) * tiles / G;

  if (threadIdx.x == 0) {
    for (int s = 0; s < C::kStages; ++s) {
      tc::mbar_init(&full[s], 1);
      tc::mbar_init(&empty[s], 1);
    }
    for (int a = 0; a < 2; ++a) {
      tc::mbar_init(&tfull[a], 1);
      // one arrival per epilogue thread, plus (pair) one forwarded from rank 1
      tc::mbar_init(&tempty[a], PAIR ? 129 : 128);
      tc::mbar_init(&relay[a], 128);
    }
    if constexpr (NL > 1) {
      for (int l = 0; l < 4 * (NL - 1); ++l) {
        tc::mbar_init(&mfull[l], 32);
        tc::mbar_init(&mempty[l], 32);
      }
      for (int l = 0; l < 4; ++l) tc::mbar_init(&flushed[l], 32);
    }
    *abort_flag = 0;
    tc::fence_mbar_init();
  }
  if (NL > 1 && threadIdx.x < BM) tau_s[threadIdx.x] = INFINITY;
  if (warp == 0 && lane == 0) {
    tc::prefetch_tmap(&tmA);
    tc::prefetch_tmap(&tmB);
  }
  if constexpr (PAIR) {
    // both CTAs' barriers are initialised before any remote arrival or TMA
    // completion reaches them; then the pair allocates TMEM together
    __syncthreads();
    tc::cluster_sync();
    if (warp == 2) tc::tmem_alloc_pair(tmem_slot, 512);
  } else {
    if (warp == 2) tc::tmem_alloc(tmem_slot, 512);
  }
  tc::tc_fence_before();
  __syncthreads();
  tc::tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;

  if (warp == 0) {
    // ---------------- TMA producer (both CTAs of a pair) ----------------
    if (lane == 0) {
      int stage = 0;
      uint32_t phase = 0;
      for (int64_t t = t_begin; t < t_end; ++t) {
        const int rb = (int)(t / col_tiles);
        const int ct = (int)(t % col_tiles);
        for (int kb = 0; kb < num_kb; ++kb) {
          if (!tc::mbar_wait(&empty[stage], phase ^ 1, abort_flag)) goto producer_done;
          uint8_t* sa = stages + stage * STAGE_BYTES;
          if constexpr (PAIR) {
            // both halves complete on rank 0's full barrier, which expects the
            // bytes of both
            const uint32_t fb = tc::mapa_shared(tc::smem_u32(&full[stage]), 0);
            if (rank == 0) tc::mbar_arrive_expect_tx(&full[stage], 2 * STAGE_BYTES);
            tc::tma_load_2d_pair(sa, &tmA, fb, kb * BK, rb * RB + (int)rank * BM);
            tc::tma_load_2d_pair(sa + A_BYTES, &tmB, fb, kb * BK, ct * BN + (int)rank * (BN / 2));
          } else {
            tc::mbar_arrive_expect_tx(&full[stage], STAGE_BYTES);
            tc::tma_load_2d(sa, &tmA, &full[stage], kb * BK, rb * BM);
            tc::tma_load_2d(sa + A_BYTES, &tmB, &full[stage], kb * BK, ct * BN);
          }
          if (++stage == C::kStages) {
            stage = 0;
            phase ^= 1;
          }
        }
      }
      if constexpr (PAIR) {
        // every stage released once more: the last MMA commits have arrived on
        // this CTA's empty barriers before it may exit
        for (int i = 0; i < C::kStages; ++i) {
          if (!tc::mbar_wait(&empty[stage], phase ^ 1, abort_flag)) break;
          if (++stage == C::kStages) {
            stage = 0;
            phase ^= 1;
          }
        }
      }
    producer_done:;
    }
  } else if (warp == 1) {
    // ---------------- MMA issuer (rank 0 of a pair) ----------------
    if (lane == 0 && rank == 0) {
      constexpr uint32_t idesc = tc::idesc_bf16_f32(PAIR ? 2 * BM : BM, BN);
      int stage = 0;
      uint32_t phase = 0;
      int acc = 0;
      uint32_t acc_phase = 0;
      bool ok = true;
      for (int64_t t = t_begin; t < t_end; ++t) {
        if (!tc::mbar_wait(&tempty[acc], acc_phase ^ 1, abort_flag)) {
          ok = false;
          break;
        }
        tc::tc_fence_after();
        const uint32_t d_tmem = tmem_base + (uint32_t)(acc * BN);
        for (int kb = 0; kb < num_kb; ++kb) {
          if (!tc::mbar_wait(&full[stage], phase, abort_flag)) {
            ok = false;
            break;
          }
          tc::tc_fence_after();
          const uint32_t a_addr = tc::smem_u32(stages + stage * STAGE_BYTES);
          const uint32_t b_addr = a_addr + A_BYTES;
#pragma unroll
          for (int k = 0; k < BK / UK; ++k) {
            const uint64_t ad = tc::sw128_kmajor_desc(a_addr + k * 32);
            const uint64_t bd = tc::sw128_kmajor_desc(b_addr + k * 32);
            const uint32_t accum = (kb | k) != 0 ? 1u : 0u;
            if constexpr (PAIR)
              tc::mma_bf16_pair(d_tmem, ad, bd, idesc, accum);
            else
              tc::mma_bf16(d_tmem, ad, bd, idesc, accum);
          }
          if constexpr (PAIR)
            tc::mma_commit_pair(&empty[stage], 0x3);
          else
            tc::mma_commit(&empty[stage]);
          if (++stage == C::kStages) {
            stage = 0;
            phase ^= 1;
          }
        }
        if (!ok) break;
        if constexpr (PAIR)
          tc::mma_commit_pair(&tfull[acc], 0x3);
        else
          tc::mma_commit(&tfull[acc]);
        acc ^= 1;
        if (acc == 0) acc_phase ^= 1;
      }
      if (PAIR && ok) {
        // both accumulators released by both CTAs' epilogues: no remote arrival
        // is still on its way to this CTA when it exits
        for (int i = 0; i < 2; ++i) {
          if (!tc::mbar_wait(&tempty[acc], acc_phase ^ 1, abort_flag)) break;
          acc ^= 1;
          if (acc == 0) acc_phase ^= 1;
        }
      }
    }
  } else if (PAIR && warp == 3) {
    // ---------------- release relay (pair, rank 1) ----------------
    // Once rank 1's epilogue has drained an accumulator (128 CTA-scope arrivals
    // on relay[acc], acquired here), one cluster-scope arrival on rank 0's
    // tempty[acc] hands it back to the MMA issuer.
    if (lane == 0 && rank == 1) {
      int acc = 0;
      uint32_t acc_phase = 0;
      for (int64_t t = t_begin; t < t_end; ++t) {
        if (!tc::mbar_wait(&relay[acc], acc_phase, abort_flag)) break;
        tc::mbar_arrive_cluster(tc::mapa_shared(tc::smem_u32(&tempty[acc]), 0));
        acc ^= 1;
        if (acc == 0) acc_phase ^= 1;
      }
    }
  } else if (warp >= 4 && warp < 8) {
    // ---------------- epilogue: batched per-row top-L ----------------
    // Thread r of the four epilogue warps owns TMEM lane r, i.e. query row
    // rb*RB + r (+ 128 in rank 1), and its list 0.  Every hit is appended to its own
    // kBuf-entry buffer in shared memory by predicated stores (no branch).  When a
    // thread of the warp holds kMergeAt hits the whole warp merges in batches of 16.
    const int q = warp & 3;
    const int r = q * 32 + lane;
    const uint32_t my_at = tc::smem_u32(list_s) + 8u * (uint32_t)r;  // [kBuf][BM] (score, column)
    float lv[32];
    int li[32];
    reset_list(lv, li);
    float tau = INFINITY;  // NL == 1: the row's L-th best score
    int cnt = 0;
    int acc = 0;
    uint32_t acc_phase = 0;
    uint32_t sent = 0, flushes = 0;  // messages to the first follower, flushes among them
    int64_t cur_rb = -1;
    bool ok = true;
    // hands the 16 pairs pushed out of list 0 (or a command) to the next list
    auto send = [&](const float (&bv)[16], const int (&bx)[16], int cmd) {
      if constexpr (NL > 1) {
        if (!tc::mbar_wait(&mempty[q], (sent & 1u) ^ 1u, abort_flag)) {
          ok = false;
          return;
        }
        if (cmd == kMailMerge) {
          const uint32_t at = tc::smem_u32(mail_s) + 8u * (uint32_t)r;
#pragma unroll
          for (int e = 0; e < 16; ++e) sts_pair(at + (uint32_t)(e * BM * 8), bv[e], bx[e]);
        }
        if (lane == 0) mail_cmd[q] = cmd;
        tc::mbar_arrive(&mfull[q]);
        ++sent;
      }
    };
    auto merge_batch = [&]() {
      const int m = cnt < 16 ? cnt : 16;
      const int base = cnt - m;
      float bv[16];
      int bx[16];
#pragma unroll
      for (int e = 0; e < 16; ++e) {
        if (e < m) {
          lds_pair(my_at + (uint32_t)((base + e) * BM * 8), bv[e], bx[e]);
        } else {
          bv[e] = INFINITY;
          bx[e] = -1;
        }
      }
      cnt = base;
      sort16(bv, bx);
      merge_32_16(lv, li, bv, bx);
      if constexpr (NL == 1)
        tau = list_at(lv, L - 1);
      else
        send(bv, bx, kMailMerge);
    };
    auto flush = [&](int64_t rb) {
      while (ok && __any_sync(0xffffffffu, cnt > 0)) merge_batch();
      const int64_t row = rb * RB + (int64_t)rank * BM + r;
      const int64_t slot = cta - first_cta(rb * col_tiles, tiles, G);
      const int64_t e0 = (row * slots + slot) * L;
      if (row < m_rows) store_list(lv, li, L < 32 ? L : 32, cand_s + e0, cand_i + e0);
      reset_list(lv, li);
      tau = INFINITY;
      if constexpr (NL > 1) {
        float bv[16];
        int bx[16];
        if (ok) send(bv, bx, kMailFlush);
        // the followers have written their lists and the threshold is infinite again
        if (ok && !tc::mbar_wait(&flushed[q], flushes & 1u, abort_flag)) ok = false;
        ++flushes;
      }
    };
    for (int64_t t = t_begin; t < t_end; ++t) {
      const int64_t rb = t / col_tiles;
      const int ct = (int)(t % col_tiles);
      const bool fresh = rb != cur_rb;  // warp-uniform: the lists are empty
      if (fresh) {
        if (cur_rb >= 0) flush(cur_rb);
        cur_rb = rb;
      }
      if (!ok || !tc::mbar_wait(&tfull[acc], acc_phase, abort_flag)) {
        ok = false;
        break;
      }
      tc::tc_fence_after();
      const int64_t row = rb * RB + (int64_t)rank * BM + r;
      const bool row_ok = row < m_rows;
      const int self_col = row_ok ? (int)(row + r0) : -1;
      const uint32_t taddr = tmem_base + ((uint32_t)(q * 32) << 16) + (uint32_t)(acc * BN);
      // Admission cap of the first tile of a row block, where the empty list
      // would admit every column: per 32-column group the 4 NL-th smallest valid
      // score, maximised over the groups.  At least 4 NL x 8 = 32 NL >= L valid scores
      // are <= that value, so the row's L best of the tile all are, and admitting
      // scores <= cap alone keeps the list exact while cutting the first tile's
      // hits from 256.  A group with fewer than 4 NL valid columns leaves the cap
      // infinite.
      float cap = INFINITY;
      if (fresh) {
        constexpr int D = 4 * NL;
        float hi = -INFINITY;
#pragma unroll 1
        for (int ch = 0; ch < BN / 32; ++ch) {
          float v[32];
          __syncwarp();
          tc::tmem_ld32(taddr + ch * 32, v);
          const int col0 = ct * BN + ch * 32;
          float a[D];  // the D smallest, sorted
#pragma unroll
          for (int d = 0; d < D; ++d) a[d] = INFINITY;
#pragma unroll
          for (int j = 0; j < 32; ++j) {
            const int col = col0 + j;
            const float x = (col != self_col && col < n) ? fminf(v[j], INFINITY) : INFINITY;  // NaN: not valid
#pragma unroll
            for (int d = D - 1; d > 0; --d) a[d] = fminf(a[d], fmaxf(a[d - 1], x));
            a[0] = fminf(a[0], x);
          }
          hi = fmaxf(hi, a[D - 1]);
        }
        // v <= hi  <=>  v < next float above hi (hi finite); infinite hi admits all
        cap = hi < INFINITY ? nextafterf(hi, INFINITY) : INFINITY;
      }
      // columns per step: 16 at 512 threads (128 registers; 672 against 726 us at 20000 x 50,
      // k = 50); at 640 threads (96 registers) 16 spill as 32 do and cost more steps
      constexpr int CW = NL == 3 ? 16 : 32;
      constexpr unsigned kAll = 0xffffffffu >> (32 - CW);
#pragma unroll 1
      for (int ch = 0; ch < BN / CW; ++ch) {
        float v[CW];
        __syncwarp();
        if constexpr (CW == 32)
          tc::tmem_ld32(taddr + ch * CW, v);
        else
          tc::tmem_ld16(taddr + ch * CW, v);
        const int col0 = ct * BN + ch * CW;
        // rows past the last one never admit
        const float lim_s = row_ok ? fminf(NL == 1 ? tau : tau_s[r], cap) : -INFINITY;
        const int self_off = self_col - col0, lim = n - col0;  // the row itself, zero-filled columns past n
        unsigned valid = kAll;
        if ((unsigned)self_off < (unsigned)CW) valid &= ~(1u << self_off);
        if (lim < CW) valid &= lim <= 0 ? 0u : ((1u << lim) - 1u);
        if (__any_sync(0xffffffffu, valid != kAll)) {
#pragma unroll
          for (int j = 0; j < CW; ++j) v[j] = (valid >> j) & 1u ? v[j] : INFINITY;  // never below the threshold
        }
        // a column's slot is computed before any store: a register that a store still
        // reads cannot be advanced, and waiting for that took 25 cycles a column
        uint32_t at = my_at + (uint32_t)(cnt * BM * 8);
        uint32_t slot[CW];
#pragma unroll
        for (int j = 0; j < CW; ++j) {
          slot[j] = at;
          at += v[j] < lim_s ? (uint32_t)(BM * 8) : 0u;
        }
#pragma unroll
        for (int j = 0; j < CW; ++j)
          asm volatile(
              "{\n\t.reg .pred p;\n\t"
              "setp.lt.f32 p, %1, %2;\n\t"
              "@p st.shared.v2.b32 [%0], {%3, %4};\n\t}"
              ::"r"(slot[j]), "f"(v[j]), "f"(lim_s), "r"(__float_as_uint(v[j])), "r"(col0 + j)
              : "memory");
        cnt = (int)(at - my_at) / (BM * 8);
        if (__any_sync(0xffffffffu, cnt >= C::kMergeAt)) {
          do merge_batch();
          while (ok && __any_sync(0xffffffffu, cnt >= C::kMergeAt));
        }
      }
      tc::tc_fence_before();
      // CTA-scope arrivals only: a cluster-scope release costs each epilogue
      // warp over a thousand cycles per tile, so rank 1's warp 3 forwards them
      tc::mbar_arrive(PAIR && rank == 1 ? &relay[acc] : &tempty[acc]);
      acc ^= 1;
      if (acc == 0) acc_phase ^= 1;
    }
    if (ok && cur_rb >= 0) flush(cur_rb);
    if constexpr (NL > 1) {
      float bv[16];
      int bx[16];
      if (ok) send(bv, bx, kMailExit);
    }
  } else if (NL > 1 && warp >= 8) {
    // ---------------- follower: list f of the rows of one lane quarter ----------------
    // Takes batches of 16 pairs from list f - 1, keeps the 32 best of what it has seen
    // and passes the rest on; the last one publishes the rows' L-th best score.
    const int q = warp & 3;
    const int f = (warp >> 2) - 1;  // 1 .. NL - 1
    const int r = q * 32 + lane;
    const bool last = f == NL - 1;
    const int in = 4 * (f - 1) + q, out = 4 * f + q;
    const uint32_t is = tc::smem_u32(mail_s) + (uint32_t)((f - 1) * C::kMailBytes) + 8u * (uint32_t)r;
    const uint32_t os = is + (uint32_t)C::kMailBytes;  // not used by the last one
    const int m = L - 32 * f < 32 ? L - 32 * f : 32;  // entries of this list that count (>= 1)
    float lv[32];
    int li[32];
    reset_list(lv, li);
    uint32_t got = 0;
    int64_t rb = t_begin / col_tiles;  // flushes come once per row block, in order
    while (true) {
      if (!tc::mbar_wait(&mfull[in], got & 1u, abort_flag)) break;
      const int cmd = mail_cmd[in];
      float bv[16];
      int bx[16];
      if (cmd == kMailMerge) {
#pragma unroll
        for (int e = 0; e < 16; ++e) lds_pair(is + (uint32_t)(e * BM * 8), bv[e], bx[e]);
      }
      ++got;
      __syncwarp();
      tc::mbar_arrive(&mempty[in]);
      if (cmd == kMailMerge) {
        clean16(bv, bx);
        merge_32_16(lv, li, bv, bx);
        if (last) tau_s[r] = list_at(lv, m - 1);
      } else if (cmd == kMailFlush) {
        const int64_t row = rb * RB + (int64_t)rank * BM + r;
        const int64_t slot = cta - first_cta(rb * col_tiles, tiles, G);
        const int64_t e0 = (row * slots + slot) * L + 32 * f;
        if (row < m_rows) store_list(lv, li, m, cand_s + e0, cand_i + e0);
        reset_list(lv, li);
        ++rb;
        if (last) {
          tau_s[r] = INFINITY;
          tc::mbar_arrive(&flushed[q]);
        }
      }
      if (!last) {
        if (!tc::mbar_wait(&mempty[out], (got & 1u), abort_flag)) break;
        if (cmd == kMailMerge) {
#pragma unroll
          for (int e = 0; e < 16; ++e) sts_pair(os + (uint32_t)(e * BM * 8), bv[e], bx[e]);
        }
        if (lane == 0) mail_cmd[out] = cmd;
        tc::mbar_arrive(&mfull[out]);
      }
      if (cmd == kMailExit) break;
    }
  }

  tc::tc_fence_before();
  __syncthreads();
  if constexpr (PAIR) {
    // neither CTA frees the pair's TMEM or leaves while the other still works
    tc::cluster_sync();
    if (warp == 2) {
      tc::tc_fence_after();
      tc::tmem_dealloc_pair(tmem_base, 512);
    }
  } else if (warp == 2) {
    tc::tc_fence_after();
    tc::tmem_dealloc(tmem_base, 512);
  }
  if (threadIdx.x == 0 && *abort_flag) atomicExch(status, (int32_t)kDevTimeoutEpilogue);
}

// ---- 3. merge slots + exact FP32 rerank -------------------------------------
__device__ __forceinline__ uint32_t score_key(float s) {  // unsigned order = float order
  const uint32_t u = __float_as_uint(s);
  return u ^ ((u & 0x80000000u) ? 0xffffffffu : 0x80000000u);
}
__device__ __forceinline__ float key_score(uint32_t k) {
  return __uint_as_float(k ^ ((k & 0x80000000u) ? 0x80000000u : 0xffffffffu));
}

constexpr int RR_WARPS = 8;
constexpr int RR_U = 4;  // candidates a lane group has in flight

// One warp per row.  Merging the row's slots is a selection, not a sort: the L-th
// smallest score by bisection (halving the score range, about a dozen steps; the ordered
// bits finish ties), then the exact distances, then each candidate's place by
// counting the smaller ones.  G lanes share one candidate's distance (32 / G * RR_U of
// them in flight), so that short rows keep every lane loading and reduce in log2(G)
// shuffles.  The summation order is the same for every G and VEC: 32 partial sums,
// partial c over the 16-byte words (VEC 4) or the elements (VEC 2, 1) whose number is c
// mod 32, added as a butterfly 16, 8, 4, 2, 1 -- in a lane's registers as far as the
// lane holds both sides.  Bound by the gather of the candidates' rows from L2 for long rows
// (20000 x 784, k = 15: 1.9 GB in 0.20 ms), by the latency of one row's chain for short
// ones: 2000 x 64, k = 15 (8 slots) 40 -> 17 us, 9999 x 50, k = 30 133 -> 50 us against
// sorting all slots in shared memory (and a launch fewer: only lists that were
// written are read, so nothing is cleared first).
template <int VEC, int G>
__global__ void __launch_bounds__(RR_WARPS * 32)
    rerank_kernel(const float* __restrict__ X, int64_t n, int d, const float* __restrict__ cand_s,
                  const int32_t* __restrict__ cand_i, int slots, int rb_rows, int64_t col_tiles, int64_t tiles,
                  int64_t units, int cols, int L, int k, int squared, int32_t* __restrict__ out_idx,
                  float* __restrict__ out_dist, int64_t r0) {
  extern __shared__ uint8_t smem_raw[];
  constexpr unsigned kAll = 0xffffffffu;
  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const unsigned below = (1u << lane) - 1u;
  const int cap = slots * L;
  uint32_t* key = reinterpret_cast<uint32_t*>(smem_raw) + (size_t)warp * 2 * cap;
  int32_t* idx = reinterpret_cast<int32_t*>(key + cap);
  const int64_t row = (int64_t)blockIdx.x * RR_WARPS + warp;
  if (row >= n) return;
  // the units that worked on this row block wrote one list each (entries outside the
  // columns are empty ones, or what a tile kernel that gave up left unwritten)
  const int64_t t0b = (row / rb_rows) * col_tiles;
  const int m = (int)(first_cta(t0b + col_tiles - 1, tiles, units) - first_cta(t0b, tiles, units) + 1) * L;
  int valid = 0;
  uint32_t lo = kAll, hi = 0u;
  for (int e = lane; e < m; e += 32) {
    int j = cand_i[row * cap + e];
    j = (unsigned)j < (unsigned)cols ? j : -1;
    const float s = cand_s[row * cap + e];
    const uint32_t x = j >= 0 ? score_key(s) : kAll;
    key[e] = x;
    idx[e] = j;
    if (j >= 0) {
      ++valid;
      lo = min(lo, x);
      hi = max(hi, x);
    }
  }
  __syncwarp();
  valid = __reduce_add_sync(kAll, valid);
  int c = valid < L ? valid : L;  // candidates to rerank
  if (valid != c || valid < m) {   // compact the c best to the front
    lo = __reduce_min_sync(kAll, lo);
    hi = __reduce_max_sync(kAll, hi);
    int ties = m;  // keys equal to hi that survive
    if (valid > L) {
      bool found = false;
      for (int step = 0; !found && lo < hi; ++step) {
        uint32_t mid = lo + (hi - lo) / 2;
        if (step < 16) {
          const uint32_t h = score_key(0.5f * key_score(lo) + 0.5f * key_score(hi));
          mid = h >= lo && h < hi ? h : mid;
        }
        int cnt = 0;
        for (int e = lane; e < m; e += 32) cnt += key[e] <= mid ? 1 : 0;
        cnt = __reduce_add_sync(kAll, cnt);
        if (cnt >= L) {
          hi = mid;
          found = cnt == L;
        } else {
          lo = mid + 1u;
        }
      }
      if (!found) {
        int less = 0;
        for (int e = lane; e < m; e += 32) less += key[e] < hi ? 1 : 0;
        ties = L - __reduce_add_sync(kAll, less);
      }
    }
    int base = 0, tied = 0;
    for (int e0 = 0; e0 < m; e0 += 32) {  // in place: an entry only moves towards the front
      const int e = e0 + lane;
      const uint32_t x = e < m ? key[e] : kAll;
      const int j = e < m ? idx[e] : -1;
      const bool tie = j >= 0 && x == hi;
      const unsigned tb = __ballot_sync(kAll, tie);
      const bool keep = j >= 0 && (x < hi || (tie && tied + __popc(tb & below) < ties));
      tied += __popc(tb);
      const unsigned kb = __ballot_sync(kAll, keep);
      if (keep) idx[base + __popc(kb & below)] = j;
      base += __popc(kb);
      __syncwarp();
    }
  }

  // exact squared distances of the candidates (direct form, FP32)
  const float* xr = X + (r0 + row) * d;  // rows: the query range [r0, r0 + n)
  constexpr int C = 32 / G;
  constexpr int B = VEC == 2 ? 2 : 1;   // partial sums per loaded word
  constexpr int R = 32 / (G * B);       // words of a lane that belong to different partial sums
  static_assert(R >= 1, "float2 words take at most 16 lanes");
  const int slot = lane / G, t0 = lane & (G - 1);
  const int V = d / VEC;
  for (int e0 = 0; e0 < c; e0 += C * RR_U) {
    const float* xc[RR_U];
    float acc[RR_U][R][B];
#pragma unroll
    for (int u = 0; u < RR_U; ++u) {
      const int e = e0 + u * C + slot;
      xc[u] = X + (int64_t)idx[e < c ? e : c - 1] * d;  // past the end: the last one again
#pragma unroll
      for (int r = 0; r < R; ++r)
#pragma unroll
        for (int v = 0; v < B; ++v) acc[u][r][v] = 0.f;
    }
    for (int tb = t0; tb < V; tb += G * R) {
#pragma unroll
      for (int r = 0; r < R; ++r) {
        const int t = tb + G * r;
        if (t >= V) continue;
        float a[VEC], b[RR_U][VEC];
        if constexpr (VEC == 4) {
          const float4 q = __ldg(reinterpret_cast<const float4*>(xr) + t);
          a[0] = q.x, a[1] = q.y, a[2] = q.z, a[3] = q.w;
#pragma unroll
          for (int u = 0; u < RR_U; ++u) {
            const float4 y = __ldg(reinterpret_cast<const float4*>(xc[u]) + t);
            b[u][0] = y.x, b[u][1] = y.y, b[u][2] = y.z, b[u][3] = y.w;
          }
        } else if constexpr (VEC == 2) {
          const float2 q = __ldg(reinterpret_cast<const float2*>(xr) + t);
          a[0] = q.x, a[1] = q.y;
#pragma unroll
          for (int u = 0; u < RR_U; ++u) {
            const float2 y = __ldg(reinterpret_cast<const float2*>(xc[u]) + t);
            b[u][0] = y.x, b[u][1] = y.y;
          }
        } else {
          a[0] = __ldg(xr + t);
#pragma unroll
          for (int u = 0; u < RR_U; ++u) b[u][0] = __ldg(xc[u] + t);
        }
#pragma unroll
        for (int u = 0; u < RR_U; ++u)
#pragma unroll
          for (int v = 0; v < VEC; ++v) {
            const float diff = a[v] - b[u][v];
            float& s = acc[u][r][VEC == 2 ? v : 0];
            s = fmaf(diff, diff, s);
          }
      }
    }
    float sum[RR_U];
#pragma unroll
    for (int u = 0; u < RR_U; ++u) {
      float p[B];
#pragma unroll
      for (int v = 0; v < B; ++v) {  // the widest steps of the butterfly, within the lane
        if constexpr (R == 4)
          p[v] = (acc[u][0][v] + acc[u][2][v]) + (acc[u][1][v] + acc[u][3][v]);
        else if constexpr (R == 2)
          p[v] = acc[u][0][v] + acc[u][1][v];
        else
          p[v] = acc[u][0][v];
#pragma unroll
        for (int o = G >> 1; o > 0; o >>= 1) p[v] += __shfl_xor_sync(kAll, p[v], o);
      }
      sum[u] = B == 2 ? p[0] + p[B - 1] : p[0];
    }
#pragma unroll
    for (int u = 0; u < RR_U; ++u) {
      const int e = e0 + u * C + slot;
      if (t0 == 0 && e < c) key[e] = __float_as_uint(sum[u]);  // not negative: the bits order like the value
    }
  }
  __syncwarp();

  // places by (distance, index)
  constexpr int NE = 4;  // L <= 128
  uint32_t mk[NE];
  int32_t mi[NE];
  int rank[NE];
#pragma unroll
  for (int u = 0; u < NE; ++u) {
    const int e = u * 32 + lane;
    mk[u] = e < c ? key[e] : kAll;
    mi[u] = e < c ? idx[e] : 0x7fffffff;
    rank[u] = 0;
  }
  const int chunks = (c + 31) / 32;
#pragma unroll 4
  for (int t = 0; t < c; ++t) {
    const uint32_t kt = key[t];
    const int32_t it = idx[t];
#pragma unroll
    for (int u = 0; u < NE; ++u)
      if (u < chunks) rank[u] += kt < mk[u] || (kt == mk[u] && it < mi[u]) ? 1 : 0;
  }
#pragma unroll
  for (int u = 0; u < NE; ++u) {
    if (u * 32 + lane < c && rank[u] < k) {
      const float v = __uint_as_float(mk[u]);
      out_idx[row * k + rank[u]] = mi[u];
      out_dist[row * k + rank[u]] = squared ? v : sqrtf(v);
    }
  }
  for (int e = c + lane; e < k; e += 32) {  // fewer candidates than k: scores that overflowed
    out_idx[row * k + e] = 0x7fffffff;
    out_dist[row * k + e] = INFINITY;
  }
}

template <int NL, bool PAIR>
static int set_smem_attr() {
  using C = Cfg<NL, PAIR>;
  static bool attr_set[64] = {false};
  int dev = 0;
  UMAPB_CUDA_TRY(cudaGetDevice(&dev), "knn_brute: cudaGetDevice");
  if (dev < 0 || dev >= 64) return set_error(UMAPB_ERR_UNSUPPORTED, "knn_brute: device index %d", dev);
  if (!attr_set[dev]) {
    UMAPB_CUDA_TRY(cudaFuncSetAttribute(topk_kernel<NL, PAIR>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                        C::kSmem),
                   "knn_brute: set smem attribute");
    attr_set[dev] = true;
  }
  return UMAPB_OK;
}

static decltype(&rerank_kernel<4, 8>) const kRerank[8] = {
    rerank_kernel<4, 8>,  rerank_kernel<4, 16>, rerank_kernel<4, 32>, rerank_kernel<2, 8>,
    rerank_kernel<2, 16>, rerank_kernel<1, 8>,  rerank_kernel<1, 16>, rerank_kernel<1, 32>};

// Enqueues the rerank of rows [r0, r0 + m).  Its dynamic shared memory (2 slots * L
// words per warp) can exceed the 48 KB default; the attribute is raised once per device
// (up to 200 KB).
static size_t rerank_smem(const Plan& p) { return (size_t)RR_WARPS * 2 * p.slots * p.L * sizeof(float); }

static int rerank_smem_attr(size_t smem) {
  if (smem <= 48 * 1024) return UMAPB_OK;
  if (smem > 200 * 1024)
    return set_error(UMAPB_ERR_UNSUPPORTED, "knn_brute: candidate merge needs %zu bytes of shared memory", smem);
  static std::mutex mu;
  static bool done[64] = {false};
  int dev = 0;
  UMAPB_CUDA_TRY(cudaGetDevice(&dev), "knn_brute: cudaGetDevice");
  if (dev < 0 || dev >= 64) return set_error(UMAPB_ERR_UNSUPPORTED, "knn_brute: device index %d", dev);
  std::lock_guard<std::mutex> lock(mu);
  if (!done[dev]) {
    for (int v = 0; v < 8; ++v)
      UMAPB_CUDA_TRY(cudaFuncSetAttribute((const void*)kRerank[v], cudaFuncAttributeMaxDynamicSharedMemorySize,
                                          (int)(200 * 1024)),
                     "knn_brute: rerank smem attribute");
    done[dev] = true;
  }
  return UMAPB_OK;
}

static int run_rerank(const Plan& p, const float* X, int squared, int32_t* out_idx, float* out_dist,
                      cudaStream_t stream) {
  const size_t smem = rerank_smem(p);
  const unsigned blocks = (unsigned)ceil_div(p.m, RR_WARPS);
  const uintptr_t at = reinterpret_cast<uintptr_t>(X);
  const int vec = (p.d & 3) == 0 && (at & 15) == 0 ? 4 : (p.d & 1) == 0 && (at & 7) == 0 ? 2 : 1;
  // lanes per candidate: the least that cover a row in a few loads each, so that short
  // rows have more candidates in flight
  const int64_t loads = p.d / vec;
  const int by8 = loads <= 32 ? 0 : 1;
  const int by32 = by8 ? (loads <= 96 ? 1 : 2) : 0;
  const auto kernel = kRerank[vec == 4 ? by32 : vec == 2 ? 3 + by8 : 5 + by32];
  kernel<<<blocks, RR_WARPS * 32, smem, stream>>>(X, p.m, (int)p.d, p.cand_s, p.cand_i, p.slots, p.rb_rows,
                                                  p.col_tiles, p.tiles, p.grid, (int)p.n, p.L, p.k, squared, out_idx,
                                                  out_dist, p.r0);
  UMAPB_LAUNCH_CHECK("knn_brute: rerank kernel launch");
  return UMAPB_OK;
}

static int64_t resident_pairs() {
  static std::mutex mu;
  static int64_t cached[64];
  static bool known[64] = {false};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 0;
  std::lock_guard<std::mutex> lock(mu);
  if (!known[dev]) {
    int64_t pairs = 0;
    if (set_smem_attr<1, true>() == UMAPB_OK) {  // every list count runs one CTA per SM
      cudaLaunchConfig_t cfg = {};
      cudaLaunchAttribute attr[1];
      attr[0].id = cudaLaunchAttributeClusterDimension;
      attr[0].val.clusterDim.x = 2;
      attr[0].val.clusterDim.y = 1;
      attr[0].val.clusterDim.z = 1;
      cfg.gridDim = dim3(2 * (unsigned)num_sms(), 1, 1);
      cfg.blockDim = dim3(THREADS, 1, 1);
      cfg.dynamicSmemBytes = Cfg<1, true>::kSmem;
      cfg.attrs = attr;
      cfg.numAttrs = 1;
      int clusters = 0;
      if (cudaOccupancyMaxActiveClusters(&clusters, topk_kernel<1, true>, &cfg) == cudaSuccess) pairs = clusters;
    }
    cudaGetLastError();  // a refused query only disables pairing
    clear_error();
    cached[dev] = pairs;
    known[dev] = true;
  }
  return cached[dev];
}

template <int NL>
static int launch_topk(const Plan& p, const CUtensorMap& ta, const CUtensorMap& tb, cudaStream_t stream) {
  int s = p.pair ? set_smem_attr<NL, true>() : set_smem_attr<NL, false>();
  if (s) return s;
  if (!p.pair) {
    topk_kernel<NL, false><<<(unsigned)p.grid, Cfg<NL, false>::kThreads, Cfg<NL, false>::kSmem, stream>>>(
        ta, tb, (int)p.n, p.num_kb, p.col_tiles, p.tiles, p.slots, p.L, p.cand_s, p.cand_i, p.status, (int)p.m,
        (int)p.r0);
    UMAPB_LAUNCH_CHECK("knn_brute: topk kernel launch");
    return UMAPB_OK;
  }
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 2;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.gridDim = dim3(2 * (unsigned)p.grid, 1, 1);
  cfg.blockDim = dim3(Cfg<NL, true>::kThreads, 1, 1);
  cfg.dynamicSmemBytes = Cfg<NL, true>::kSmem;
  cfg.stream = stream;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  UMAPB_CUDA_TRY(cudaLaunchKernelEx(&cfg, topk_kernel<NL, true>, ta, tb, (int)p.n, p.num_kb, p.col_tiles, p.tiles,
                                    p.slots, p.L, p.cand_s, p.cand_i, p.status, (int)p.m, (int)p.r0),
                 "knn_brute: pair topk kernel launch");
  return UMAPB_OK;
}

// Tensor maps of both operands (B box: the CTA's share of a 256-point tile) and
// the tile kernel the plan chose.
static int run_tiles(const Plan& p, cudaStream_t stream) {
  CUtensorMap ta, tb;
  int s;
  if ((s = make_tmap_bf16_2d(&ta, p.xa + p.r0 * p.ld, (uint64_t)p.m, (uint64_t)p.ld, (uint64_t)p.ld, BM, BK)))
    return s;
  if ((s = make_tmap_bf16_2d(&tb, p.xb, (uint64_t)p.n, (uint64_t)p.ld, (uint64_t)p.ld, p.pair ? BN / 2 : BN, BK)))
    return s;
  switch (p.lists) {
    case 1: return launch_topk<1>(p, ta, tb, stream);
    case 2: return launch_topk<2>(p, ta, tb, stream);
    case 3: return launch_topk<3>(p, ta, tb, stream);
    default: return launch_topk<4>(p, ta, tb, stream);
  }
}

}  // namespace knn
}  // namespace umapb

using namespace umapb;

extern "C" int umapb_knn_brute_workspace(int64_t n, int64_t d, int32_t k, int32_t extra, size_t* bytes) {
  clear_error();
  if (!bytes) return set_error(UMAPB_ERR_ARG, "bytes is null");
  knn::Plan p;
  int s = knn::make_plan(n, d, k, extra, nullptr, p);
  if (s) return s;
  *bytes = p.ws_bytes;
  return UMAPB_OK;
}

// The three stages of one call; with `ev` (4 events) each stage boundary is recorded.
static int enqueue_knn(const float* X, int64_t n, int64_t d, int32_t k, int32_t squared, int32_t* out_idx,
                       float* out_dist, const knn::Plan& p, cudaStream_t stream, cudaEvent_t* ev) {
  if (p.exact) {
    if (ev) return set_error(UMAPB_ERR_UNSUPPORTED, "knn_brute_timed: k + extra must be <= 128");
    return knnx::run(X, p.xp, squared, out_idx, out_dist, stream);
  }
  int s;
  if ((s = knn::rerank_smem_attr(knn::rerank_smem(p)))) return s;
  if (ev) UMAPB_CUDA_TRY(cudaEventRecord(ev[0], stream), "knn_brute: event");
  {
    const int64_t warps = n;
    const unsigned blocks = (unsigned)ceil_div(warps * 32, 256);
    knn::prep_kernel<<<blocks, 256, 0, stream>>>(X, n, (int)d, (int)p.ld, p.xa, p.xb, p.status);
    UMAPB_LAUNCH_CHECK("knn_brute: prep kernel launch");
  }
  if (ev) UMAPB_CUDA_TRY(cudaEventRecord(ev[1], stream), "knn_brute: event");
  if ((s = knn::run_tiles(p, stream))) return s;
  if (ev) UMAPB_CUDA_TRY(cudaEventRecord(ev[2], stream), "knn_brute: event");
  if ((s = knn::run_rerank(p, X, squared, out_idx, out_dist, stream))) return s;
  if (ev) UMAPB_CUDA_TRY(cudaEventRecord(ev[3], stream), "knn_brute: event");
  count_launches(3);
  return UMAPB_OK;
}

extern "C" int umapb_knn_brute(const float* X, int64_t n, int64_t d, int32_t k, int32_t extra, int32_t squared,
                               int32_t* out_idx, float* out_dist, void* workspace, size_t workspace_bytes,
                               umapb_stream_t stream_) {
  clear_error();
  cudaStream_t stream = reinterpret_cast<cudaStream_t>(stream_);
  UMAPB_REQUIRE(X && out_idx && out_dist, "knn_brute: null array argument");
  knn::Plan p;
  int s = knn::make_plan(n, d, k, extra, nullptr, p);
  if (s) return s;
  if (!workspace || workspace_bytes < p.ws_bytes)
    return set_error(UMAPB_ERR_WORKSPACE, "knn_brute: workspace of %zu bytes, need %zu", workspace_bytes, p.ws_bytes);
  knn::make_plan(n, d, k, extra, workspace, p);
  return enqueue_knn(X, n, d, k, squared, out_idx, out_dist, p, stream, nullptr);
}

extern "C" int umapb_knn_brute_rows_workspace(int64_t n, int64_t d, int32_t k, int32_t extra, int64_t row_begin,
                                              int64_t row_count, size_t* bytes) {
  clear_error();
  if (!bytes) return set_error(UMAPB_ERR_ARG, "bytes is null");
  knn::Plan p;
  int s = knn::make_plan(n, d, k, extra, nullptr, p, row_begin, row_count);
  if (s) return s;
  *bytes = p.ws_bytes;
  return UMAPB_OK;
}

extern "C" int umapb_knn_brute_rows(const float* X, int64_t n, int64_t d, int32_t k, int32_t extra, int32_t squared,
                                    int64_t row_begin, int64_t row_count, int32_t* out_idx, float* out_dist,
                                    void* workspace, size_t workspace_bytes, umapb_stream_t stream_) {
  clear_error();
  cudaStream_t stream = reinterpret_cast<cudaStream_t>(stream_);
  UMAPB_REQUIRE(X && out_idx && out_dist, "knn_brute_rows: null array argument");
  knn::Plan p;
  int s = knn::make_plan(n, d, k, extra, nullptr, p, row_begin, row_count);
  if (s) return s;
  if (!workspace || workspace_bytes < p.ws_bytes)
    return set_error(UMAPB_ERR_WORKSPACE, "knn_brute_rows: workspace of %zu bytes, need %zu", workspace_bytes,
                     p.ws_bytes);
  knn::make_plan(n, d, k, extra, workspace, p, row_begin, row_count);
  return enqueue_knn(X, n, d, k, squared, out_idx, out_dist, p, stream, nullptr);
}

extern "C" int umapb_knn_brute_timed(const float* X, int64_t n, int64_t d, int32_t k, int32_t extra, int32_t squared,
                                     int32_t* out_idx, float* out_dist, void* workspace, size_t workspace_bytes,
                                     float* stage_ms, umapb_stream_t stream_) {
  clear_error();
  cudaStream_t stream = reinterpret_cast<cudaStream_t>(stream_);
  UMAPB_REQUIRE(X && out_idx && out_dist && stage_ms, "knn_brute_timed: null argument");
  knn::Plan p;
  int s = knn::make_plan(n, d, k, extra, nullptr, p);
  if (s) return s;
  if (!workspace || workspace_bytes < p.ws_bytes)
    return set_error(UMAPB_ERR_WORKSPACE, "knn_brute: workspace of %zu bytes, need %zu", workspace_bytes, p.ws_bytes);
  knn::make_plan(n, d, k, extra, workspace, p);
  cudaEvent_t ev[4] = {};
  for (int i = 0; i < 4; ++i) UMAPB_CUDA_TRY(cudaEventCreate(&ev[i]), "knn_brute_timed: event create");
  s = enqueue_knn(X, n, d, k, squared, out_idx, out_dist, p, stream, ev);
  if (s == UMAPB_OK) {
    cudaError_t e = cudaEventSynchronize(ev[3]);
    for (int i = 0; i < 3 && e == cudaSuccess; ++i) e = cudaEventElapsedTime(&stage_ms[i], ev[i], ev[i + 1]);
    if (e != cudaSuccess) s = set_error(UMAPB_ERR_CUDA, "knn_brute_timed: %s", cudaGetErrorString(e));
  }
  for (int i = 0; i < 4; ++i) cudaEventDestroy(ev[i]);
  return s;
}

// ---------------------------------------------------------------------------
// Allocation-free variant of umapb_knn_brute.
//
// Some callers cannot hand this library a device workspace: cudaMalloc and
// cudaFree synchronise the whole device (a stall that latency-bound callers
// cannot take), they fail outright when another framework's pooled allocator
// already owns the device memory, and thin FFI bindings often have no way to
// keep a device buffer alive between calls.  This entry point therefore uses a
// fixed scratch array that lives in the library itself: a file-scope
// __device__ array of UMAPB_NOALLOC_SCRATCH_BYTES, which every GPU that loads
// the library holds until the process exits.  Requests whose workspace would
// exceed it are rejected.  The first call on each device looks up that
// device's address of the array with cudaGetSymbolAddress (with the device
// current); make that first call before any stream capture begins.  All calls
// share the one array and it keeps the previous call's contents, so the parts
// that must start at a known value (the status word) are reset
// by each call, and calls whose work overlaps on the GPU (for example on two
// streams at once) race on it: serialise them.
// ---------------------------------------------------------------------------
namespace {

static __device__ __align__(256) unsigned char g_knn_scratch[UMAPB_NOALLOC_SCRATCH_BYTES];

std::mutex g_scratch_mu;
void* g_scratch_addr[64] = {nullptr};

int scratch_address(void** out) {
  int dev = 0;
  UMAPB_CUDA_TRY(cudaGetDevice(&dev), "knn_brute_noalloc: cudaGetDevice");
  if (dev < 0 || dev >= 64) return set_error(UMAPB_ERR_UNSUPPORTED, "knn_brute_noalloc: device index %d", dev);
  std::lock_guard<std::mutex> lock(g_scratch_mu);
  if (!g_scratch_addr[dev]) {
    void* p = nullptr;
    const cudaError_t e = cudaGetSymbolAddress(&p, g_knn_scratch);
    if (e != cudaSuccess)
      return set_error(UMAPB_ERR_CUDA, "knn_brute_noalloc: cudaGetSymbolAddress: %s", cudaGetErrorString(e));
    g_scratch_addr[dev] = p;
  }
  *out = g_scratch_addr[dev];
  return UMAPB_OK;
}

}  // namespace

extern "C" int umapb_knn_brute_noalloc(const float* X, int64_t n, int64_t d, int32_t k, int32_t extra,
                                       int32_t squared, int32_t* out_idx, float* out_dist, int32_t* device_status,
                                       umapb_stream_t stream_) {
  clear_error();
  cudaStream_t stream = reinterpret_cast<cudaStream_t>(stream_);
  UMAPB_REQUIRE(X && out_idx && out_dist, "knn_brute_noalloc: null array argument");
  knn::Plan p;
  int s = knn::make_plan(n, d, k, extra, nullptr, p);
  if (s) return s;
  // a few shapes need one slot per row more on CTA pairs than on single CTAs
  bool pair_ok = true;
  if (p.ws_bytes > (size_t)UMAPB_NOALLOC_SCRATCH_BYTES && !p.exact && p.pair) {
    pair_ok = false;
    if ((s = knn::make_plan(n, d, k, extra, nullptr, p, 0, -1, pair_ok))) return s;
  }
  if (p.ws_bytes > (size_t)UMAPB_NOALLOC_SCRATCH_BYTES)
    return set_error(UMAPB_ERR_UNSUPPORTED,
                     "knn_brute_noalloc: n=%lld, d=%lld, k+extra=%d needs %zu bytes of scratch but the static array "
                     "holds %zu; use umapb_knn_brute with a caller-owned workspace",
                     (long long)n, (long long)d, p.L, p.ws_bytes, (size_t)UMAPB_NOALLOC_SCRATCH_BYTES);
  void* scratch = nullptr;
  if ((s = scratch_address(&scratch))) return s;
  knn::make_plan(n, d, k, extra, scratch, p, 0, -1, pair_ok);
  if (p.exact) {
    if ((s = knnx::run(X, p.xp, squared, out_idx, out_dist, stream))) return s;
    if (device_status)
      UMAPB_CUDA_TRY(cudaMemcpyAsync(device_status, p.status, sizeof(int32_t), cudaMemcpyDeviceToDevice, stream),
                     "knn_brute_noalloc: status copy");
    return UMAPB_OK;
  }

  if ((s = knn::rerank_smem_attr(knn::rerank_smem(p)))) return s;  // before any launch: a refusal leaves nothing enqueued

  knn::prep_kernel<<<(unsigned)ceil_div(n * 32, 256), 256, 0, stream>>>(X, n, (int)d, (int)p.ld, p.xa, p.xb, p.status);
  UMAPB_LAUNCH_CHECK("knn_brute_noalloc: prep kernel launch");
  if ((s = knn::run_tiles(p, stream))) return s;
  if ((s = knn::run_rerank(p, X, squared, out_idx, out_dist, stream))) return s;
  if (device_status)
    UMAPB_CUDA_TRY(cudaMemcpyAsync(device_status, p.status, sizeof(int32_t), cudaMemcpyDeviceToDevice, stream),
                   "knn_brute_noalloc: status copy");
  count_launches(3);
  return UMAPB_OK;
}
