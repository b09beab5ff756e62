// BF16 tensor-core GEMM with fused MLP epilogues, for the learned warm-start
// encoder (no counterpart in the reference; its nearest idiom is the MMAE MLP,
// mlx_vis/_mmae/mmae.py:22-38, 258-281).
//
//   C[M, N] = sum_k A[m, k] B[n, k]      A (M x K), B (N x K): BF16, K-major
//
// Either operand may instead be stored with K as its row index (K x M or K x N, "MN-major"
// for the tensor core, a bit of the instruction descriptor): weight gradients dZ^T X
// read their batches as they were written, without transposed copies.
//
// One CTA per 128 x BN output tile and K slice (gridDim.z slices of the K
// blocks; the F32 epilogue then writes each slice's partial tile to its own
// M x ldc block of C, for the consumer to sum): warp 0
// streams 64-wide K blocks of A and B with TMA (128-byte swizzle, zero fill past
// M, N, K) through 3 stages, one thread of warp 1 issues tcgen05.mma (M=128, N=BN,
// K=16, FP32 accumulation in TMEM), warps 2-5 (one per TMEM lane quarter) read the
// accumulator with tcgen05.ld, 64 columns at a time, and apply the epilogue:
//   EPI_F32        C (f32, row-major, pitch ldc); with K slices, slice z at C + z M ldc
//   EPI_BIAS_GELU  z = C + bias[n]; Z (f32), H = bf16(gelu(z)) row-major and,
//                  when HT != null, its transpose H^T (N x M, pitch ldt)
//   EPI_GELU_BACK  g = C; dZ = g * gelu'(Z) -> bf16 row-major, optional transpose,
//                  optional column sums of the bf16 values in colsum
//   EPI_BIAS_GELU_H  H alone (inference)
// The accumulator rows sit one per thread; each 32 x 64 chunk passes through
// shared memory (the drained operand stages) so outputs are written a row per warp
// instruction, two columns per lane.
// What bounds it: K is short (8 to 13 blocks), so a tile is one pipeline fill and one
// epilogue; several CTAs share an SM (two of BN = 128, three of BN = 64, which is taken
// when 128-wide tiles would leave SMs idle) and fill each other's gaps.  B200, forward
// layer of a 4096-row batch, 784 -> 512: 23 -> 13 us; 16384 rows, inference: 68 -> 32 us
// (one CTA per SM, one column per lane and a branch per row before).
// gelu(z) = z * Phi(z); gelu'(z) = Phi(z) + z phi(z) (gelu.cuh).
// Every mbarrier wait is bounded (2 s) and reports through *status.
#include <cuda_bf16.h>
#include <math.h>

#include "common.cuh"
#include "gelu.cuh"
#include "tc.cuh"

namespace umapb {
namespace gemm {

constexpr int BM = 128, BN = 128, BK = 64, UK = 16;
constexpr int A_BYTES = BM * BK * 2;
constexpr int THREADS = 192;  // warp 0 TMA, warp 1 MMA, warps 2-5 epilogue (lane quarters 2, 3, 0, 1)
constexpr int STAGES = 3;
constexpr int S_PITCH = 66;   // floats per staged epilogue row (64 columns + padding)

template <int TBN>
struct Tile {
  static constexpr int kStageBytes = A_BYTES + TBN * BK * 2;
  static constexpr int kSmem = 1024 + STAGES * kStageBytes + 256;
  static constexpr int kPerSm = TBN == 64 ? 3 : 2;
  static_assert(kPerSm * (kSmem + 1024) <= 227 * 1024 + 1024, "resident CTAs");
  static_assert(4 * 32 * S_PITCH * 4 <= STAGES * kStageBytes, "epilogue staging");
};

enum Epi : int { EPI_F32 = 0, EPI_BIAS_GELU = 1, EPI_GELU_BACK = 2, EPI_BIAS_GELU_H = 3 };

struct EpiArgs {
  int M, N;
  float* C;  // EPI_F32 output
  int ldc;
  const float* bias;      // EPI_BIAS_GELU
  float* Z;               // EPI_BIAS_GELU output / EPI_GELU_BACK input (pre-activation), pitch ldz
  int ldz;
  __nv_bfloat16* H;       // bf16 output (row-major, pitch ldh)
  int ldh;
  __nv_bfloat16* HT;      // optional bf16 transposed output (N x M, pitch ldt)
  int ldt;
  float* colsum;          // EPI_GELU_BACK: optional column sums of H (atomic adds)
  int64_t slice;          // EPI_F32 with K slices: slice z is written at C + z * slice
};


// Shared-memory descriptor of an operand tile whose rows are K (64 MN values, 128 bytes,
// 128-byte swizzle): blocks of 64 MN values 8 KB apart, groups of 8 K rows 1 KB apart.
__device__ __forceinline__ uint64_t sw128_mnmajor_desc(uint32_t smem_addr) {
  uint64_t d = 0;
  d |= static_cast<uint64_t>((smem_addr >> 4) & 0x3FFF);      // start address
  d |= static_cast<uint64_t>((64 * BK * 2) >> 4) << 16;       // leading byte offset: next 64 MN values
  d |= static_cast<uint64_t>(1024 >> 4) << 32;                // stride byte offset: next 8 K rows
  d |= static_cast<uint64_t>(1) << 46;                        // descriptor version (sm_100)
  d |= static_cast<uint64_t>(2) << 61;                        // layout: SWIZZLE_128B
  return d;
}

// two adjacent outputs of one row; `pair` when the address allows one store
__device__ __forceinline__ void store2(float* p, float x, float y, bool pair, bool second) {
  if (pair) {
    *reinterpret_cast<float2*>(p) = make_float2(x, y);
  } else {
    p[0] = x;
    if (second) p[1] = y;
  }
}
__device__ __forceinline__ void store2(__nv_bfloat16* p, __nv_bfloat16 x, __nv_bfloat16 y, bool pair, bool second) {
  if (pair) {
    *reinterpret_cast<__nv_bfloat162*>(p) = __halves2bfloat162(x, y);
  } else {
    p[0] = x;
    if (second) p[1] = y;
  }
}

// TA, TB: the operand is stored with K as its row index
template <int EPI, bool TA, bool TB, int TBN>
__global__ void __launch_bounds__(THREADS, Tile<TBN>::kPerSm)
    gemm_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB, int num_kb,
                EpiArgs e, int32_t* __restrict__ status) {
  constexpr int STAGE_BYTES = Tile<TBN>::kStageBytes;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + STAGES * STAGE_BYTES);
  uint64_t* full = bars;
  uint64_t* empty = bars + STAGES;
  uint64_t* done = bars + 2 * STAGES;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(done + 1);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // blockIdx.x walks the N tiles of an M tile first, so CTAs launched together share an A
  // tile in L2
  const int n_tiles = (e.N + TBN - 1) / TBN;
  const int n0 = (blockIdx.x % n_tiles) * TBN, m0 = (blockIdx.x / n_tiles) * BM;
  // this CTA's K blocks [kb0, kb1); the host sizes the slices so none is empty
  const int per = (num_kb + gridDim.z - 1) / gridDim.z;
  const int kb0 = blockIdx.z * per;
  const int kb1 = kb0 + per < num_kb ? kb0 + per : num_kb;

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      tc::mbar_init(&full[s], 1);
      tc::mbar_init(&empty[s], 1);
    }
    tc::mbar_init(done, 1);
    *abort_flag = 0;
    tc::fence_mbar_init();
  }
  if (warp == 0 && lane == 0) {
    tc::prefetch_tmap(&tmA);
    tc::prefetch_tmap(&tmB);
  }
  if (warp == 2) tc::tmem_alloc(tmem_slot, TBN);
  tc::tc_fence_before();
  __syncthreads();
  tc::tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;

  if (warp == 0) {
    if (lane == 0) {
      for (int kb = kb0; kb < kb1; ++kb) {
        const int i = kb - kb0;
        const int s = i % STAGES;
        const uint32_t ph = (uint32_t)(i / STAGES) & 1u;
        if (!tc::mbar_wait(&empty[s], ph ^ 1u, abort_flag)) break;
        uint8_t* sa = smem + s * STAGE_BYTES;
        tc::mbar_arrive_expect_tx(&full[s], STAGE_BYTES);
        if constexpr (TA) {
#pragma unroll
          for (int h = 0; h < BM / 64; ++h) tc::tma_load_2d(sa + h * 64 * BK * 2, &tmA, &full[s], m0 + 64 * h, kb * BK);
        } else {
          tc::tma_load_2d(sa, &tmA, &full[s], kb * BK, m0);
        }
        if constexpr (TB) {
#pragma unroll
          for (int h = 0; h < TBN / 64; ++h)
            tc::tma_load_2d(sa + A_BYTES + h * 64 * BK * 2, &tmB, &full[s], n0 + 64 * h, kb * BK);
        } else {
          tc::tma_load_2d(sa + A_BYTES, &tmB, &full[s], kb * BK, n0);
        }
      }
    }
  } else if (warp == 1) {
    if (lane == 0) {
      constexpr uint32_t idesc = tc::idesc_bf16_f32(BM, TBN) | (TA ? 1u << 15 : 0u) | (TB ? 1u << 16 : 0u);
      bool ok = true;
      for (int kb = kb0; kb < kb1; ++kb) {
        const int i = kb - kb0;
        const int s = i % STAGES;
        const uint32_t ph = (uint32_t)(i / STAGES) & 1u;
        if (!tc::mbar_wait(&full[s], ph, abort_flag)) {
          ok = false;
          break;
        }
        tc::tc_fence_after();
        const uint32_t a_addr = tc::smem_u32(smem + s * STAGE_BYTES);
        const uint32_t b_addr = a_addr + A_BYTES;
#pragma unroll
        for (int k = 0; k < BK / UK; ++k) {  // 16 K values: 32 bytes along a K-major row, 16 rows of an MN-major tile
          const uint64_t ad = TA ? sw128_mnmajor_desc(a_addr + k * UK * 128) : tc::sw128_kmajor_desc(a_addr + k * 32);
          const uint64_t bd = TB ? sw128_mnmajor_desc(b_addr + k * UK * 128) : tc::sw128_kmajor_desc(b_addr + k * 32);
          tc::mma_bf16(tmem_base, ad, bd, idesc, (i | k) != 0 ? 1u : 0u);
        }
        tc::mma_commit(&empty[s]);
      }
      if (ok) tc::mma_commit(done);
    }
  } else {
    // epilogue: thread = accumulator row (TMEM lane), 64 columns at a time staged through
    // this warp's 32 x S_PITCH float tile in the drained stage memory
    // (every MMA, and so every TMA load, has completed once `done` fires)
    const int q = warp & 3;
    const int rbase = m0 + q * 32;  // first row of this warp's quarter
    const int rows = e.M - rbase < 32 ? e.M - rbase : 32;
    float* S = reinterpret_cast<float*>(smem) + q * 32 * S_PITCH;
    if (tc::mbar_wait(done, 0, abort_flag)) {
      tc::tc_fence_after();
#pragma unroll 1
      for (int ch = 0; ch < TBN / 64; ++ch) {
        const int nb = n0 + ch * 64;
        if (nb >= e.N) break;
        __syncwarp();
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          float v[32];
          __syncwarp();
          tc::tmem_ld32(tmem_base + ((uint32_t)(q * 32) << 16) + (uint32_t)(ch * 64 + h * 32), v);
#pragma unroll
          for (int j = 0; j < 32; j += 2)
            *reinterpret_cast<float2*>(S + lane * S_PITCH + h * 32 + j) = make_float2(v[j], v[j + 1]);
        }
        __syncwarp();
        // column phase: lane = columns n and n + 1, one accumulator row per step
        const int n = nb + 2 * lane;
        const bool in0 = n < e.N, in1 = n + 1 < e.N;
        if (EPI == EPI_F32) {
          float* C = e.C + blockIdx.z * e.slice + (int64_t)rbase * e.ldc + n;
          const bool pair = in1 && ((reinterpret_cast<uintptr_t>(C) | (uintptr_t)(e.ldc * 4)) & 7) == 0;
          if (in0) {
#pragma unroll 8
            for (int rr = 0; rr < rows; ++rr) {
              const float2 x = *reinterpret_cast<const float2*>(S + rr * S_PITCH + 2 * lane);
              store2(C + (int64_t)rr * e.ldc, x.x, x.y, pair, in1);
            }
          }
        } else if (EPI == EPI_BIAS_GELU || EPI == EPI_BIAS_GELU_H) {
          const float b0 = in0 ? e.bias[n] : 0.f, b1 = in1 ? e.bias[n + 1] : 0.f;
          float* Z = EPI == EPI_BIAS_GELU ? e.Z + (int64_t)rbase * e.ldz + n : nullptr;
          __nv_bfloat16* H = e.H + (int64_t)rbase * e.ldh + n;
          const bool zpair = in1 && ((reinterpret_cast<uintptr_t>(Z) | (uintptr_t)(e.ldz * 4)) & 7) == 0;
          const bool hpair = in1 && ((reinterpret_cast<uintptr_t>(H) | (uintptr_t)(e.ldh * 2)) & 3) == 0;
          if (in0) {
#pragma unroll 4
            for (int rr = 0; rr < rows; ++rr) {
              float2 x = *reinterpret_cast<const float2*>(S + rr * S_PITCH + 2 * lane);
              x.x += b0;
              x.y += b1;
              if (EPI == EPI_BIAS_GELU) store2(Z + (int64_t)rr * e.ldz, x.x, x.y, zpair, in1);
              const __nv_bfloat16 h0 = __float2bfloat16_rn(gelu(x.x)), h1 = __float2bfloat16_rn(gelu(x.y));
              store2(H + (int64_t)rr * e.ldh, h0, h1, hpair, in1);
              if (EPI == EPI_BIAS_GELU && e.HT)
                *reinterpret_cast<float2*>(S + rr * S_PITCH + 2 * lane) =
                    make_float2(__bfloat162float(h0), __bfloat162float(h1));
            }
          }
        } else {
          const float* Z = e.Z + (int64_t)rbase * e.ldz + n;
          __nv_bfloat16* H = e.H + (int64_t)rbase * e.ldh + n;
          const bool zpair = in1 && ((reinterpret_cast<uintptr_t>(Z) | (uintptr_t)(e.ldz * 4)) & 7) == 0;
          const bool hpair = in1 && ((reinterpret_cast<uintptr_t>(H) | (uintptr_t)(e.ldh * 2)) & 3) == 0;
          float c0 = 0.f, c1 = 0.f;
          if (in0) {
#pragma unroll 1
            for (int r8 = 0; r8 < rows; r8 += 8) {
              float2 z[8];  // the pre-activations of 8 rows, all loads issued first
#pragma unroll
              for (int u = 0; u < 8; ++u) {
                z[u] = make_float2(0.f, 0.f);
                if (r8 + u < rows) {
                  const float* p = Z + (int64_t)(r8 + u) * e.ldz;
                  if (zpair) z[u] = *reinterpret_cast<const float2*>(p);
                  else z[u] = make_float2(p[0], in1 ? p[1] : 0.f);
                }
              }
#pragma unroll
              for (int u = 0; u < 8; ++u) {
                const int rr = r8 + u;
                if (rr >= rows) break;
                const float2 x = *reinterpret_cast<const float2*>(S + rr * S_PITCH + 2 * lane);
                const __nv_bfloat16 h0 = __float2bfloat16_rn(x.x * gelu_grad(z[u].x));
                const __nv_bfloat16 h1 = __float2bfloat16_rn(x.y * gelu_grad(z[u].y));
                store2(H + (int64_t)rr * e.ldh, h0, h1, hpair, in1);
                const float f0 = __bfloat162float(h0), f1 = __bfloat162float(h1);
                c0 += f0;
                c1 += f1;
                if (e.HT) *reinterpret_cast<float2*>(S + rr * S_PITCH + 2 * lane) = make_float2(f0, f1);
              }
            }
            if (e.colsum) {
              atomicAdd(&e.colsum[n], c0);
              if (in1) atomicAdd(&e.colsum[n + 1], c1);
            }
          }
        }
        if ((EPI == EPI_BIAS_GELU || EPI == EPI_GELU_BACK) && e.HT) {  // row phase: lane = row m, one column per step
          __syncwarp();
          if (lane < rows) {
            for (int j = 0; j < 64 && nb + j < e.N; ++j)
              e.HT[(int64_t)(nb + j) * e.ldt + rbase + lane] = __float2bfloat16_rn(S[lane * S_PITCH + j]);
          }
        }
      }
    }
  }
  tc::tc_fence_before();
  __syncthreads();
  if (warp == 2) {
    tc::tc_fence_after();
    tc::tmem_dealloc(tmem_base, TBN);
  }
  if (threadIdx.x == 0 && *abort_flag) atomicExch(status, (int32_t)kDevTimeoutEpilogue);
}

// Split-precision products: A and B hold three BF16 parts per value,
// x = x0 + x1 + x2 (x0 = bf16(x), x1 = bf16(x - x0), x2 = bf16(x - x0 - x1)), side
// by side at column offsets 0, kp and 2 kp of each row.  A stage holds all six part
// tiles of one 64-wide K block (A0 A1 A2 B0 B1 B2, 96 KB; two stages), loaded once,
// and the MMA thread issues the pairs (0,0) (0,1) (1,0) (0,2) (2,0) (1,1) from them
// into one FP32 TMEM tile: the dropped terms are below 2^-24 of |a||b|, so C carries
// FP32-level error.  K slices (gridDim.z) cut the K blocks; the F32 epilogue writes
// slice z at C + z * slice.
constexpr int S3_TILE = BM * BK * 2;              // one 128 x 64 BF16 part tile (BM == BN)
constexpr int S3_STAGES = 2;
constexpr int S3_STAGE_BYTES = 6 * S3_TILE;
constexpr int S3_SMEM = 1024 + S3_STAGES * S3_STAGE_BYTES + 256;
static_assert(BM == BN, "the split kernel's part tiles share one size");

__global__ void __launch_bounds__(THREADS, 1)
    split3_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB, int num_kb,
                  EpiArgs e, int32_t* __restrict__ status, int kp) {
  constexpr int kPa[6] = {0, 0, 1, 0, 2, 1};
  constexpr int kPb[6] = {0, 1, 0, 2, 0, 1};
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + S3_STAGES * S3_STAGE_BYTES);
  uint64_t* full = bars;
  uint64_t* empty = bars + S3_STAGES;
  uint64_t* done = bars + 2 * S3_STAGES;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(done + 1);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // blockIdx.x walks the N tiles, so CTAs launched together share an A tile in L2
  const int n0 = blockIdx.x * BN, m0 = blockIdx.y * BM;
  const int per = (num_kb + gridDim.z - 1) / gridDim.z;  // the host sizes the slices so none is empty
  const int kb0 = blockIdx.z * per;
  const int kb1 = kb0 + per < num_kb ? kb0 + per : num_kb;

  if (threadIdx.x == 0) {
    for (int s = 0; s < S3_STAGES; ++s) {
      tc::mbar_init(&full[s], 1);
      tc::mbar_init(&empty[s], 1);
    }
    tc::mbar_init(done, 1);
    *abort_flag = 0;
    tc::fence_mbar_init();
  }
  if (warp == 0 && lane == 0) {
    tc::prefetch_tmap(&tmA);
    tc::prefetch_tmap(&tmB);
  }
  if (warp == 2) tc::tmem_alloc(tmem_slot, BN);
  tc::tc_fence_before();
  __syncthreads();
  tc::tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;

  if (warp == 0) {
    if (lane == 0) {
      for (int kb = kb0; kb < kb1; ++kb) {
        const int i = kb - kb0;
        const int s = i % S3_STAGES;
        const uint32_t ph = (uint32_t)(i / S3_STAGES) & 1u;
        if (!tc::mbar_wait(&empty[s], ph ^ 1u, abort_flag)) break;
        uint8_t* st = smem + s * S3_STAGE_BYTES;
        tc::mbar_arrive_expect_tx(&full[s], S3_STAGE_BYTES);
#pragma unroll
        for (int p = 0; p < 3; ++p) {
          tc::tma_load_2d(st + p * S3_TILE, &tmA, &full[s], p * kp + kb * BK, m0);
          tc::tma_load_2d(st + (3 + p) * S3_TILE, &tmB, &full[s], p * kp + kb * BK, n0);
        }
      }
    }
  } else if (warp == 1) {
    if (lane == 0) {
      constexpr uint32_t idesc = tc::idesc_bf16_f32(BM, BN);
      bool ok = true;
      for (int kb = kb0; kb < kb1; ++kb) {
        const int i = kb - kb0;
        const int s = i % S3_STAGES;
        const uint32_t ph = (uint32_t)(i / S3_STAGES) & 1u;
        if (!tc::mbar_wait(&full[s], ph, abort_flag)) {
          ok = false;
          break;
        }
        tc::tc_fence_after();
        const uint32_t st = tc::smem_u32(smem + s * S3_STAGE_BYTES);
#pragma unroll
        for (int pr = 0; pr < 6; ++pr) {
          const uint32_t a_addr = st + kPa[pr] * S3_TILE, b_addr = st + (3 + kPb[pr]) * S3_TILE;
#pragma unroll
          for (int k = 0; k < BK / UK; ++k)
            tc::mma_bf16(tmem_base, tc::sw128_kmajor_desc(a_addr + k * 32), tc::sw128_kmajor_desc(b_addr + k * 32),
                         idesc, (i | pr | k) != 0 ? 1u : 0u);
        }
        tc::mma_commit(&empty[s]);
      }
      if (ok) tc::mma_commit(done);
    }
  } else {
    // epilogue: thread = accumulator row (TMEM lane), 32 columns per tcgen05.ld,
    // staged through this warp's 32 x 33 float tile in the drained stage memory so a
    // warp instruction writes 32 consecutive columns of one row
    const int q = warp & 3;
    const int rbase = m0 + q * 32;
    float* S = reinterpret_cast<float*>(smem) + q * 32 * 33;
    if (tc::mbar_wait(done, 0, abort_flag)) {
      tc::tc_fence_after();
      float* C = e.C + blockIdx.z * e.slice;
      for (int ch = 0; ch < BN / 32 && n0 + ch * 32 < e.N; ++ch) {
        float v[32];
        __syncwarp();
        tc::tmem_ld32(tmem_base + ((uint32_t)(q * 32) << 16) + (uint32_t)(ch * 32), v);
#pragma unroll
        for (int j = 0; j < 32; ++j) S[lane * 33 + j] = v[j];
        __syncwarp();
        const int n = n0 + ch * 32 + lane;
        if (n < e.N)
          for (int rr = 0; rr < 32 && rbase + rr < e.M; ++rr) C[(int64_t)(rbase + rr) * e.ldc + n] = S[rr * 33 + lane];
      }
    }
  }
  tc::tc_fence_before();
  __syncthreads();
  if (warp == 2) {
    tc::tc_fence_after();
    tc::tmem_dealloc(tmem_base, BN);
  }
  if (threadIdx.x == 0 && *abort_flag) atomicExch(status, (int32_t)kDevTimeoutEpilogue);
}

template <int EPI, bool TA, bool TB, int TBN>
static int launch_tile(const void* A, const void* B, int M, int N, int K, int lda, int ldb, int num_kb, int slices,
                       const EpiArgs& e, int32_t* status, cudaStream_t stream) {
  static bool attr[64] = {false};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 64 && !attr[dev]) {
    UMAPB_CUDA_TRY(cudaFuncSetAttribute(gemm_kernel<EPI, TA, TB, TBN>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                        Tile<TBN>::kSmem),
                   "gemm: smem attribute");
    attr[dev] = true;
  }
  CUtensorMap ta, tb;
  int s;
  if ((s = TA ? make_tmap_bf16_2d(&ta, A, (uint64_t)K, (uint64_t)M, (uint64_t)lda, BK, 64)
              : make_tmap_bf16_2d(&ta, A, (uint64_t)M, (uint64_t)K, (uint64_t)lda, BM, BK)))
    return s;
  if ((s = TB ? make_tmap_bf16_2d(&tb, B, (uint64_t)K, (uint64_t)N, (uint64_t)ldb, BK, 64)
              : make_tmap_bf16_2d(&tb, B, (uint64_t)N, (uint64_t)K, (uint64_t)ldb, TBN, BK)))
    return s;
  dim3 grid((unsigned)(ceil_div(N, TBN) * ceil_div(M, BM)), 1, (unsigned)slices);
  gemm_kernel<EPI, TA, TB, TBN><<<grid, THREADS, Tile<TBN>::kSmem, stream>>>(ta, tb, num_kb, e, status);
  UMAPB_LAUNCH_CHECK("gemm kernel launch");
  count_launches(1);
  return UMAPB_OK;
}

template <int EPI, bool TA, bool TB>
static int launch(const void* A, const void* B, int M, int N, int K, int lda, int ldb, int ksplit, const EpiArgs& e,
                  int32_t* status, cudaStream_t stream) {
  const int num_kb = (int)ceil_div(K, BK);
  const int per = (int)ceil_div(num_kb, ksplit);
  const int slices = (int)ceil_div(num_kb, per);  // every slice gets at least one K block
  if (slices < ksplit)  // the caller sums ksplit slices: the ones without K blocks hold zeros
    UMAPB_CUDA_TRY(cudaMemsetAsync(e.C + slices * e.slice, 0, sizeof(float) * (size_t)(ksplit - slices) * e.slice,
                                   stream),
                   "gemm: empty slices");
  // 128-wide tiles read A half as often; 64-wide ones when those would not give every SM a tile
  if (ceil_div(M, BM) * ceil_div(N, 128) * slices >= num_sms())
    return launch_tile<EPI, TA, TB, 128>(A, B, M, N, K, lda, ldb, num_kb, slices, e, status, stream);
  return launch_tile<EPI, TA, TB, 64>(A, B, M, N, K, lda, ldb, num_kb, slices, e, status, stream);
}

template <bool TA, bool TB>
static int run(const void* A, const void* B, int M, int N, int K, int lda, int ldb, int epilogue, int ksplit,
               const EpiArgs& e, int32_t* status, cudaStream_t stream) {
  switch (epilogue) {
    case EPI_F32:
      UMAPB_REQUIRE(e.C && e.ldc >= N, "gemm: EPI_F32 needs C with ldc >= N");
      return launch<EPI_F32, TA, TB>(A, B, M, N, K, lda, ldb, ksplit, e, status, stream);
    case EPI_BIAS_GELU:
      UMAPB_REQUIRE(e.bias && e.Z && e.H && e.ldz >= N && e.ldh >= N && (!e.HT || e.ldt >= M),
                    "gemm: EPI_BIAS_GELU needs bias, Z and H (and ldt >= M for HT)");
      if constexpr (!TA && !TB)
        return launch<EPI_BIAS_GELU, TA, TB>(A, B, M, N, K, lda, ldb, 1, e, status, stream);
      break;
    case EPI_GELU_BACK:
      UMAPB_REQUIRE(e.Z && e.H && e.ldz >= N && e.ldh >= N && (!e.HT || e.ldt >= M),
                    "gemm: EPI_GELU_BACK needs Z and H (and ldt >= M for HT)");
      if constexpr (!TA) {
        if (e.colsum) UMAPB_CUDA_TRY(cudaMemsetAsync(e.colsum, 0, sizeof(float) * N, stream), "gemm: colsum reset");
        return launch<EPI_GELU_BACK, TA, TB>(A, B, M, N, K, lda, ldb, 1, e, status, stream);
      }
      break;
    case EPI_BIAS_GELU_H:
      UMAPB_REQUIRE(e.bias && e.H && e.ldh >= N, "gemm: EPI_BIAS_GELU_H needs bias and H");
      if constexpr (!TA && !TB)
        return launch<EPI_BIAS_GELU_H, TA, TB>(A, B, M, N, K, lda, ldb, 1, e, status, stream);
      break;
    default:
      return set_error(UMAPB_ERR_ARG, "gemm: unknown epilogue %d", epilogue);
  }
  return set_error(UMAPB_ERR_UNSUPPORTED, "gemm: epilogue %d is not built for these operand layouts", epilogue);
}

}  // namespace gemm
}  // namespace umapb

using namespace umapb;

extern "C" int umapb_gemm_bf16_layout(const void* A, int32_t a_mn, const void* B, int32_t b_mn, int32_t M, int32_t N,
                                      int32_t K, int32_t lda, int32_t ldb, int32_t epilogue, int32_t ksplit, float* C,
                                      int32_t ldc, const float* bias, float* Z, int32_t ldz, void* H, int32_t ldh,
                                      void* HT, int32_t ldt, float* colsum, int32_t* status, umapb_stream_t stream_) {
  clear_error();
  cudaStream_t stream = reinterpret_cast<cudaStream_t>(stream_);
  UMAPB_REQUIRE(A && B && status, "gemm: null operand");
  UMAPB_REQUIRE(M >= 1 && N >= 1 && K >= 1, "gemm: empty shape");
  UMAPB_REQUIRE(lda >= (a_mn ? M : K) && ldb >= (b_mn ? N : K) && lda % 8 == 0 && ldb % 8 == 0,
                "gemm: lda/ldb must be >= K and multiples of 8 elements (16-byte rows)");
  UMAPB_REQUIRE(ksplit >= 1 && ksplit <= 64, "gemm: ksplit must be in [1, 64]");
  UMAPB_REQUIRE(ksplit == 1 || epilogue == gemm::EPI_F32, "gemm: K slices need the F32 epilogue");
  gemm::EpiArgs e{M, N, C, ldc, bias, Z, ldz, static_cast<__nv_bfloat16*>(H), ldh, static_cast<__nv_bfloat16*>(HT),
                  ldt, colsum, (int64_t)M * ldc};
  if (!a_mn && !b_mn) return gemm::run<false, false>(A, B, M, N, K, lda, ldb, epilogue, ksplit, e, status, stream);
  if (!a_mn) return gemm::run<false, true>(A, B, M, N, K, lda, ldb, epilogue, ksplit, e, status, stream);
  if (b_mn) return gemm::run<true, true>(A, B, M, N, K, lda, ldb, epilogue, ksplit, e, status, stream);
  return set_error(UMAPB_ERR_UNSUPPORTED, "gemm: A by K rows with B by N rows is not built");
}

extern "C" int umapb_gemm_bf16(const void* A, const void* B, int32_t M, int32_t N, int32_t K, int32_t lda,
                               int32_t ldb, int32_t epilogue, int32_t ksplit, float* C, int32_t ldc, const float* bias,
                               float* Z, int32_t ldz, void* H, int32_t ldh, void* HT, int32_t ldt, float* colsum,
                               int32_t* status, umapb_stream_t stream_) {
  return umapb_gemm_bf16_layout(A, 0, B, 0, M, N, K, lda, ldb, epilogue, ksplit, C, ldc, bias, Z, ldz, H, ldh, HT, ldt,
                                colsum, status, stream_);
}

extern "C" int umapb_gemm_split3(const void* A3, const void* B3, int32_t M, int32_t N, int32_t kp, int32_t ksplit,
                                 float* C, int32_t ldc, int32_t* status, umapb_stream_t stream_) {
  clear_error();
  cudaStream_t stream = reinterpret_cast<cudaStream_t>(stream_);
  UMAPB_REQUIRE(A3 && B3 && C && status, "gemm_split3: null argument");
  UMAPB_REQUIRE(M >= 1 && N >= 1 && kp >= gemm::BK && kp % gemm::BK == 0,
                "gemm_split3: need M, N >= 1 and kp a positive multiple of 64");
  UMAPB_REQUIRE((int64_t)kp * 3 < ((int64_t)1 << 31), "gemm_split3: kp too large");
  UMAPB_REQUIRE(ldc >= N, "gemm_split3: ldc must be >= N");
  UMAPB_REQUIRE(ksplit >= 1 && ksplit <= 4096, "gemm_split3: ksplit must be in [1, 4096]");
  static bool attr[64] = {false};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev >= 0 && dev < 64 && !attr[dev]) {
    UMAPB_CUDA_TRY(cudaFuncSetAttribute(gemm::split3_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                        gemm::S3_SMEM),
                   "gemm_split3: smem attribute");
    attr[dev] = true;
  }
  CUtensorMap ta, tb;
  int s;
  const uint64_t w = (uint64_t)kp * 3;
  if ((s = make_tmap_bf16_2d(&ta, A3, (uint64_t)M, w, w, gemm::BM, gemm::BK))) return s;
  if ((s = make_tmap_bf16_2d(&tb, B3, (uint64_t)N, w, w, gemm::BN, gemm::BK))) return s;
  const int num_kb = kp / gemm::BK;
  const int per = (int)ceil_div(num_kb, ksplit);
  const int slices = (int)ceil_div(num_kb, per);  // every slice gets at least one K block
  gemm::EpiArgs e{M, N, C, ldc, nullptr, nullptr, 0, nullptr, 0, nullptr, 0, nullptr, (int64_t)M * ldc};
  if (slices < ksplit)  // the caller sums ksplit slices: the ones without K blocks hold zeros
    UMAPB_CUDA_TRY(cudaMemsetAsync(C + slices * e.slice, 0, sizeof(float) * (size_t)(ksplit - slices) * e.slice,
                                   stream),
                   "gemm_split3: empty slices");
  dim3 grid((unsigned)ceil_div(N, gemm::BN), (unsigned)ceil_div(M, gemm::BM), (unsigned)slices);
  gemm::split3_kernel<<<grid, gemm::THREADS, gemm::S3_SMEM, stream>>>(ta, tb, num_kb, e, status, kp);
  UMAPB_LAUNCH_CHECK("gemm_split3 kernel launch");
  count_launches(1);
  return UMAPB_OK;
}
