// Spectral initialisation — replaces UMAP._spectral_init, mlx_vis/_umap/umap.py:298-348.
//
// The reference: degrees by scatter-add (float32, edge order), d^-1/2, normalised
// weights w * d_r^-1/2 * d_c^-1/2, then 100 x { V = W V (gather + scatter-add);
// modified Gram-Schmidt with norm sqrt(|v|^2 + 1e-10) } on V (n x (c+1)), take
// columns 1..c, scale by 10 / max|e|, add N(0, 1e-4) noise (NumPy, host) and
// min-max each column to [0, 10].
//
// Here the edges are in row-major order, so W V is a CSR SpMV without atomics
// (2 lanes per row, FP64 partial sums combined by shuffles; V kept in FP32 rows
// padded to 16 bytes, one vector load per edge, Gram matrix and R^-1 in FP64).  MGS of the
// (c+1)-column block equals Q = V R^-1 with R the Cholesky factor of the Gram
// matrix V^T V (+1e-10 on each pivot, as in the reference's norms), so each
// iteration is ONE kernel: it applies the previous iteration's R^-1 and accumulates
// the new Gram matrix in FP64.  By default all iterations run in one cooperative
// launch (power_kernel).
#include <math.h>
#include <stdlib.h>

#include <mutex>

#include "cluster.cuh"
#include "common.cuh"
#include "philox.cuh"

namespace umapb {
namespace spectral {

constexpr int kBlock = 256;
constexpr int kMaxCols = 5;   // the fused kernels: n_components <= 4
constexpr int kLanes = 2;     // lanes per row in the power iteration
constexpr int kWideCols = 33; // the warp-per-row kernels: n_components <= 32
constexpr int kWideRows = 32; // rows per block in the warp-per-row SpMV

__global__ void row_ptr_kernel(const int32_t* __restrict__ rows, const int64_t* __restrict__ n_edges, int64_t n,
                               int64_t* __restrict__ row_ptr) {
  const int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (r > n) return;
  const int64_t E = *n_edges;
  int64_t lo = 0, hi = E;  // lower_bound of r in rows[0, E)
  while (lo < hi) {
    const int64_t mid = (lo + hi) >> 1;
    if (rows[mid] < r) lo = mid + 1;
    else hi = mid;
  }
  row_ptr[r] = lo;
}

// degree (float32, reference edge order), then normalised weights
__global__ void degree_kernel(const float* __restrict__ vals, const int64_t* __restrict__ row_ptr, int64_t n,
                              float* __restrict__ dis) {
  const int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (r >= n) return;
  float d = 0.f;
  for (int64_t e = row_ptr[r]; e < row_ptr[r + 1]; ++e) d = __fadd_rn(d, vals[e]);
  d = fmaxf(d, 1e-10f);
  dis[r] = __fdiv_rn(1.0f, sqrtf(d));
}

__global__ void norm_weight_kernel(const int32_t* __restrict__ rows, const int32_t* __restrict__ cols,
                                   const float* __restrict__ vals, const int64_t* __restrict__ n_edges,
                                   const float* __restrict__ dis, float* __restrict__ wn) {
  const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= *n_edges) return;
  wn[e] = __fmul_rn(__fmul_rn(vals[e], dis[rows[e]]), dis[cols[e]]);
}

// R (upper triangular) from the Gram matrix G with pivots sqrt(g - sum r^2 + 1e-10);
// returns Rinv (upper triangular) in `ri`.  kk <= kMaxCols.
__device__ void chol_inverse(const double* G, int kk, double* ri) {
  double R[kMaxCols][kMaxCols];
  for (int j = 0; j < kk; ++j) {
    for (int i = 0; i < j; ++i) {
      double s = G[i * kk + j];
      for (int p = 0; p < i; ++p) s -= R[p][i] * R[p][j];
      R[i][j] = s / R[i][i];
    }
    double s = G[j * kk + j];
    for (int p = 0; p < j; ++p) s -= R[p][j] * R[p][j];
    R[j][j] = sqrt(fmax(s, 0.0) + 1e-10);
    for (int i = j + 1; i < kk; ++i) R[i][j] = 0.0;
  }
  // invert the upper-triangular R column by column
  for (int j = 0; j < kk; ++j) {
    for (int i = kk - 1; i >= 0; --i) {
      double s = (i == j) ? 1.0 : 0.0;
      for (int p = i + 1; p < kk; ++p) s -= R[i][p] * ri[p * kk + j];
      ri[i * kk + j] = (i <= j) ? s / R[i][i] : 0.0;
    }
  }
}

// One power iteration: Vout = W (Vin Rinv_in); G_out += Vout^T Vout.  Rinv_in ==
// nullptr means the identity (the first multiplication uses V0 as is).  kLanes
// lanes per row stride over its edges (rows of the symmetrised graph range from a
// few edges to hundreds) and meet by shuffles.  The last block to finish (a counter
// per iteration) factors the completed G_out once and writes Rinv_out for the next
// iteration.
__global__ void spmv_gram_kernel(const float* __restrict__ Vin, const double* __restrict__ Rinv_in,
                                 const int64_t* __restrict__ row_ptr, const int32_t* __restrict__ cols,
                                 const float* __restrict__ wn, int64_t n, int kk, int vp, float* __restrict__ Vout,
                                 double* __restrict__ G_out, unsigned* __restrict__ counter,
                                 double* __restrict__ Rinv_out) {
  __shared__ double ri[kMaxCols * kMaxCols];
  __shared__ double gsum[kBlock / 32][kMaxCols * kMaxCols];
  __shared__ bool last;
  if (threadIdx.x < kk * kk)
    ri[threadIdx.x] = Rinv_in ? Rinv_in[threadIdx.x] : ((threadIdx.x % (kk + 1) == 0) ? 1.0 : 0.0);
  __syncthreads();
  const int sub = threadIdx.x & (kLanes - 1);
  const int64_t r = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) / kLanes;
  double acc[kMaxCols] = {0, 0, 0, 0, 0};
  if (r < n) {
    const int64_t e1 = row_ptr[r + 1];
    for (int64_t e = row_ptr[r] + sub; e < e1; e += kLanes) {
      const int64_t c = cols[e];
      const double w = (double)wn[e];
      double v[kMaxCols];
      const float4 a = reinterpret_cast<const float4*>(Vin + c * vp)[0];  // rows padded to 4 or 8 floats
      v[0] = a.x, v[1] = a.y, v[2] = a.z, v[3] = a.w;
      if (kk > 4) v[4] = Vin[c * vp + 4];
      for (int j = 0; j < kk; ++j) {  // q_j = sum_i v_i Rinv[i][j]
        double q = 0.0;
        for (int i = 0; i <= j; ++i) q += v[i] * ri[i * kk + j];
        acc[j] += w * q;
      }
    }
  }
  for (int j = 0; j < kk; ++j) {
#pragma unroll
    for (int o = kLanes / 2; o > 0; o >>= 1) acc[j] += __shfl_xor_sync(0xffffffffu, acc[j], o);
  }
  if (r < n && sub == 0)
    for (int j = 0; j < vp; ++j) Vout[r * vp + j] = j < kk ? (float)acc[j] : 0.f;
  if (sub != 0)
    for (int j = 0; j < kk; ++j) acc[j] = 0.0;  // one copy of each row in the Gram sum
  // block reduction of the Gram matrix
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int i = 0; i < kk; ++i) {
    for (int j = i; j < kk; ++j) {
      double g = acc[i] * acc[j];
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) g += __shfl_xor_sync(0xffffffffu, g, o);
      if (lane == 0) gsum[warp][i * kk + j] = g;
    }
  }
  __syncthreads();
  if (threadIdx.x < kk * kk) {
    const int i = threadIdx.x / kk, j = threadIdx.x % kk;
    if (i <= j) {
      double g = 0.0;
      for (int w = 0; w < kBlock / 32; ++w) g += gsum[w][i * kk + j];
      atomicAdd(&G_out[i * kk + j], g);
      if (i != j) atomicAdd(&G_out[j * kk + i], g);
    }
  }
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) last = atomicAdd(counter, 1u) == gridDim.x - 1;
  __syncthreads();
  if (last && threadIdx.x == 0) {
    __threadfence();
    double G[kMaxCols * kMaxCols];
    for (int i = 0; i < kk * kk; ++i) G[i] = __ldcg(G_out + i);
    chol_inverse(G, kk, Rinv_out);
  }
}


// ---- n_components 5..32: one warp per row, lane j holds column j (and j + 32) ----
// Cholesky factor R of the kk x kk Gram matrix (pivots sqrt(g - sum r^2 + 1e-10),
// the same expressions and summation order as chol_inverse) and its inverse, by the
// whole block in shared memory.  g is overwritten with R (upper triangle).
__device__ void chol_inverse_block(double* g, int kk, double* ri) {
  for (int i = 0; i < kk; ++i) {
    if (threadIdx.x == 0) {
      double s = g[i * kk + i];
      for (int p = 0; p < i; ++p) s -= g[p * kk + i] * g[p * kk + i];
      g[i * kk + i] = sqrt(fmax(s, 0.0) + 1e-10);
    }
    __syncthreads();
    for (int j = i + 1 + threadIdx.x; j < kk; j += blockDim.x) {
      double s = g[i * kk + j];
      for (int p = 0; p < i; ++p) s -= g[p * kk + i] * g[p * kk + j];
      g[i * kk + j] = s / g[i * kk + i];
    }
    __syncthreads();
  }
  for (int j = threadIdx.x; j < kk; j += blockDim.x) {  // column j of R^-1
    for (int i = kk - 1; i >= 0; --i) {
      double s = (i == j) ? 1.0 : 0.0;
      for (int p = i + 1; p < kk; ++p) s -= (p > j ? 0.0 : g[i * kk + p] * ri[p * kk + j]);
      ri[i * kk + j] = (i <= j) ? s / g[i * kk + i] : 0.0;
    }
  }
  __syncthreads();
}

// q_j = sum_{i <= j} u_i Rinv[i][j] for the columns j = lane and lane + 32 of a warp's row
__device__ __forceinline__ void apply_rinv_wide(double u0, double u1, const double* ri, int kk, int lane,
                                                double& q0, double& q1) {
  q0 = 0.0, q1 = 0.0;
  for (int i = 0; i < kk; ++i) {
    const double ui = __shfl_sync(0xffffffffu, i < 32 ? u0 : u1, i & 31);
    if (lane < kk && i <= lane) q0 += ui * ri[i * kk + lane];
    if (lane + 32 < kk && i <= lane + 32) q1 += ui * ri[i * kk + lane + 32];
  }
}

// One power iteration for kk > kMaxCols: Vout = (W Vin) Rinv_in (W Vin in FP64 per
// row, one warp per row), G_out += Vout^T Vout from the block's rows staged in
// shared memory; the last block factors G_out into Rinv_out.
__global__ void __launch_bounds__(kBlock) spmv_gram_wide_kernel(
    const float* __restrict__ Vin, const double* __restrict__ Rinv_in, const int64_t* __restrict__ row_ptr,
    const int32_t* __restrict__ cols, const float* __restrict__ wn, int64_t n, int kk, int vp,
    float* __restrict__ Vout, double* __restrict__ G_out, unsigned* __restrict__ counter,
    double* __restrict__ Rinv_out) {
  __shared__ double ri[kWideCols * kWideCols];
  __shared__ double gl[kWideCols * kWideCols];
  __shared__ double vs[kWideRows][kWideCols];
  __shared__ bool last;
  for (int t = threadIdx.x; t < kk * kk; t += blockDim.x)
    ri[t] = Rinv_in ? Rinv_in[t] : ((t % (kk + 1) == 0) ? 1.0 : 0.0);
  __syncthreads();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t rb = (int64_t)blockIdx.x * kWideRows;
  for (int lr = warp; lr < kWideRows; lr += kBlock / 32) {
    const int64_t r = rb + lr;
    double u0 = 0.0, u1 = 0.0;
    if (r < n) {
      const int64_t e1 = row_ptr[r + 1];
      for (int64_t e = row_ptr[r]; e < e1; ++e) {
        const int64_t c = cols[e];
        const double w = (double)wn[e];
        if (lane < kk) u0 += w * (double)Vin[c * vp + lane];
        if (lane + 32 < kk) u1 += w * (double)Vin[c * vp + lane + 32];
      }
    }
    double q0, q1;
    apply_rinv_wide(u0, u1, ri, kk, lane, q0, q1);
    if (r < n) {
      if (lane < vp) Vout[r * vp + lane] = lane < kk ? (float)q0 : 0.f;
      if (lane + 32 < vp) Vout[r * vp + lane + 32] = lane + 32 < kk ? (float)q1 : 0.f;
    }
    vs[lr][lane] = (r < n && lane < kk) ? q0 : 0.0;
    if (lane + 32 < kWideCols) vs[lr][lane + 32] = (r < n && lane + 32 < kk) ? q1 : 0.0;
  }
  __syncthreads();
  for (int t = threadIdx.x; t < kk * kk; t += blockDim.x) {
    const int i = t / kk, j = t % kk;
    if (i <= j) {
      double g = 0.0;
      for (int lr = 0; lr < kWideRows; ++lr) g += vs[lr][i] * vs[lr][j];
      atomicAdd(&G_out[i * kk + j], g);
      if (i != j) atomicAdd(&G_out[j * kk + i], g);
    }
  }
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) last = atomicAdd(counter, 1u) == gridDim.x - 1;
  __syncthreads();
  if (!last) return;
  __threadfence();
  for (int t = threadIdx.x; t < kk * kk; t += blockDim.x) gl[t] = __ldcg(G_out + t);
  __syncthreads();
  chol_inverse_block(gl, kk, ri);
  for (int t = threadIdx.x; t < kk * kk; t += blockDim.x) Rinv_out[t] = ri[t];
}

// embedding = (V R^-1)[:, 1:] and max |embedding| for kk > kMaxCols (one warp per row)
__global__ void __launch_bounds__(kBlock) finish_orth_wide_kernel(const float* __restrict__ V,
                                                                  const double* __restrict__ Rinv, int64_t n, int kk,
                                                                  int vp, float* __restrict__ emb,
                                                                  unsigned* __restrict__ absmax) {
  __shared__ double ri[kWideCols * kWideCols];
  for (int t = threadIdx.x; t < kk * kk; t += blockDim.x) ri[t] = Rinv[t];
  __syncthreads();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t r = (int64_t)blockIdx.x * (kBlock / 32) + warp;
  float m = 0.f;
  const double v0 = (r < n && lane < kk) ? (double)V[r * vp + lane] : 0.0;
  const double v1 = (r < n && lane + 32 < kk) ? (double)V[r * vp + lane + 32] : 0.0;
  double q0, q1;
  apply_rinv_wide(v0, v1, ri, kk, lane, q0, q1);
  if (r < n) {
    if (lane >= 1 && lane < kk) {
      const float f = (float)q0;
      emb[r * (kk - 1) + (lane - 1)] = f;
      m = fabsf(f);
    }
    if (lane + 32 < kk) {
      const float f = (float)q1;
      emb[r * (kk - 1) + (lane + 31)] = f;
      m = fmaxf(m, fabsf(f));
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
  if (lane == 0) atomicMax(absmax, __float_as_uint(m));
}

// ---- all power iterations in one cooperative launch ---------------------------
// The grid stays resident, one block per SM: a block owns a contiguous range of rows
// and keeps their edges (ids, weights and row offsets) in shared memory, as many as
// fit, so that an iteration reads nothing but the gathered rows of V, which other blocks
// write and which come through L2 (ld.global.cg).  One grid barrier ends an
// iteration.  R^-1 is applied to a row's sums, after the gather, so the block's last warp
// factors the completed Gram matrix while the others gather; it has no rows.
//
// What bounds it: n k random 16-byte reads of V from L2 an iteration (1.05 M of the
// 70,000-row iteration's 7.7 us are 3.6 us at the measured random-access rate), then the
// barrier.  B200, 100 iterations, k = 15, 2 components: 70,000 rows 1072 -> 768 us against
// one thread's factorisation between the barrier and the gather, the edges read from L2
// and 4 blocks per SM in the barrier.
// (A factorisation every few iterations only, as the shrinkage of the columns allows, is
// as exact but rounds V to FP32 in another basis; 25 layout epochs later that differs
// visibly from a factorisation per iteration.)
//
// The barrier gives up after limit_ns (umapb_set_wait_limit_ns, 2 s by default), raises
// a shared abort flag and the status word, and every block then returns.

// the inverse of R in registers (KK a constant), one reciprocal square root per pivot
template <int KK>
__device__ __forceinline__ void chol_inverse_fixed(const double (&G)[KK * KK], double (&ri)[KK * KK]) {
  double R[KK][KK], inv[KK];
#pragma unroll
  for (int j = 0; j < KK; ++j) {
#pragma unroll
    for (int i = 0; i < j; ++i) {
      double s = G[i * KK + j];
#pragma unroll
      for (int p = 0; p < i; ++p) s -= R[p][i] * R[p][j];
      R[i][j] = s * inv[i];
    }
    double s = G[j * KK + j];
#pragma unroll
    for (int p = 0; p < j; ++p) s -= R[p][j] * R[p][j];
    inv[j] = rsqrt(fmax(s, 0.0) + 1e-10);  // the pivot itself is not needed
  }
#pragma unroll
  for (int j = 0; j < KK; ++j) {
#pragma unroll
    for (int i = KK - 1; i >= 0; --i) {
      double s = (i == j) ? 1.0 : 0.0;
#pragma unroll
      for (int p = i + 1; p <= j; ++p) s -= R[i][p] * ri[p * KK + j];
      ri[i * KK + j] = (i <= j) ? s * inv[i] : 0.0;
    }
  }
}

__device__ __forceinline__ unsigned long long gtimer() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

__device__ bool grid_barrier(unsigned* bar, unsigned target, int* abort_g, unsigned long long limit_ns) {
  __shared__ int s_ok;
  __syncthreads();
  if (threadIdx.x == 0) {
    int ok = 1;
    // the block's writes are ordered before this by the block barrier
    asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(bar) : "memory");
    const unsigned long long t0 = gtimer();
    for (unsigned i = 1;; ++i) {
      unsigned v;
      asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(bar) : "memory");
      if (v >= target) break;
      if ((i & 255) == 0 && *(volatile int*)abort_g) {
        ok = 0;
        break;
      }
      if (gtimer() - t0 > limit_ns) {
        atomicExch(abort_g, 1);
        ok = 0;
        break;
      }
    }
    s_ok = ok;
  }
  __syncthreads();
  return s_ok != 0;
}

// The upper triangle of a block's Gram matrix.  Both lanes of a row hold the same products, so
// each sums half of the entries over its warp; warp e then adds entry e over the warps and holds it
// in every lane.  (Every entry over all lanes and one thread's chain over 32 warps were
// 0.2 us more of an iteration: 788 -> 768 us at 70,000 rows, 354 -> 325 us in the cluster at 2,000.)
template <int KK>
struct Upper {
  static constexpr int kEntries = KK * (KK + 1) / 2, kHalf = (kEntries + 1) / 2;
  static __host__ __device__ constexpr int at(int e) {  // entry e of the triangle in KK x KK
    int i = 0;
    while (e >= KK - i) {
      e -= KK - i;
      ++i;
    }
    return i * KK + i + e;
  }
};

template <int KK, int WARPS>
__device__ __forceinline__ double block_gram(const double (&part)[KK * KK], double (*gsum)[WARPS]) {
  using U = Upper<KK>;
  static_assert(U::kEntries <= WARPS && WARPS <= 32, "one warp per entry, one lane per warp");
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, sub = threadIdx.x & 1;
  double tri[2 * U::kHalf];
  tri[2 * U::kHalf - 1] = 0.0;
#pragma unroll
  for (int i = 0, e = 0; i < KK; ++i)
#pragma unroll
    for (int j = i; j < KK; ++j, ++e) tri[e] = part[i * KK + j];
#pragma unroll
  for (int h = 0; h < U::kHalf; ++h) {
    double g = sub ? tri[U::kHalf + h] : tri[h];
#pragma unroll
    for (int o = 16; o > 1; o >>= 1) g += __shfl_xor_sync(0xffffffffu, g, o);
    if (lane < 2 && sub * U::kHalf + h < U::kEntries) gsum[sub * U::kHalf + h][warp] = g;
  }
  __syncthreads();
  double g = 0.0;
  if (warp < U::kEntries) {
    g = lane < WARPS ? gsum[warp][lane] : 0.0;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) g += __shfl_xor_sync(0xffffffffu, g, o);
  }
  return g;
}

constexpr int kPowerThreads = 1024;  // two lanes for each of 496 rows (one pass up to 73,408 rows) and the factor warp
constexpr int kPowerRowThreads = kPowerThreads - 32;
// Dynamic shared memory at most: with the static part within the 196 KB setting of an SM, which
// leaves L1 60 KB.  The next setting leaves 28, too little for the gathers in flight: 100 iterations
// of 150,000 rows, k = 20, 2 components, 200 KB and 188 KB 2628 and 1765 us; 300,000 rows, k = 10, 4
// components 5764 and 3895.
constexpr size_t kPowerSmem = 188 * 1024;

template <int KK>  // columns of V: n_components + 1
__global__ void __launch_bounds__(kPowerThreads, 1)
    power_kernel(float* __restrict__ V0, float* __restrict__ V1, const int64_t* __restrict__ row_ptr,
                 const int32_t* __restrict__ cols, const float* __restrict__ wn, int64_t n, int rows_per_block,
                 int off_cap, int edge_cap, int n_iter, double* __restrict__ G, double* __restrict__ Rinv,
                 unsigned* __restrict__ bar, int* __restrict__ abort_g, int32_t* __restrict__ status,
                 unsigned long long limit_ns) {
  constexpr int vp = KK <= 4 ? 4 : 8;
  constexpr int kWarps = kPowerThreads / 32;
  extern __shared__ __align__(16) unsigned char power_smem[];
  int32_t* s_off = reinterpret_cast<int32_t*>(power_smem);  // off_cap (rows_per_block + 1, or 0) edge offsets
  int32_t* s_col = s_off + off_cap;                         // edge_cap ids
  float* s_w = reinterpret_cast<float*>(s_col + edge_cap);  // edge_cap weights
  __shared__ double ri[KK * KK];
  __shared__ double gsum[Upper<KK>::kEntries][kWarps];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int sub = threadIdx.x & (kLanes - 1);
  const int64_t r_first = (int64_t)blockIdx.x * rows_per_block;
  const int rows = (int)(r_first + rows_per_block < n ? rows_per_block : (n > r_first ? n - r_first : 0));
  const int64_t e_first = rows > 0 ? row_ptr[r_first] : 0;
  const int n_edges = rows > 0 ? (int)(row_ptr[r_first + rows] - e_first) : 0;
  const int staged = n_edges < edge_cap ? n_edges : edge_cap;
  // offset of a row's first edge from the block's first one
  auto off = [&](int t) { return off_cap ? s_off[t] : (int)(row_ptr[r_first + t] - e_first); };
  for (int t = threadIdx.x; off_cap && rows > 0 && t <= rows; t += kPowerThreads)
    s_off[t] = (int)(row_ptr[r_first + t] - e_first);
  for (int e = threadIdx.x; e < staged; e += kPowerThreads) {
    s_col[e] = cols[e_first + e];
    s_w[e] = wn[e_first + e];
  }
  cols += e_first;
  wn += e_first;
  __syncthreads();

  for (int it = 0; it <= n_iter; ++it) {
    // the factor warp: R^-1 of the previous iteration's product, for this one's rows
    if (warp == kWarps - 1 && it > 0) {
      const double* Gp = G + (size_t)(it - 1) * KK * KK;
      const double mine = lane < KK * KK ? __ldcg(Gp + lane) : 0.0;
      double Gl[KK * KK], rl[KK * KK];
#pragma unroll
      for (int t = 0; t < KK * KK; ++t) Gl[t] = __shfl_sync(0xffffffffu, mine, t);  // the upper triangle counts
      chol_inverse_fixed<KK>(Gl, rl);
      if (lane == 0) {
#pragma unroll
        for (int t = 0; t < KK * KK; ++t) ri[t] = rl[t];
        if (blockIdx.x == 0)
          for (int t = 0; t < KK * KK; ++t) Rinv[(size_t)(it - 1) * KK * KK + t] = rl[t];
      }
    }
    if (it == n_iter) break;
    const float* Vin = (it & 1) ? V1 : V0;
    float* Vout = (it & 1) ? V0 : V1;
    double part[KK * KK];
#pragma unroll
    for (int t = 0; t < KK * KK; ++t) part[t] = 0.0;
    // every warp takes the first pass (R^-1 is ready after it) and then the passes that begin at
    // a row of the block, so its lanes meet the shuffle below; rows past the last do no work
    bool first = true;
    for (int w0 = warp * (32 / kLanes); first || w0 < rows; w0 += kPowerRowThreads / kLanes) {
      const int lr = w0 + lane / kLanes;
      const bool valid = lr < rows && warp < kWarps - 1;
      double acc[KK];
#pragma unroll
      for (int j = 0; j < KK; ++j) acc[j] = 0.0;
      const int e1 = valid ? off(lr + 1) : 0;
      int e = valid ? off(lr) + sub : 0;
      // four edges per step: their rows of V are loaded together; the sums keep edge order
      for (; e < e1; e += 4 * kLanes) {
        int c[4];
        float w[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const int x = e + u * kLanes;
          const bool on = x < e1;
          c[u] = on ? (x < staged ? s_col[x] : cols[x]) : -1;
          w[u] = on ? (x < staged ? s_w[x] : wn[x]) : 0.f;
        }
        float4 a[4];
        float a4[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          a[u] = c[u] >= 0 ? __ldcg(reinterpret_cast<const float4*>(Vin + (int64_t)c[u] * vp))  // rows of 4 or 8
                           : make_float4(0.f, 0.f, 0.f, 0.f);
          a4[u] = KK > 4 && c[u] >= 0 ? __ldcg(Vin + (int64_t)c[u] * vp + 4) : 0.f;
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const double wd = (double)w[u];
          const float v[5] = {a[u].x, a[u].y, a[u].z, a[u].w, a4[u]};
#pragma unroll
          for (int j = 0; j < KK; ++j) acc[j] += wd * (double)v[j];
        }
      }
#pragma unroll
      for (int j = 0; j < KK; ++j) acc[j] += __shfl_xor_sync(0xffffffffu, acc[j], 1);  // kLanes == 2
      if (first) __syncthreads();  // R^-1
      first = false;
      if (valid) {
        double q[KK];
#pragma unroll
        for (int j = 0; j < KK; ++j) {
          q[j] = acc[j];
          if (it > 0) {
            q[j] = 0.0;
#pragma unroll
            for (int i = 0; i <= j; ++i) q[j] += acc[i] * ri[i * KK + j];
          }
        }
        float out[vp];
#pragma unroll
        for (int j = 0; j < vp; ++j) out[j] = j < KK ? (float)q[j < KK ? j : 0] : 0.f;
        float4* dst = reinterpret_cast<float4*>(Vout + (r_first + lr) * vp);
        if (sub == 0) dst[0] = make_float4(out[0], out[1], out[2], out[3]);
        if constexpr (vp == 8)
          if (sub == 1) dst[1] = make_float4(out[4], out[5], out[6], out[7]);
#pragma unroll
        for (int i = 0; i < KK; ++i)
#pragma unroll
          for (int j = i; j < KK; ++j) part[i * KK + j] += q[i] * q[j];
      }
    }
    // one atomic per entry and block
    const double gram = block_gram<KK, kWarps>(part, gsum);
    if (warp < Upper<KK>::kEntries && lane == 0) atomicAdd(G + (size_t)it * KK * KK + Upper<KK>::at(warp), gram);
    if (!grid_barrier(bar, (unsigned)(it + 1) * gridDim.x, abort_g, limit_ns)) {
      if (threadIdx.x == 0) atomicExch(status, (int32_t)kDevTimeoutEpilogue);
      return;
    }
  }
}

// The same iterations for few rows by one cluster of 8 CTAs: every CTA holds all of V (two
// buffers) in its shared memory, computes its share of the rows and stores them into
// all eight copies, so an iteration gathers from its own shared memory and ends with the
// cluster's hardware barrier.  The CTAs' Gram matrices are exchanged the same way and
// added in rank order, without atomics.  B200, 2,000 rows, k = 15: 613 -> 325 us against 16
// blocks over L2, where every iteration pays a round trip each for V and the barrier.
// Eight SMs gather an edge a cycle each, the chip 148, so the form is for the rows that one pass of
// the CTAs takes (2,048) as long as shared memory holds their edges, and for few edges in two
// passes.  100 iterations, cluster and grid (its blocks by edges as below), 2 components: 2,048
// rows, k = 15 363 and 486 us, k = 75 814 and 875, k = 90 (not all staged) 1062 and 980; 3,000 rows,
// k = 12 470 and 480; 4,000 rows, k = 10 493 and 499, k = 15 525 and 490; 5,000 rows, k = 50 2166 and 749.
constexpr int kClusterCtas = 8;
constexpr int kClusterThreads = 544;  // 16 warps with rows and the factor warp
constexpr int kClusterRowThreads = kClusterThreads - 32;
constexpr size_t kClusterSmem = 216 * 1024;
constexpr int kClusterPass = kClusterCtas * kClusterRowThreads / kLanes;  // rows of one pass
constexpr int64_t kClusterTwoPassEdges = 40000;  // rows of 16 bytes (up to 3 components) only

template <int KK>
__global__ void __launch_bounds__(kClusterThreads, 1)
    power_cluster_kernel(float* __restrict__ V0, float* __restrict__ V1, const int64_t* __restrict__ row_ptr,
                         const int32_t* __restrict__ cols, const float* __restrict__ wn, int n, int rows_per_cta,
                         int edge_cap, int n_iter, double* __restrict__ Rinv) {
  constexpr int vp = KK <= 4 ? 4 : 8;
  constexpr int kWarps = kClusterThreads / 32;
  extern __shared__ __align__(16) unsigned char power_smem[];
  float4* v_all = reinterpret_cast<float4*>(power_smem);  // two buffers of n rows
  const int v_words = n * (vp / 4);
  int32_t* s_off = reinterpret_cast<int32_t*>(v_all + 2 * v_words);  // rows_per_cta + 1 offsets from the first edge
  int32_t* s_col = s_off + rows_per_cta + 1;
  float* s_w = reinterpret_cast<float*>(s_col + edge_cap);
  __shared__ double ri[KK * KK];
  __shared__ double gsum[Upper<KK>::kEntries][kWarps];
  __shared__ double parts[2][kClusterCtas][KK * KK];  // the CTAs' Gram matrices, by parity of the iteration
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int sub = threadIdx.x & (kLanes - 1);
  const int rank = (int)cluster::rank();
  const int r_first = rank * rows_per_cta;
  const int rows = r_first < n ? (n - r_first < rows_per_cta ? n - r_first : rows_per_cta) : 0;
  const int64_t e_first = rows > 0 ? row_ptr[r_first] : 0;
  const int n_edges = rows > 0 ? (int)(row_ptr[r_first + rows] - e_first) : 0;
  const int staged = n_edges < edge_cap ? n_edges : edge_cap;
  for (int t = threadIdx.x; rows > 0 && t <= rows; t += kClusterThreads)
    s_off[t] = (int)(row_ptr[r_first + t] - e_first);
  for (int e = threadIdx.x; e < staged; e += kClusterThreads) {
    s_col[e] = cols[e_first + e];
    s_w[e] = wn[e_first + e];
  }
  for (int t = threadIdx.x; t < v_words; t += kClusterThreads) v_all[t] = reinterpret_cast<const float4*>(V0)[t];
  cols += e_first;
  wn += e_first;
  const uint32_t v_at = cluster::smem_address(v_all);
  const uint32_t parts_at = cluster::smem_address(parts);
  // every CTA runs and has read V0 before its neighbours store into its copy
  cluster::barrier();

  for (int it = 0; it <= n_iter; ++it) {
    // the factor warp: R^-1 of the previous iteration's product, for this one's rows
    if (warp == kWarps - 1 && it > 0) {
      const int t0 = lane < KK * KK ? lane : 0;
      double mine = 0.0;
      for (int p = 0; p < kClusterCtas; ++p) mine += parts[(it - 1) & 1][p][t0];
      double Gl[KK * KK], rl[KK * KK];
#pragma unroll
      for (int t = 0; t < KK * KK; ++t) Gl[t] = __shfl_sync(0xffffffffu, mine, t);  // the upper triangle counts
      chol_inverse_fixed<KK>(Gl, rl);
      if (lane == 0) {
#pragma unroll
        for (int t = 0; t < KK * KK; ++t) ri[t] = rl[t];
        if (rank == 0)
          for (int t = 0; t < KK * KK; ++t) Rinv[(size_t)(it - 1) * KK * KK + t] = rl[t];
      }
    }
    if (it == n_iter) break;
    const float4* Vin = v_all + (it & 1) * v_words;
    const uint32_t out_at = v_at + (uint32_t)(((it + 1) & 1) * v_words) * 16u;
    double part[KK * KK];
#pragma unroll
    for (int t = 0; t < KK * KK; ++t) part[t] = 0.0;
    bool first = true;  // every warp takes the first pass: R^-1 is ready after it
    for (int w0 = warp * (32 / kLanes); first || w0 < rows; w0 += kClusterRowThreads / kLanes) {
      const int lr = w0 + lane / kLanes;
      const bool valid = lr < rows && warp < kWarps - 1;
      double acc[KK];
#pragma unroll
      for (int j = 0; j < KK; ++j) acc[j] = 0.0;
      const int e1 = valid ? s_off[lr + 1] : 0;
      for (int e = valid ? s_off[lr] + sub : 0; e < e1; e += 4 * kLanes) {
        int c[4];
        float w[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const int x = e + u * kLanes;
          const bool on = x < e1;
          c[u] = on ? (x < staged ? s_col[x] : cols[x]) : 0;
          w[u] = on ? (x < staged ? s_w[x] : wn[x]) : 0.f;
        }
        float4 a[4];
        float a4[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          a[u] = Vin[c[u] * (vp / 4)];
          a4[u] = KK > 4 ? Vin[c[u] * (vp / 4) + vp / 4 - 1].x : 0.f;
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          if (e + u * kLanes >= e1) continue;
          const double wd = (double)w[u];
          const float v[5] = {a[u].x, a[u].y, a[u].z, a[u].w, a4[u]};
#pragma unroll
          for (int j = 0; j < KK; ++j) acc[j] += wd * (double)v[j];
        }
      }
#pragma unroll
      for (int j = 0; j < KK; ++j) acc[j] += __shfl_xor_sync(0xffffffffu, acc[j], 1);  // kLanes == 2
      if (first) __syncthreads();  // R^-1
      first = false;
      if (valid) {  // both lanes hold the sums: each stores the row into half of the copies
        double q[KK];
#pragma unroll
        for (int j = 0; j < KK; ++j) {
          q[j] = acc[j];
          if (it > 0) {
            q[j] = 0.0;
#pragma unroll
            for (int i = 0; i <= j; ++i) q[j] += acc[i] * ri[i * KK + j];
          }
        }
        float out[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) out[j] = j < KK ? (float)q[j < KK ? j : 0] : 0.f;
        const uint32_t at = out_at + (uint32_t)((r_first + lr) * (vp / 4)) * 16u;
#pragma unroll
        for (int p = 0; p < kClusterCtas / 2; ++p) {
          const uint32_t dst = cluster::peer(at, (uint32_t)(2 * p + sub));
          asm volatile("st.shared::cluster.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(dst), "f"(out[0]), "f"(out[1]),
                       "f"(out[2]), "f"(out[3])
                       : "memory");
          if constexpr (vp == 8)
            asm volatile("st.shared::cluster.v4.f32 [%0 + 16], {%1, %2, %3, %4};" ::"r"(dst), "f"(out[4]), "f"(out[5]),
                         "f"(out[6]), "f"(out[7])
                         : "memory");
        }
#pragma unroll
        for (int i = 0; i < KK; ++i)
#pragma unroll
          for (int j = i; j < KK; ++j) part[i * KK + j] += q[i] * q[j];
      }
    }
    const double gram = block_gram<KK, kWarps>(part, gsum);
    if (warp < Upper<KK>::kEntries && lane < kClusterCtas) {
      const uint32_t at = parts_at + (uint32_t)(((it & 1) * kClusterCtas + rank) * KK * KK + Upper<KK>::at(warp)) * 8u;
      asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(cluster::peer(at, (uint32_t)lane)), "d"(gram) : "memory");
    }
    __syncwarp();
    cluster::barrier();
  }
  float4* out = reinterpret_cast<float4*>((n_iter & 1) ? V1 : V0) + (int64_t)r_first * (vp / 4);
  const float4* mine = v_all + (n_iter & 1) * v_words + r_first * (vp / 4);
  for (int t = threadIdx.x; t < rows * (vp / 4); t += kClusterThreads) out[t] = mine[t];
}

// Enqueues the cluster form where it is the faster one; false: use another form.
template <int KK>
static bool launch_power_cluster(const int64_t* row_ptr, const int32_t* cols, const float* wn, int64_t e_cap,
                                 int64_t n, int n_iter, float* V0, float* V1, double* Rinv, cudaStream_t stream) {
  constexpr int vp = KK <= 4 ? 4 : 8;
  const bool one_pass = n <= kClusterPass;
  if (!one_pass && (KK > 4 || n > 2 * kClusterPass || e_cap > kClusterTwoPassEdges)) return false;
  const size_t v_bytes = 2 * (size_t)n * vp * sizeof(float);  // at most 128 KB
  const int per = (int)ceil_div(n, kClusterCtas);
  const size_t fixed = v_bytes + ((size_t)per + 1) * 4;
  // a CTA's share of the edges, and half as many again for uneven rows; the rest from L2
  int64_t cap = e_cap / kClusterCtas + e_cap / kClusterCtas / 2 + 64;
  const int64_t room = (int64_t)(kClusterSmem - fixed) / 8;
  if (one_pass && ceil_div(e_cap, kClusterCtas) > room) return false;
  if (cap > room) cap = room;
  const size_t smem = fixed + (size_t)cap * 8;
  {
    static std::mutex mu;
    static bool set[64] = {false};
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return false;
    std::lock_guard<std::mutex> lock(mu);
    if (!set[dev]) {
      if (cudaFuncSetAttribute(power_cluster_kernel<KK>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                               (int)kClusterSmem) != cudaSuccess) {
        cudaGetLastError();
        return false;
      }
      set[dev] = true;
    }
  }
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = kClusterCtas;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.gridDim = dim3(kClusterCtas, 1, 1);
  cfg.blockDim = dim3(kClusterThreads, 1, 1);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  if (cudaLaunchKernelEx(&cfg, power_cluster_kernel<KK>, V0, V1, row_ptr, cols, wn, (int)n, per, (int)cap, n_iter,
                         Rinv) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  return true;
}

__device__ __forceinline__ unsigned f2ord(float f) {
  const unsigned u = __float_as_uint(f);
  return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
__device__ __forceinline__ float ord2f(unsigned u) {
  return __uint_as_float((u & 0x80000000u) ? (u & 0x7fffffffu) : ~u);
}

// embedding = (V R^-1)[:, 1:], max |embedding|
__global__ void finish_orth_kernel(const float* __restrict__ V, const double* __restrict__ Rinv, int64_t n, int kk,
                                   int vp, float* __restrict__ emb, unsigned* __restrict__ absmax) {
  __shared__ double ri[kMaxCols * kMaxCols];
  if (threadIdx.x < kk * kk) ri[threadIdx.x] = Rinv[threadIdx.x];
  __syncthreads();
  const int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  float m = 0.f;
  if (r < n) {
    for (int j = 1; j < kk; ++j) {
      double q = 0.0;
      for (int i = 0; i <= j; ++i) q += (double)V[r * vp + i] * ri[i * kk + j];
      const float f = (float)q;
      emb[r * (kk - 1) + (j - 1)] = f;
      m = fmaxf(m, fabsf(f));
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
  if ((threadIdx.x & 31) == 0) atomicMax(absmax, __float_as_uint(m));
}

// e = f32(emb * (10 / max|emb|)) + noise (umap.py:344-346); per-column min/max: a thread
// per row, the block's extremes through shuffles and shared memory, then one atomic per
// column and block (one per element queued 105 us at 70,000 rows; now 2.6)
__global__ void __launch_bounds__(kBlock) scale_noise_kernel(float* __restrict__ emb, const float* __restrict__ noise,
                                                             int64_t n, int dim, const unsigned* __restrict__ absmax,
                                                             unsigned* __restrict__ colmin,
                                                             unsigned* __restrict__ colmax) {
  __shared__ unsigned s_lo[kBlock / 32], s_hi[kBlock / 32];
  const int64_t r = (int64_t)blockIdx.x * kBlock + threadIdx.x;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const float expansion = __fdiv_rn(10.0f, __uint_as_float(*absmax));
  for (int c = 0; c < dim; ++c) {
    unsigned lo = 0xffffffffu, hi = 0u;
    if (r < n) {
      const int64_t t = r * dim + c;
      const float v = __fadd_rn(__fmul_rn(emb[t], expansion), noise[t]);
      emb[t] = v;
      lo = hi = f2ord(v);
    }
    lo = __reduce_min_sync(0xffffffffu, lo);
    hi = __reduce_max_sync(0xffffffffu, hi);
    if (lane == 0) {
      s_lo[warp] = lo;
      s_hi[warp] = hi;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
      for (int w = 1; w < kBlock / 32; ++w) {
        lo = min(lo, s_lo[w]);
        hi = max(hi, s_hi[w]);
      }
      atomicMin(&colmin[c], lo);
      atomicMax(&colmax[c], hi);
    }
    __syncthreads();
  }
}

// Y = 10 (e - min) / (max - min + 1e-10) per column (umap.py:347)
__global__ void minmax_kernel(const float* __restrict__ emb, int64_t n, int dim, const unsigned* __restrict__ colmin,
                              const unsigned* __restrict__ colmax, float* __restrict__ Y) {
  const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= n * dim) return;
  const int c = (int)(t % dim);
  const float mn = ord2f(colmin[c]), mx = ord2f(colmax[c]);
  const float num = __fmul_rn(10.0f, __fsub_rn(emb[t], mn));
  const float den = __fadd_rn(__fsub_rn(mx, mn), 1e-10f);
  Y[t] = __fdiv_rn(num, den);
}

struct Layout {
  int32_t* status;
  int64_t* row_ptr;
  float* dis;
  float* wn;
  float* V[2];  // n rows of vp floats (kk values, zero padded to 4 or 8)
  double* G;       // n_iter blocks of kk*kk
  double* Rinv;    // n_iter blocks of kk*kk: the inverse Cholesky factor after each iteration
  unsigned* done;  // per-iteration block counters; done[n_iter] the grid barrier
  int* abort_g;    // cooperative path: barrier abort flag
  float* emb;
  unsigned* red;  // absmax, colmin[kWideCols], colmax[kWideCols]
  size_t bytes;
};

static int vpitch(int kk) { return kk <= 4 ? 4 : (kk + 3) / 4 * 4; }

static Layout carve(void* ws, int64_t n, int dim, int64_t e_cap, int n_iter) {
  const int kk = dim + 1;
  Carver c(ws);
  Layout l;
  l.status = c.take<int32_t>(64);
  // cleared with the status word by one memset
  l.abort_g = c.take<int>(1);
  l.done = c.take<unsigned>((size_t)(n_iter > 0 ? n_iter : 1) + 1);
  l.G = c.take<double>((size_t)(n_iter > 0 ? n_iter : 1) * kk * kk);
  l.Rinv = c.take<double>((size_t)(n_iter > 0 ? n_iter : 1) * kk * kk);
  l.row_ptr = c.take<int64_t>((size_t)n + 1);
  l.dis = c.take<float>((size_t)n);
  l.wn = c.take<float>((size_t)(e_cap > 0 ? e_cap : 1));
  l.V[0] = c.take<float>((size_t)n * vpitch(kk));
  l.V[1] = c.take<float>((size_t)n * vpitch(kk));
  l.emb = c.take<float>((size_t)n * dim);
  l.red = c.take<unsigned>(1 + 2 * kWideCols);
  l.bytes = c.bytes();
  return l;
}

// V0 (n x kk) into rows of vp floats, zero padded
__global__ void pad_rows_kernel(const float* __restrict__ a, int64_t n, int kk, int vp, float* __restrict__ b) {
  const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= n * vp) return;
  const int64_t r = t / vp;
  const int j = (int)(t - r * vp);
  b[t] = j < kk ? a[r * kk + j] : 0.f;
}

// Standard normal draws: element i of the stream (seed) comes from Philox block i/4
// and the Box-Muller transform of its two 32-bit pairs.
__device__ __forceinline__ void normal4(int64_t blk, uint32_t k0, uint32_t k1, float (&z)[4]) {
  const U4 r = philox4x32_10(U4{(uint32_t)blk, (uint32_t)(blk >> 32), 0x5eedu, 0u}, k0, k1);
  float s0, c0, s1, c1;
  const float r0 = sqrtf(-2.0f * logf(to_unit(r.x)));
  const float r1 = sqrtf(-2.0f * logf(to_unit(r.z)));
  sincospif(2.0f * to_unit(r.y), &s0, &c0);
  sincospif(2.0f * to_unit(r.w), &s1, &c1);
  z[0] = r0 * c0, z[1] = r0 * s0, z[2] = r1 * c1, z[3] = r1 * s1;
}

__global__ void normal_fill_kernel(float* __restrict__ out, int64_t count, uint32_t k0, uint32_t k1) {
  const int64_t blk = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (blk * 4 >= count) return;
  float z[4];
  normal4(blk, k0, k1, z);
  for (int u = 0; u < 4; ++u)
    if (blk * 4 + u < count) out[blk * 4 + u] = z[u];
}

__global__ void init_red_kernel(unsigned* red, int dim) {
  if (threadIdx.x == 0) red[0] = 0u;
  if (threadIdx.x < (unsigned)dim) {
    red[1 + threadIdx.x] = 0xFFFFFFFFu;          // min
    red[1 + kWideCols + threadIdx.x] = 0u;       // max
  }
}

// The reference falls back to a random start when its spectral init fails
// (umap.py:354-357).  When the power iteration's grid barrier gave up (status word
// non-zero), Y is replaced on the device by N(0, 1) * 0.01 drawn from the Philox
// stream of umapb_normal_fill(seed), so no host round trip sits between the
// spectral init and the layout.
__global__ void fallback_kernel(const int32_t* __restrict__ status, float* __restrict__ Y, int64_t count,
                                uint32_t k0, uint32_t k1) {
  if (*status == 0) return;
  const int64_t blk = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (blk * 4 >= count) return;
  float z[4];
  normal4(blk, k0, k1, z);
  for (int u = 0; u < 4; ++u)
    if (blk * 4 + u < count) Y[blk * 4 + u] = __fmul_rn(z[u], 0.01f);
}

}  // namespace spectral
}  // namespace umapb

using namespace umapb;

extern "C" int umapb_spectral_workspace(int64_t n, int32_t dim, int64_t e_cap, int32_t n_iter, size_t* bytes) {
  clear_error();
  UMAPB_REQUIRE(bytes, "bytes is null");
  UMAPB_REQUIRE(n >= 1 && dim >= 1 && dim <= 32, "spectral: need n >= 1 and 1 <= dim <= 32");
  UMAPB_REQUIRE(n_iter >= 1 && n_iter <= 128, "spectral: need 1 <= n_iter <= 128");
  UMAPB_REQUIRE(e_cap >= 0, "spectral: e_cap must be >= 0");
  *bytes = spectral::carve(nullptr, n, dim, e_cap, n_iter).bytes;
  return UMAPB_OK;
}

extern "C" int umapb_spectral(const int32_t* rows, const int32_t* cols, const float* vals, const int64_t* n_edges,
                              int64_t e_cap, int64_t n, int32_t dim, const float* V0, int32_t n_iter,
                              const float* noise, float* Y, void* workspace, size_t workspace_bytes,
                              umapb_stream_t stream_) {
  clear_error();
  cudaStream_t stream = reinterpret_cast<cudaStream_t>(stream_);
  UMAPB_REQUIRE(rows && cols && vals && n_edges && V0 && noise && Y, "spectral: null array argument");
  UMAPB_REQUIRE(n >= 1 && dim >= 1 && dim <= 32, "spectral: need n >= 1 and 1 <= dim <= 32");
  UMAPB_REQUIRE(n_iter >= 1 && n_iter <= 128, "spectral: need 1 <= n_iter <= 128");
  UMAPB_REQUIRE(e_cap >= 0, "spectral: e_cap must be >= 0");
  spectral::Layout l = spectral::carve(nullptr, n, dim, e_cap, n_iter);
  if (!workspace || workspace_bytes < l.bytes)
    return set_error(UMAPB_ERR_WORKSPACE, "spectral: workspace of %zu bytes, need %zu", workspace_bytes, l.bytes);
  l = spectral::carve(workspace, n, dim, e_cap, n_iter);
  const int kk = dim + 1;
  const unsigned rb = (unsigned)ceil_div(n, spectral::kBlock);
  UMAPB_CUDA_TRY(cudaMemsetAsync(l.status, 0, reinterpret_cast<char*>(l.Rinv) - reinterpret_cast<char*>(l.status),
                                 stream),
                 "spectral: status, counter and gram reset");
  spectral::row_ptr_kernel<<<(unsigned)ceil_div(n + 1, spectral::kBlock), spectral::kBlock, 0, stream>>>(
      rows, n_edges, n, l.row_ptr);
  spectral::degree_kernel<<<rb, spectral::kBlock, 0, stream>>>(vals, l.row_ptr, n, l.dis);
  if (e_cap > 0)
    spectral::norm_weight_kernel<<<(unsigned)ceil_div(e_cap, spectral::kBlock), spectral::kBlock, 0, stream>>>(
        rows, cols, vals, n_edges, l.dis, l.wn);
  const int vp = spectral::vpitch(kk);
  spectral::pad_rows_kernel<<<(unsigned)ceil_div(n * vp, spectral::kBlock), spectral::kBlock, 0, stream>>>(
      V0, n, kk, vp, l.V[0]);
  UMAPB_LAUNCH_CHECK("spectral: setup kernels");
  const unsigned pb = (unsigned)ceil_div(n * spectral::kLanes, spectral::kBlock);
  // one cooperative launch for all iterations, one resident block per SM, fewer when that
  // would leave a block little to do (a smaller barrier); the
  // per-iteration launches remain for devices that refuse it and behind
  // UMAPB_SPECTRAL_COOP=0
  int coop = 0, dev = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev);
  {
    const char* e = getenv("UMAPB_SPECTRAL_COOP");
    if (e && e[0] == '0' && e[1] == 0) coop = 0;
  }
  bool launched = false;
  const bool wide = kk > spectral::kMaxCols;
  if (wide) coop = 0;
  if (coop) {  // few rows: one cluster
    const auto f = kk == 2   ? spectral::launch_power_cluster<2>
                   : kk == 3 ? spectral::launch_power_cluster<3>
                   : kk == 4 ? spectral::launch_power_cluster<4>
                             : spectral::launch_power_cluster<5>;
    launched = f(l.row_ptr, cols, l.wn, e_cap, n, n_iter, l.V[0], l.V[1], l.Rinv, stream);
  }
  if (coop && !launched) {
    const void* pk = kk == 2   ? (const void*)spectral::power_kernel<2>
                     : kk == 3 ? (const void*)spectral::power_kernel<3>
                     : kk == 4 ? (const void*)spectral::power_kernel<4>
                               : (const void*)spectral::power_kernel<5>;
    // A block for every 248 rows (half a pass; 124 of the wider rows, whose FP64 arithmetic is
    // longer) and for every 2,048 edges, which an SM gathers in about a microsecond: by rows alone a
    // few SMs had all edges of a wide neighbourhood.  100 iterations, 2 components, by
    // rows alone and now: 5,121 rows, k = 50 1007 -> 744 us, k = 100 2610 -> 1084; 20,000 rows, k = 50
    // 1039 -> 853; 10,000 rows, k = 15 554 -> 503; 4 components, 10,000 rows, k = 10 898 -> 760.  The last
    // third of the SMs is for 4,096 edges a block: 20,000 rows, k = 15, 3 components 638 us at 81 blocks,
    // 628 at 98, 663 at 147; k = 30 841, 806 at 147.
    const int64_t min_rows = spectral::kPowerRowThreads / spectral::kLanes / (kk > 4 ? 4 : 2);
    int64_t grid = ceil_div(n, min_rows);
    int64_t by_edges = ceil_div(e_cap, 2048);
    if (by_edges > num_sms() * 2 / 3) {
      by_edges = num_sms() * 2 / 3;
      if (ceil_div(e_cap, 4096) > by_edges) by_edges = ceil_div(e_cap, 4096);
    }
    if (by_edges > grid) grid = by_edges;
    if (grid > ceil_div(n, 16)) grid = ceil_div(n, 16);  // a warp's rows at least
    if (grid > num_sms()) grid = num_sms();
    int per = (int)ceil_div(n, grid);
    grid = ceil_div(n, per);
    int off_cap = (size_t)per < spectral::kPowerSmem / 8 ? per + 1 : 0;  // more rows: offsets from L2
    const size_t off_bytes = (size_t)off_cap * 4;
    // the block's share of the edges, and half as many again for uneven rows
    int64_t cap = e_cap / grid + e_cap / grid / 2 + 64;
    const int64_t room = (int64_t)(spectral::kPowerSmem - off_bytes) / 8;
    // A share that does not fit stays in L2, all of it, and L1 keeps its size: staging the part that
    // fits took the start of 1,000,000 rows from 10.3 to 16.6 ms; without, graph and start of
    // 1,000,000 rows 11.9 -> 9.2 ms, 300,000 3.8 -> 2.9, against the form before.
    if (cap > room) cap = e_cap / grid > room ? 0 : room;
    const size_t smem = off_bytes + (size_t)cap * 8;
    int edge_cap = (int)cap;
    int per_sm = 0;
    if (smem <= spectral::kPowerSmem &&
        cudaFuncSetAttribute(pk, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)spectral::kPowerSmem) ==
            cudaSuccess &&
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, pk, spectral::kPowerThreads, smem) == cudaSuccess &&
        per_sm > 0) {
      float* v0 = l.V[0];
      float* v1 = l.V[1];
      const int64_t* rp = l.row_ptr;
      const float* w = l.wn;
      int64_t nn = n;
      int ni = n_iter;
      double* G = l.G;
      double* R = l.Rinv;
      unsigned* bar = l.done + n_iter;
      int* ab = l.abort_g;
      int32_t* st = l.status;
      unsigned long long lim = wait_limit_ns();
      void* args[] = {&v0, &v1, &rp, &cols, &w, &nn, &per, &off_cap, &edge_cap, &ni, &G, &R, &bar, &ab, &st, &lim};
      launched = cudaLaunchCooperativeKernel(pk, dim3((unsigned)grid), dim3(spectral::kPowerThreads), args, smem,
                                             stream) == cudaSuccess;
    }
    if (!launched) cudaGetLastError();
  }
  if (!launched && wide) {
    const unsigned wb = (unsigned)ceil_div(n, spectral::kWideRows);
    for (int it = 0; it < n_iter; ++it) {
      const double* rprev = it == 0 ? nullptr : l.Rinv + (size_t)(it - 1) * kk * kk;
      spectral::spmv_gram_wide_kernel<<<wb, spectral::kBlock, 0, stream>>>(
          l.V[it & 1], rprev, l.row_ptr, cols, l.wn, n, kk, vp, l.V[(it + 1) & 1], l.G + (size_t)it * kk * kk,
          l.done + it, l.Rinv + (size_t)it * kk * kk);
    }
  } else if (!launched) {
    for (int it = 0; it < n_iter; ++it) {
      const double* rprev = it == 0 ? nullptr : l.Rinv + (size_t)(it - 1) * kk * kk;
      spectral::spmv_gram_kernel<<<pb, spectral::kBlock, 0, stream>>>(
          l.V[it & 1], rprev, l.row_ptr, cols, l.wn, n, kk, vp, l.V[(it + 1) & 1], l.G + (size_t)it * kk * kk,
          l.done + it, l.Rinv + (size_t)it * kk * kk);
    }
  }
  UMAPB_LAUNCH_CHECK("spectral: power iteration");
  spectral::init_red_kernel<<<1, 32, 0, stream>>>(l.red, dim);
  if (wide)
    spectral::finish_orth_wide_kernel<<<(unsigned)ceil_div(n, spectral::kBlock / 32), spectral::kBlock, 0, stream>>>(
        l.V[n_iter & 1], l.Rinv + (size_t)(n_iter - 1) * kk * kk, n, kk, vp, l.emb, l.red);
  else
    spectral::finish_orth_kernel<<<rb, spectral::kBlock, 0, stream>>>(l.V[n_iter & 1],
                                                                       l.Rinv + (size_t)(n_iter - 1) * kk * kk, n,
                                                                       kk, vp, l.emb, l.red);
  const unsigned eb = (unsigned)ceil_div(n * dim, spectral::kBlock);
  unsigned* colmin = l.red + 1;
  unsigned* colmax = l.red + 1 + spectral::kWideCols;
  spectral::scale_noise_kernel<<<rb, spectral::kBlock, 0, stream>>>(l.emb, noise, n, dim, l.red, colmin, colmax);
  spectral::minmax_kernel<<<eb, spectral::kBlock, 0, stream>>>(l.emb, n, dim, colmin, colmax, Y);
  UMAPB_LAUNCH_CHECK("spectral: rescale kernels");
  count_launches((e_cap > 0 ? 3 : 2) + 1 + (launched ? 1 : n_iter) + 4);
  return UMAPB_OK;
}

extern "C" int umapb_spectral_fallback(const void* workspace, float* Y, int64_t n, int32_t dim, uint64_t seed,
                                       umapb_stream_t stream_) {
  clear_error();
  UMAPB_REQUIRE(workspace && Y, "spectral_fallback: null argument");
  UMAPB_REQUIRE(n >= 1 && dim >= 1 && dim <= 32, "spectral_fallback: need n >= 1 and 1 <= dim <= 32");
  const int64_t count = n * dim;
  const int64_t blocks4 = ceil_div(count, 4);
  spectral::fallback_kernel<<<(unsigned)ceil_div(blocks4, 256), 256, 0, reinterpret_cast<cudaStream_t>(stream_)>>>(
      static_cast<const int32_t*>(workspace), Y, count, (uint32_t)seed, (uint32_t)(seed >> 32));
  UMAPB_LAUNCH_CHECK("spectral_fallback kernel");
  count_launches(1);
  return UMAPB_OK;
}

extern "C" int umapb_normal_fill(float* out, int64_t count, uint64_t seed, umapb_stream_t stream_) {
  clear_error();
  UMAPB_REQUIRE(out || count == 0, "normal_fill: null output");
  UMAPB_REQUIRE(count >= 0, "normal_fill: count must be >= 0");
  if (count == 0) return UMAPB_OK;
  const int64_t blocks4 = ceil_div(count, 4);
  spectral::normal_fill_kernel<<<(unsigned)ceil_div(blocks4, 256), 256, 0, reinterpret_cast<cudaStream_t>(stream_)>>>(
      out, count, (uint32_t)seed, (uint32_t)(seed >> 32));
  UMAPB_LAUNCH_CHECK("normal_fill kernel");
  count_launches(1);
  return UMAPB_OK;
}
