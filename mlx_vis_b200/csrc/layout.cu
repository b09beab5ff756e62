// Layout optimisation — replaces UMAP._optimize and UMAP._sgd_step,
// mlx_vis/_umap/umap.py:359-449.
//
// Schedule (umap.py:398-414): eps_e = n_epochs / (n_epochs * (w_e / max w)) in
// float32, next_e starts at eps_e; edge e is active in epoch t when
// next_e <= t, after which next_e += eps_e (float32).  The reference builds all
// active sets on the host up front; here every epoch kernel re-evaluates the
// same float32 recurrence per edge, so the sets are identical and no host work
// or per-epoch index list is needed.
//
// Epoch (umap.py:359-387): every gather reads the epoch-start Y; the moves of
// all pairs are accumulated into dY with float atomics and applied by a second
// kernel (few rows: after a barrier of one kernel), which reproduces the reference's synchronous scatter-add semantics.
// Per active edge (i, j): attractive move clip(-2ab d^{2(b-1)}/(1+a d^{2b}) diff,
// +-4) * alpha added to i and subtracted from j; neg_rate negatives (i, t) each
// add clip(2b/((0.001+d^2)(1+a d^{2b})) diff, +-4) * alpha to i only.  The moves
// of one edge on its head are summed in registers before one atomic.
//
// Negatives: the reference pairs sample s of an epoch with head ef[s % A] and a
// uniform tail from mx.random.randint (umap.py:433-436).  The fast path draws
// the tail of (epoch, edge e, sample m) from Philox4x32-10 (Salmon et al., SC'11)
// keyed by the seed, mapped to [0, n) by a 32x32->64 multiply-high (bias below
// n / 2^32).  The injected path takes the reference's own tails: it ranks the
// active edges in edge order (block counts + scan) and uses tail neg_to[r + m A]
// for the r-th active edge.
#include <math.h>
#include <stdlib.h>
#include <string.h>

#include <mutex>

#include "cluster.cuh"
#include "common.cuh"
#include "philox.cuh"
#include "scan.cuh"

namespace umapb {
namespace layout {

constexpr int kBlock = 256;
constexpr int kEdgesPerBlock = 1024;
constexpr size_t kClusterSmem = 216 * 1024;

// one launch for all epochs: row ids of 16 bits, a copy of Y in one SM's shared memory
static bool resident_rows(int64_t n, int dim) {
  return dim <= 4 && n < 65536 && 4 * n * dim + 64 <= (int64_t)kClusterSmem;
}
#ifndef UMAPB_LAYOUT_BLOCKS_PER_SM
#define UMAPB_LAYOUT_BLOCKS_PER_SM 4
#endif
// resident blocks per SM the epoch kernel is compiled for (register cap) and launched with
constexpr int kEpochBlocksPerSM = UMAPB_LAYOUT_BLOCKS_PER_SM;
#ifndef UMAPB_LAYOUT_BLOCKS_PER_SM5
#define UMAPB_LAYOUT_BLOCKS_PER_SM5 4
#endif
// the same for the kernel specialised to 5 negatives per edge (the default rate)
constexpr int kEpochBlocksPerSM5 = UMAPB_LAYOUT_BLOCKS_PER_SM5;
constexpr int kPreMin = 5, kPreMax = 8;  // epoch kernel: chunks of 32 edges whose schedule words load together

// ---- reference pair math (float32, evaluation order of umap.py:361-383) ----
struct Params {
  float a, b, m2ab, two_b, alpha;
};

// d^(2b) is evaluated once per pair as exp2(b log2 d2) (CUDA's log2f / exp2f, a few
// ulp); d^(2(b-1)) = d^(2b) / d2.  The reference evaluates mx.power twice in float32;
// the difference is a few float32 ulp of the coefficient.
__device__ __forceinline__ float pow_b(float d2, float b) { return exp2f(__fmul_rn(b, log2f(d2))); }

template <int DIM>
__device__ __forceinline__ void attract(const float (&yi)[DIM], const float (&yj)[DIM], const Params& p,
                                        float (&out)[DIM]) {
  float diff[DIM];
  float d2 = 0.f;
#pragma unroll
  for (int c = 0; c < DIM; ++c) {
    diff[c] = __fsub_rn(yi[c], yj[c]);
    d2 = __fadd_rn(d2, __fmul_rn(diff[c], diff[c]));
  }
  d2 = fmaxf(d2, 1e-6f);
  const float pw = pow_b(d2, p.b);
  // -2ab d^(2(b-1)) / (1 + a d^(2b)) = (-2ab) d^(2b) / (d2 (1 + a d^(2b)))
  const float coeff = __fdiv_rn(__fmul_rn(p.m2ab, pw), __fmul_rn(d2, __fadd_rn(1.0f, __fmul_rn(p.a, pw))));
#pragma unroll
  for (int c = 0; c < DIM; ++c) out[c] = __fmul_rn(fminf(fmaxf(__fmul_rn(coeff, diff[c]), -4.0f), 4.0f), p.alpha);
}

template <int DIM>
__device__ __forceinline__ void repel_add(const float (&yi)[DIM], const float (&yt)[DIM], const Params& p,
                                          float (&acc)[DIM]) {
  float diff[DIM];
  float d2 = 0.f;
#pragma unroll
  for (int c = 0; c < DIM; ++c) {
    diff[c] = __fsub_rn(yi[c], yt[c]);
    d2 = __fadd_rn(d2, __fmul_rn(diff[c], diff[c]));
  }
  d2 = fmaxf(d2, 1e-6f);
  const float pw = pow_b(d2, p.b);
  const float den = __fmul_rn(__fadd_rn(0.001f, d2), __fadd_rn(1.0f, __fmul_rn(p.a, pw)));
  const float coeff = __fdiv_rn(p.two_b, den);
#pragma unroll
  for (int c = 0; c < DIM; ++c)
    acc[c] = __fadd_rn(acc[c], __fmul_rn(fminf(fmaxf(__fmul_rn(coeff, diff[c]), -4.0f), 4.0f), p.alpha));
}

// coherent loads: Y may have been written by a grid that this one has waited for
template <int DIM>
__device__ __forceinline__ void load_row(const float* Y, int i, float (&v)[DIM]) {
  if constexpr (DIM == 2) {
    const float2 t = reinterpret_cast<const float2*>(Y)[i];
    v[0] = t.x;
    v[1] = t.y;
  } else if constexpr (DIM == 4) {
    const float4 t = reinterpret_cast<const float4*>(Y)[i];
    v[0] = t.x;
    v[1] = t.y;
    v[2] = t.z;
    v[3] = t.w;
  } else {
#pragma unroll
    for (int c = 0; c < DIM; ++c) v[c] = Y[(int64_t)i * DIM + c];
  }
}

// Programmatic dependent launch: the next grid of the stream may start once every block of this
// one has called next_may_start() or ended; await_previous() returns when the grid before has
// ended and its writes are visible (no fence: one more per block costs 2 us an epoch).
// Without the launch attribute neither does anything.
__device__ __forceinline__ void next_may_start() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void await_previous() {
  asm volatile("griddepcontrol.wait;" ::: "memory");
}

template <int DIM>
__device__ __forceinline__ void atomic_add_row(float* __restrict__ dY, int i, const float (&v)[DIM]) {
  if constexpr (DIM == 2) {
    atomicAdd(reinterpret_cast<float2*>(dY) + i, make_float2(v[0], v[1]));
  } else if constexpr (DIM == 4) {
    atomicAdd(reinterpret_cast<float4*>(dY) + i, make_float4(v[0], v[1], v[2], v[3]));
  } else {
#pragma unroll
    for (int c = 0; c < DIM; ++c) atomicAdd(dY + (int64_t)i * DIM + c, v[c]);
  }
}

// ---- schedule ----------------------------------------------------------------
__global__ void max_kernel(const float* __restrict__ vals, const int64_t* __restrict__ n_edges, float* __restrict__ wmax) {
  const int64_t E = *n_edges;
  float m = 0.f;
  for (int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < E; e += (int64_t)gridDim.x * blockDim.x)
    m = fmaxf(m, vals[e]);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
  if ((threadIdx.x & 31) == 0) atomicMax(reinterpret_cast<int*>(wmax), __float_as_int(m));
}

__global__ void eps_kernel(const float* __restrict__ vals, const int64_t* __restrict__ n_edges,
                           const float* __restrict__ wmax, int n_epochs, float* __restrict__ eps,
                           float* __restrict__ next) {
  const int64_t E = *n_edges;
  const float wm = *wmax;
  const float ne = (float)n_epochs;
  for (int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < E; e += (int64_t)gridDim.x * blockDim.x) {
    const float ns = __fmul_rn(ne, __fdiv_rn(vals[e], wm));
    const float v = ns > 0.f ? __fdiv_rn(ne, ns) : -1.0f;
    eps[e] = v;
    next[e] = v;
  }
}

// ---- fast path epoch ---------------------------------------------------------
// Only the edges due in an epoch do work, about a third of them on average, so a
// thread-per-edge loop leaves most lanes idle.  Each warp scans a contiguous
// segment of edges, advances the schedule of the due ones and queues them in
// shared memory; the warps work through the queue 32 edges at a time with every
// lane busy (at most one partial batch per block and pass).
//
// Two grids an epoch, this one and the apply.  Each is launched to overlap the one before:
// the apply's blocks start as the epoch's end, and the next epoch scans its first pass
// while the apply runs, so that neither launch gap nor the scan's round trip is on the
// chain.  What bounds it: the random 8-byte accesses (the two ends, five negatives, two sums
// per due edge, 290 G/s measured), then the scan of the schedule.  B200, per epoch, k = 15,
// 5 negatives, dim 2: 30,000 points 11.1 -> 10.2 us, 70,000 20.6 -> 19.8, 200,000 51.4 -> 50.0; the
// graph of 70,000 images over 500 epochs 16.8 -> 16.2.  (The apply let in from the epoch's start:
// 0.6 to 1.3 us more.  Passes of 4 chunks gain 0.4 us at most and lose 0.8 on the images' graph.)
// NEG > 0: compiled for exactly NEG (<= 8) negatives per edge (neg_rate == NEG), so
// the registers of the unused sample slots are not held.
template <int DIM, int NEG>
__device__ __forceinline__ void edge_update(const float* Y, float* __restrict__ dY, int n, int i,
                                            int j, int64_t e, int epoch, const Params& p, int neg_rate, uint32_t k0,
                                            uint32_t k1) {
  static_assert(NEG >= 0 && NEG <= 8, "NEG is 0 (any rate) or a rate <= 8");
  float yi[DIM], yj[DIM], acc[DIM], pos[DIM], neg_pos[DIM];
  constexpr int kSlots = NEG > 0 ? NEG : 8;
  const int nr = NEG > 0 ? NEG : neg_rate;
  if (NEG > 0 || neg_rate <= 8) {
    // up to 8 negatives: draw their tails and issue every gather of Y before the
    // arithmetic, so the seven or so random reads of an edge are in flight together
    const U4 r0 = philox4x32_10(U4{(uint32_t)e, (uint32_t)(e >> 32), (uint32_t)epoch, 0u}, k0, k1);
    U4 r1 = r0;
    if (nr > 4) r1 = philox4x32_10(U4{(uint32_t)e, (uint32_t)(e >> 32), (uint32_t)epoch, 1u}, k0, k1);
    const uint32_t rr[8] = {r0.x, r0.y, r0.z, r0.w, r1.x, r1.y, r1.z, r1.w};
    float yt[kSlots][DIM];
    load_row<DIM>(Y, i, yi);
    load_row<DIM>(Y, j, yj);
#pragma unroll
    for (int u = 0; u < kSlots; ++u)
      if (u < nr) load_row<DIM>(Y, to_range(rr[u], (uint32_t)n), yt[u]);
    attract<DIM>(yi, yj, p, pos);
#pragma unroll
    for (int c = 0; c < DIM; ++c) {
      acc[c] = pos[c];
      neg_pos[c] = -pos[c];
    }
#pragma unroll
    for (int u = 0; u < kSlots; ++u)
      if (u < nr) repel_add<DIM>(yi, yt[u], p, acc);
    atomic_add_row<DIM>(dY, j, neg_pos);
    atomic_add_row<DIM>(dY, i, acc);
    return;
  }
  load_row<DIM>(Y, i, yi);
  load_row<DIM>(Y, j, yj);
  attract<DIM>(yi, yj, p, pos);
#pragma unroll
  for (int c = 0; c < DIM; ++c) {
    acc[c] = pos[c];
    neg_pos[c] = -pos[c];
  }
  atomic_add_row<DIM>(dY, j, neg_pos);
  auto repel = [&](uint32_t r) {
    float yt[DIM];
    load_row<DIM>(Y, to_range(r, (uint32_t)n), yt);
    repel_add<DIM>(yi, yt, p, acc);
  };
#pragma unroll 1
  for (int m0 = 0; m0 < neg_rate; m0 += 4) {
    const U4 r = philox4x32_10(U4{(uint32_t)e, (uint32_t)(e >> 32), (uint32_t)epoch, (uint32_t)(m0 >> 2)}, k0, k1);
    repel(r.x);
    if (m0 + 1 < neg_rate) repel(r.y);
    if (m0 + 2 < neg_rate) repel(r.z);
    if (m0 + 3 < neg_rate) repel(r.w);
  }
  atomic_add_row<DIM>(dY, i, acc);
}

template <int DIM, int NEG, int kPre>
__global__ void __launch_bounds__(kBlock, NEG == 5 ? kEpochBlocksPerSM5 : kEpochBlocksPerSM) sgd_epoch_kernel(const float* Y, float* __restrict__ dY, int n,
                                                           const int32_t* __restrict__ rows,
                                                           const int32_t* __restrict__ cols,
                                                           const float* __restrict__ eps, float* __restrict__ next,
                                                           const int64_t* __restrict__ n_edges, int epoch, Params p,
                                                           int neg_rate, uint32_t k0, uint32_t k1) {
  // A pass: every warp loads the schedule words of kPre chunks of 32 edges of its
  // segment at once (one round trip instead of kPre), advances the due edges and
  // appends them to the block's queue; then the block's 8 warps take the queue 32
  // edges at a time, so only the block's last batch of the pass runs partly empty.
  static_assert(kPre * 32 <= 4096, "an edge of a warp's pass has 12 bits in the queue");
  __shared__ uint16_t bq[(kBlock / 32) * kPre * 32];  // warp << 12 | edge of the warp's pass
  __shared__ int s_cnt;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t E = *n_edges;
  const float ep = (float)epoch;
  const int64_t n_warps = (int64_t)gridDim.x * (kBlock / 32);
  const int64_t seg = (((E + 31) / 32 + n_warps - 1) / n_warps) * 32;
  const int64_t b0 = (int64_t)blockIdx.x * (kBlock / 32) * seg;
  const int64_t e0 = b0 + (int64_t)warp * seg;
  const int64_t e1 = e0 + seg < E ? e0 + seg : E;
  const unsigned below = (1u << lane) - 1u;
  // the same for every warp of the grid
  const int passes = (int)((seg + 32 * kPre - 1) / (32 * kPre));
  for (int ps = 0; ps < passes; ++ps) {
    if (threadIdx.x == 0) s_cnt = 0;
    __syncthreads();
    const int64_t done = (int64_t)ps * 32 * kPre, sb = e0 + done;
    float nx[kPre], ex[kPre];
#pragma unroll
    for (int u = 0; u < kPre; ++u) {
      const int64_t e = sb + 32 * u + lane;
      nx[u] = e < e1 ? __ldcg(next + e) : INFINITY;  // through L2: the epoch before wrote it
      ex[u] = e < e1 ? eps[e] : 0.f;
    }
#pragma unroll
    for (int u = 0; u < kPre; ++u) {
      const int64_t e = sb + 32 * u + lane;
      const bool due = nx[u] <= ep;
      if (due) next[e] = __fadd_rn(nx[u], ex[u]);
      const unsigned b = __ballot_sync(0xffffffffu, due);
      int slot = 0;
      if (lane == 0 && b) slot = atomicAdd(&s_cnt, __popc(b));
      slot = __shfl_sync(0xffffffffu, slot, 0);
      if (due) bq[slot + __popc(b & below)] = (uint16_t)(warp << 12 | 32 * u | lane);
    }
    __syncthreads();
    // the warp's batches: the head and tail ids of the next batch load while this
    // batch's rows of Y are gathered, one round trip per batch instead of two
    const int total = s_cnt;
    int base = warp * 32;
    auto edge = [&](int q) { return b0 + done + (int64_t)(bq[q] >> 12) * seg + (bq[q] & 4095); };
    int64_t e = 0;
    int i = 0, j = 0;
    if (base + lane < total) {
      e = edge(base + lane);
      i = rows[e];
      j = cols[e];
    }
    if (ps == 0) await_previous();  // from here on Y and dY
    for (; base < total; base += kBlock) {
      const int nb = base + kBlock;
      int64_t e2 = 0;
      int i2 = 0, j2 = 0;
      if (nb + lane < total) {
        e2 = edge(nb + lane);
        i2 = rows[e2];
        j2 = cols[e2];
      }
      if (base + lane < total) edge_update<DIM, NEG>(Y, dY, n, i, j, e, epoch, p, neg_rate, k0, k1);
      e = e2;
      i = i2;
      j = j2;
    }
    __syncthreads();
  }
  if (passes == 0) await_previous();  // a grid ends after the one before it
  next_may_start();  // here and not at the start: the apply's waiting blocks would take issue slots
}

// The next epoch's grid starts while this one runs: the epoch whose schedule it reads has ended.
__global__ void apply_kernel(float* Y, float* dY, int64_t m) {
  await_previous();
  next_may_start();
  const int64_t first = (int64_t)blockIdx.x * blockDim.x + threadIdx.x, step = (int64_t)gridDim.x * blockDim.x;
  const int64_t m4 = (reinterpret_cast<uintptr_t>(Y) | reinterpret_cast<uintptr_t>(dY)) % 16 == 0 ? m / 4 : 0;
  float4 *Y4 = reinterpret_cast<float4*>(Y), *dY4 = reinterpret_cast<float4*>(dY);
  for (int64_t t = first; t < m4; t += step) {
    float4 y = __ldcg(Y4 + t);
    const float4 d = __ldcg(dY4 + t);
    y.x = __fadd_rn(y.x, d.x);
    y.y = __fadd_rn(y.y, d.y);
    y.z = __fadd_rn(y.z, d.z);
    y.w = __fadd_rn(y.w, d.w);
    Y4[t] = y;
    dY4[t] = make_float4(0.f, 0.f, 0.f, 0.f);
  }
  for (int64_t t = 4 * m4 + first; t < m; t += step) {
    Y[t] = __fadd_rn(__ldcg(Y + t), __ldcg(dY + t));
    dY[t] = 0.f;
  }
}

// ---- few rows: all epochs in one launch ------------------------------------------
// Two launches per epoch cost more than the work of a few thousand due edges (6.7 to 8.3 us an
// epoch from 2,000 to 10,000 points, most of it launches and L2 round trips).  Here every CTA
// keeps a copy of Y and an equal share of the edges (schedule, ids) in shared memory for
// all epochs.  An epoch is: queue the due edges; gather from the own copy of Y, add the moves to
// dY in L2; barrier; every CTA adds all of dY to its copy.  dY is one of three arrays
// in turn: while an epoch adds to one, a CTA may still be reading the previous one, and the
// next one, which every CTA has read before the last barrier, is cleared.  The draws and
// the pair math are those of the launches.
// Up to kClusterEdges edges the CTAs are one cluster of 16 and the barrier is the
// cluster's; beyond, a resident grid with a barrier in L2 (bounded by umapb_set_wait_limit_ns,
// then the status word), since the pair math of more edges wants more SMs.  Either form needs Y
// and the share in one SM's shared memory (about 22,000 rows of two components).
// Y and the schedule are written at the end only, and a barrier that gives up gives up for every
// CTA, so after an expired wait both are as they were before the launch.
// B200, per epoch, overlapping launches and one: 600 points, k = 5 8.3 and 3.7 us (4.1 as a grid);
// 1,000, k = 12 7.5 and 4.2 (either way); 2,000, k = 15 6.6 and 4.3 (5.3 as a cluster); 9,999, k = 10 8.5
// and 6.0; 10,000, k = 100 10.8 and 8.7; 20,000, k = 5 9.6 and 7.6, k = 15 9.0 either way, k = 28 at 0 / 5 /
// 10 negatives 8.5 / 11.3 / 16.6 and 9.1 / 10.7 / 13.6; 12,500, k = 24, 3 components 13.0 and 10.7; 9,500, k =
// 40, 4 components 9.3 and 8.9: what fits is at worst a few percent slower than the launches.
// (Moves added in the owners' shared memory took 23 us an epoch: float adds there are
// compare-and-swap loops, remote ones a round trip a try.  Owners that apply their rows and
// store them into all copies need a second barrier: 6.3 us.)
constexpr int kClusterThreads = 1024;
constexpr int kClusterMax = 16;             // CTAs; 8 where 16 cannot be scheduled together
constexpr int64_t kClusterEdges = 12288;

struct ClusterArgs {
  float *Y, *dY;  // dY: three arrays of n * DIM
  const int32_t *rows, *cols;
  const float* eps;
  float* next;
  const int64_t* n_edges;
  int n, epoch_begin, epoch_end, n_epochs, neg_rate;
  int rows_per;  // rows that a CTA owns
  int cap;       // edges per CTA
  float a, b, m2ab, two_b, lr;
  uint32_t k0, k1;
  unsigned* bar;  // grid form: barrier counter, zero at launch; kGaveUp once a wait has expired
  int32_t* status;
  unsigned long long limit_ns;
};

constexpr unsigned kGaveUp = 1u << 31;

__device__ __forceinline__ unsigned long long gtimer() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

// Barrier of the resident grid; false once a wait at it has lasted limit_ns.  The counter itself
// carries the failure: a CTA whose time is up sets kGaveUp by compare-and-swap while
// the count is short of the target, and a CTA passes on a count without it.  So either every CTA
// passes a barrier or none does.
__device__ __forceinline__ bool grid_barrier(const ClusterArgs& a, unsigned target) {
  __shared__ int s_ok;
  __syncthreads();
  if (threadIdx.x == 0) {
    // the block's writes are ordered before this by the block barrier
    asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(a.bar) : "memory");
    const unsigned long long t0 = gtimer();
    unsigned v;
    while (true) {
      asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(a.bar) : "memory");
      if (v >= target) break;  // kGaveUp is above every target
      if (gtimer() - t0 > a.limit_ns) {
        while (v < target) {  // ends: the count has moved on whenever the swap fails
          unsigned was;
          asm volatile("atom.acquire.gpu.global.cas.b32 %0, [%1], %2, %3;"
                       : "=r"(was)
                       : "l"(a.bar), "r"(v), "r"(v | kGaveUp)
                       : "memory");
          v = was == v ? v | kGaveUp : was;
        }
        break;
      }
    }
    s_ok = (v & kGaveUp) == 0;
  }
  __syncthreads();
  return s_ok != 0;
}

static size_t cluster_smem(int64_t n, int dim, int cap) { return 4 * (size_t)n * dim + (size_t)cap * 14 + 64; }

template <int DIM, int NEG, bool GRID>
__global__ void __launch_bounds__(kClusterThreads, 1) layout_cluster_kernel(ClusterArgs a) {
  extern __shared__ __align__(16) unsigned char layout_smem[];
  float* sy = reinterpret_cast<float*>(layout_smem);  // Y
  float* s_next = sy + (size_t)a.n * DIM;             // the share's edges: schedule ...
  float* s_eps = s_next + a.cap;
  uint32_t* s_ids = reinterpret_cast<uint32_t*>(s_eps + a.cap);  // ... head | tail << 16
  uint16_t* s_queue = reinterpret_cast<uint16_t*>(s_ids + a.cap);
  __shared__ int s_due;
  const int tid = threadIdx.x, lane = tid & 31;
  const unsigned below = (1u << lane) - 1u;
  const int rank = GRID ? (int)blockIdx.x : (int)cluster::rank(), ctas = GRID ? (int)gridDim.x : (int)cluster::size();
  unsigned meetings = 0;
  auto meet = [&]() {
    if constexpr (GRID) {
      return grid_barrier(a, ++meetings * gridDim.x);
    } else {
      __syncwarp();
      cluster::barrier();
      return true;
    }
  };
  const int64_t E = *a.n_edges < (int64_t)a.cap * ctas ? *a.n_edges : (int64_t)a.cap * ctas;
  const int per = (int)((E + ctas - 1) / ctas);
  const int64_t e0 = (int64_t)rank * per;
  const int m = (int)(E - e0 < 0 ? 0 : E - e0 < per ? E - e0 : per);
  const int r0 = rank * a.rows_per;
  const int own = a.n - r0 < 0 ? 0 : a.n - r0 < a.rows_per ? a.n - r0 : a.rows_per;
  for (int t = tid; t < a.n * DIM; t += kClusterThreads) sy[t] = a.Y[t];
  const int values = a.n * DIM;
  for (int t = tid; t < own * DIM; t += kClusterThreads) __stcg(a.dY + r0 * DIM + t, 0.f);  // the first array
  for (int t = tid; t < m; t += kClusterThreads) {
    s_next[t] = a.next[e0 + t];
    s_eps[t] = a.eps[e0 + t];
    s_ids[t] = (uint32_t)a.rows[e0 + t] | ((uint32_t)a.cols[e0 + t] << 16);
  }
  auto row = [&](uint32_t i, float (&v)[DIM]) {
    if constexpr (DIM == 2) {
      const float2 t = *reinterpret_cast<const float2*>(sy + 2 * i);
      v[0] = t.x;
      v[1] = t.y;
    } else {
#pragma unroll
      for (int c = 0; c < DIM; ++c) v[c] = sy[i * DIM + c];
    }
  };
  if (tid == 0) s_due = 0;
  bool ok = meet();  // the first array is zero

  Params p;
  p.a = a.a;
  p.b = a.b;
  p.m2ab = a.m2ab;
  p.two_b = a.two_b;
  int turn = 0;
  for (int ep = a.epoch_begin; ok && ep < a.epoch_end; ++ep) {
    float* dY = a.dY + (size_t)turn * values;
    const int then = turn == 2 ? 0 : turn + 1;
    float* next_dY = a.dY + (size_t)then * values;
    // make_params' double arithmetic
    p.alpha = (float)__dmul_rn((double)a.lr, __dsub_rn(1.0, __ddiv_rn((double)ep, (double)a.n_epochs)));
    const float epf = (float)ep;
    for (int b0 = tid - lane; b0 < m; b0 += kClusterThreads) {
      const int t = b0 + lane;
      bool due = false;
      if (t < m) {
        const float nx = s_next[t];
        due = nx <= epf;
        if (due) s_next[t] = __fadd_rn(nx, s_eps[t]);
      }
      const unsigned b = __ballot_sync(0xffffffffu, due);
      int slot = 0;
      if (lane == 0 && b) slot = atomicAdd(&s_due, __popc(b));
      slot = __shfl_sync(0xffffffffu, slot, 0);
      if (due) s_queue[slot + __popc(b & below)] = (uint16_t)t;
    }
    __syncthreads();
    const int total = s_due;
    for (int q = tid; q < total; q += kClusterThreads) {
      const int t = s_queue[q];
      const uint32_t e = (uint32_t)(e0 + t);  // below 2^32: the share fits a CTA
      const uint32_t ij = s_ids[t], i = ij & 0xffffu, j = ij >> 16;
      float yi[DIM], yj[DIM], acc[DIM], pos[DIM], neg_pos[DIM];
      row(i, yi);
      row(j, yj);
      attract<DIM>(yi, yj, p, pos);
#pragma unroll
      for (int c = 0; c < DIM; ++c) {
        acc[c] = pos[c];
        neg_pos[c] = -pos[c];
      }
      atomic_add_row<DIM>(dY, (int)j, neg_pos);
      const int nr = NEG > 0 ? NEG : a.neg_rate;
#pragma unroll 1
      for (int m0 = 0; m0 < nr; m0 += 4) {
        const U4 r = philox4x32_10(U4{e, 0u, (uint32_t)ep, (uint32_t)(m0 >> 2)}, a.k0, a.k1);
        const uint32_t w[4] = {r.x, r.y, r.z, r.w};
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          if (m0 + u < nr) {
            float yt[DIM];
            row((uint32_t)to_range(w[u], (uint32_t)a.n), yt);
            repel_add<DIM>(yi, yt, p, acc);
          }
        }
      }
      atomic_add_row<DIM>(dY, (int)i, acc);
    }
    for (int t = tid; t < own * DIM; t += kClusterThreads) __stcg(next_dY + r0 * DIM + t, 0.f);
    ok = meet();  // all moves have been added, and the next array is zero
    if (!ok) break;
    if (tid == 0) s_due = 0;
    for (int t = tid; t < values; t += kClusterThreads) sy[t] = __fadd_rn(sy[t], __ldcg(dY + t));
    turn = then;
    __syncthreads();
  }
  if (!ok) {  // every CTA is here: Y and the schedule stay as they were
    if (tid == 0) atomicExch(a.status, (int32_t)kDevTimeoutEpilogue);
    return;
  }
  for (int t = tid; t < m; t += kClusterThreads) a.next[e0 + t] = s_next[t];
  for (int t = tid; t < own * DIM; t += kClusterThreads) a.Y[r0 * DIM + t] = sy[r0 * DIM + t];
}

// ---- injected path (reference-ordered negatives) ------------------------------
__global__ void count_active_kernel(const float* __restrict__ next, const int64_t* __restrict__ n_edges, int epoch,
                                    int32_t* __restrict__ block_counts) {
  __shared__ int warp_counts[kBlock / 32];
  const int64_t E = *n_edges;
  const float ep = (float)epoch;
  const int64_t base = (int64_t)blockIdx.x * kEdgesPerBlock;
  int c = 0;
  for (int u = 0; u < kEdgesPerBlock / kBlock; ++u) {
    const int64_t e = base + u * kBlock + threadIdx.x;
    c += (e < E && next[e] <= ep) ? 1 : 0;
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) c += __shfl_xor_sync(0xffffffffu, c, o);
  if ((threadIdx.x & 31) == 0) warp_counts[threadIdx.x >> 5] = c;
  __syncthreads();
  if (threadIdx.x == 0) {
    int t = 0;
    for (int i = 0; i < kBlock / 32; ++i) t += warp_counts[i];
    block_counts[blockIdx.x] = t;
  }
}

template <int DIM>
__global__ void __launch_bounds__(kBlock) sgd_injected_kernel(
    const float* __restrict__ Y, float* __restrict__ dY, const int32_t* __restrict__ rows,
    const int32_t* __restrict__ cols, const float* __restrict__ eps, float* __restrict__ next,
    const int64_t* __restrict__ n_edges, int epoch, Params p, int neg_rate, const int32_t* __restrict__ neg_to,
    const int32_t* __restrict__ block_offsets, const int64_t* __restrict__ n_active) {
  __shared__ int warp_base[kBlock / 32];
  __shared__ int running;
  const int64_t E = *n_edges;
  const int64_t A = *n_active;
  const float ep = (float)epoch;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (threadIdx.x == 0) running = block_offsets[blockIdx.x];
  __syncthreads();
  const int64_t base = (int64_t)blockIdx.x * kEdgesPerBlock;
  for (int u = 0; u < kEdgesPerBlock / kBlock; ++u) {
    const int64_t e = base + u * kBlock + threadIdx.x;
    const float nx = e < E ? next[e] : 1.0f;
    const bool act = e < E && nx <= ep;
    const unsigned ballot = __ballot_sync(0xffffffffu, act);
    if (lane == 0) warp_base[warp] = __popc(ballot);
    __syncthreads();
    if (threadIdx.x == 0) {
      int s = running;
      for (int w = 0; w < kBlock / 32; ++w) {
        const int c = warp_base[w];
        warp_base[w] = s;
        s += c;
      }
      running = s;
    }
    __syncthreads();
    if (act) {
      const int64_t rank = warp_base[warp] + __popc(ballot & ((1u << lane) - 1u));
      next[e] = __fadd_rn(nx, eps[e]);
      const int i = rows[e], j = cols[e];
      float yi[DIM], yj[DIM], acc[DIM], pos[DIM], neg_pos[DIM];
      load_row<DIM>(Y, i, yi);
      load_row<DIM>(Y, j, yj);
      attract<DIM>(yi, yj, p, pos);
#pragma unroll
      for (int c = 0; c < DIM; ++c) {
        acc[c] = pos[c];
        neg_pos[c] = -pos[c];
      }
      atomic_add_row<DIM>(dY, j, neg_pos);
      for (int m = 0; m < neg_rate; ++m) {
        float yt[DIM];
        load_row<DIM>(Y, neg_to[rank + (int64_t)m * A], yt);
        repel_add<DIM>(yi, yt, p, acc);
      }
      atomic_add_row<DIM>(dY, i, acc);
    }
    __syncthreads();
  }
}

// ---- n_components 5..32: one warp per edge, lane c holds component c ---------
// The same pair formulas as attract / repel_add; |diff|^2 is summed across the warp
// (butterfly), so its float32 rounding order differs from the sequential sum of the
// narrow kernels by a few ulp.
__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = __fadd_rn(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}

__device__ __forceinline__ float attract_wide(float yi, float yj, const Params& p) {
  const float diff = __fsub_rn(yi, yj);
  const float d2 = fmaxf(warp_sum(__fmul_rn(diff, diff)), 1e-6f);
  const float pw = pow_b(d2, p.b);
  const float coeff = __fdiv_rn(__fmul_rn(p.m2ab, pw), __fmul_rn(d2, __fadd_rn(1.0f, __fmul_rn(p.a, pw))));
  return __fmul_rn(fminf(fmaxf(__fmul_rn(coeff, diff), -4.0f), 4.0f), p.alpha);
}

__device__ __forceinline__ float repel_wide(float yi, float yt, const Params& p) {
  const float diff = __fsub_rn(yi, yt);
  const float d2 = fmaxf(warp_sum(__fmul_rn(diff, diff)), 1e-6f);
  const float pw = pow_b(d2, p.b);
  const float den = __fmul_rn(__fadd_rn(0.001f, d2), __fadd_rn(1.0f, __fmul_rn(p.a, pw)));
  const float coeff = __fdiv_rn(p.two_b, den);
  return __fmul_rn(fminf(fmaxf(__fmul_rn(coeff, diff), -4.0f), 4.0f), p.alpha);
}

// One active edge by a whole warp.  Tails: Philox words of counter (e, epoch, m/4)
// in the order of the narrow kernels; with neg_to, the injected tails of rank `rank`.
__device__ __forceinline__ void edge_update_wide(const float* __restrict__ Y, float* __restrict__ dY, int n, int dim,
                                                 int lane, int i, int j, int64_t e, int epoch, const Params& p,
                                                 int neg_rate, uint32_t k0, uint32_t k1,
                                                 const int32_t* __restrict__ neg_to, int64_t rank, int64_t A) {
  const bool on = lane < dim;
  const float yi = on ? __ldg(Y + (int64_t)i * dim + lane) : 0.f;
  const float yj = on ? __ldg(Y + (int64_t)j * dim + lane) : 0.f;
  const float pos = attract_wide(yi, yj, p);
  if (on) atomicAdd(dY + (int64_t)j * dim + lane, -pos);
  float acc = pos;
  for (int m0 = 0; m0 < neg_rate; m0 += 4) {
    uint32_t r[4];
    if (!neg_to) {
      const U4 q = philox4x32_10(U4{(uint32_t)e, (uint32_t)(e >> 32), (uint32_t)epoch, (uint32_t)(m0 >> 2)}, k0, k1);
      r[0] = q.x, r[1] = q.y, r[2] = q.z, r[3] = q.w;
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      if (m0 + u >= neg_rate) break;
      const int t = neg_to ? neg_to[rank + (int64_t)(m0 + u) * A] : to_range(r[u], (uint32_t)n);
      const float yt = on ? __ldg(Y + (int64_t)t * dim + lane) : 0.f;
      acc = __fadd_rn(acc, repel_wide(yi, yt, p));
    }
  }
  if (on) atomicAdd(dY + (int64_t)i * dim + lane, acc);
}

__global__ void __launch_bounds__(kBlock) sgd_epoch_wide_kernel(const float* __restrict__ Y, float* __restrict__ dY,
                                                                int n, int dim, const int32_t* __restrict__ rows,
                                                                const int32_t* __restrict__ cols,
                                                                const float* __restrict__ eps,
                                                                float* __restrict__ next,
                                                                const int64_t* __restrict__ n_edges, int epoch,
                                                                Params p, int neg_rate, uint32_t k0, uint32_t k1) {
  const int lane = threadIdx.x & 31;
  const int64_t E = *n_edges;
  const float ep = (float)epoch;
  const int64_t warps = (int64_t)gridDim.x * (kBlock / 32);
  for (int64_t base = ((int64_t)blockIdx.x * (kBlock / 32) + (threadIdx.x >> 5)) * 32; base < E; base += warps * 32) {
    const int64_t e = base + lane;
    bool due = false;
    if (e < E) {
      const float nx = next[e];
      due = nx <= ep;
      if (due) next[e] = __fadd_rn(nx, eps[e]);
    }
    unsigned b = __ballot_sync(0xffffffffu, due);
    while (b) {
      const int t = __ffs(b) - 1;
      b &= b - 1;
      const int64_t ed = base + t;
      edge_update_wide(Y, dY, n, dim, lane, rows[ed], cols[ed], ed, epoch, p, neg_rate, k0, k1, nullptr, 0, 0);
    }
  }
}

// Injected tails for n_components 5..32: active edges of each 256-edge chunk are
// ranked like sgd_injected_kernel (block offsets from the scan), queued in shared
// memory, and each queued edge is processed by one warp.
__global__ void __launch_bounds__(kBlock) sgd_injected_wide_kernel(
    const float* __restrict__ Y, float* __restrict__ dY, int n, int dim, const int32_t* __restrict__ rows,
    const int32_t* __restrict__ cols, const float* __restrict__ eps, float* __restrict__ next,
    const int64_t* __restrict__ n_edges, int epoch, Params p, int neg_rate, const int32_t* __restrict__ neg_to,
    const int32_t* __restrict__ block_offsets, const int64_t* __restrict__ n_active) {
  __shared__ int warp_base[kBlock / 32];
  __shared__ int running;
  __shared__ int64_t q_edge[kBlock];
  __shared__ int64_t q_rank[kBlock];
  __shared__ int chunk_start, chunk_count;
  const int64_t E = *n_edges;
  const int64_t A = *n_active;
  const float ep = (float)epoch;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (threadIdx.x == 0) running = block_offsets[blockIdx.x];
  __syncthreads();
  const int64_t base = (int64_t)blockIdx.x * kEdgesPerBlock;
  for (int u = 0; u < kEdgesPerBlock / kBlock; ++u) {
    const int64_t e = base + u * kBlock + threadIdx.x;
    const float nx = e < E ? next[e] : 1.0f;
    const bool act = e < E && nx <= ep;
    const unsigned ballot = __ballot_sync(0xffffffffu, act);
    if (lane == 0) warp_base[warp] = __popc(ballot);
    __syncthreads();
    if (threadIdx.x == 0) {
      int s = running;
      chunk_start = s;
      for (int w = 0; w < kBlock / 32; ++w) {
        const int c = warp_base[w];
        warp_base[w] = s;
        s += c;
      }
      chunk_count = s - running;
      running = s;
    }
    __syncthreads();
    if (act) {
      const int64_t rank = warp_base[warp] + __popc(ballot & ((1u << lane) - 1u));
      next[e] = __fadd_rn(nx, eps[e]);
      q_edge[rank - chunk_start] = e;
      q_rank[rank - chunk_start] = rank;
    }
    __syncthreads();
    for (int t = warp; t < chunk_count; t += kBlock / 32) {
      const int64_t ed = q_edge[t];
      edge_update_wide(Y, dY, n, dim, lane, rows[ed], cols[ed], ed, epoch, p, neg_rate, 0, 0, neg_to, q_rank[t], A);
    }
    __syncthreads();
  }
}

struct Layout {
  int32_t* status;
  float* dY;
  float* wmax;
  int32_t* block_counts;
  int64_t* total;
  int64_t* scan_ws;  // scan_exclusive's block totals
  size_t bytes;
};

static Layout carve(void* ws, int64_t n, int dim, int64_t e_cap) {
  Carver c(ws);
  Layout l;
  l.status = c.take<int32_t>(64);
  l.wmax = c.take<float>(64);
  l.dY = c.take<float>((size_t)n * dim * (resident_rows(n, dim) ? 3 : 1));  // three arrays in turn
  l.block_counts = c.take<int32_t>((size_t)ceil_div(e_cap > 0 ? e_cap : 1, kEdgesPerBlock) + 1);
  l.total = c.take<int64_t>(8);
  l.scan_ws = c.take<int64_t>(kScanMaxBlocks);
  l.bytes = c.bytes();
  return l;
}

static Params make_params(float a, float b, float lr, int epoch, int n_epochs) {
  Params p;
  p.a = a;
  p.b = b;
  p.m2ab = (-2.0f * a) * b;
  p.two_b = 2.0f * b;
  // the reference computes alpha in Python double and casts it to float32 (umap.py:431)
  p.alpha = (float)((double)lr * (1.0 - (double)epoch / (double)n_epochs));
  return p;
}

static unsigned edge_grid(int64_t e_cap) {
  const int64_t want = ceil_div(e_cap > 0 ? e_cap : 1, kBlock);
  const int64_t cap = (int64_t)num_sms() * 16;
  return (unsigned)(want < cap ? want : cap);
}

// a few resident blocks per SM: long warp segments keep the partial batches rare
static unsigned epoch_grid(int64_t e_cap, int blocks_per_sm) {
  const int64_t want = ceil_div(e_cap > 0 ? e_cap : 1, kBlock * 4);
  const int64_t cap = (int64_t)num_sms() * blocks_per_sm;
  return (unsigned)(want < cap ? want : cap);
}

// The kernels compiled for 5 negatives (of the launches and of the single launch) run at that rate
// unless the environment sets UMAPB_LAYOUT_NEG5=0 (read per call): the same draws and sums.
static bool neg5_kernel_enabled() {
  const char* e = getenv("UMAPB_LAYOUT_NEG5");
  return !(e && e[0] == '0' && e[1] == 0);
}

// A launch that may start before the grid before it has ended (overlap), or not.
template <typename... P, typename... A>
static void launch_overlapping(void (*kernel)(P...), unsigned grid, bool overlap, cudaStream_t stream, A... args) {
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(kBlock);
  cfg.stream = stream;
  cfg.attrs = attr;
  cfg.numAttrs = overlap ? 1 : 0;
  cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);  // an error is seen by the launch check
}

// Chunks in a pass of the epoch kernel, so that a warp's segment is cut into passes of equal length: a
// short last pass leaves most of a block's batches out.  The length is compiled in: a branch in front
// of every chunk cost more than it gave.  B200, per epoch, passes of 8 chunks / equal ones by a
// branch / by the kernel: 70,000 points, k = 15 (7 chunks a warp) 20.0 / 20.0 / 19.2 us, 85,000, 3
// components (9) 40.6 / 40.1 / 39.3, 170,000, 1 component (17) 39.9 / 39.4 / 38.1, 40,000, k = 100 (27)
// 26.7 / 27.2 / 25.1; 1,000,000 (99) 229.4 / 233.2 / 229.5.
static int pass_chunks(int64_t e_cap, unsigned grid) {
  const int64_t chunks = ceil_div(ceil_div(e_cap > 0 ? e_cap : 1, 32), (int64_t)grid * (kBlock / 32));
  const int64_t passes = ceil_div(chunks, kPreMax);
  const int64_t c = ceil_div(chunks, passes);
  return (int)(c < kPreMin ? kPreMin : c);
}

template <int DIM, int NEG>
static auto epoch_kernel(int chunks) -> decltype(&sgd_epoch_kernel<DIM, NEG, kPreMax>) {
  return chunks == 5   ? sgd_epoch_kernel<DIM, NEG, 5>
         : chunks == 6 ? sgd_epoch_kernel<DIM, NEG, 6>
         : chunks == 7 ? sgd_epoch_kernel<DIM, NEG, 7>
                       : sgd_epoch_kernel<DIM, NEG, 8>;
}

// first: the grid before is not an epoch's apply
template <int DIM>
static void launch_epoch(const Layout& l, float* Y, int64_t n, const int32_t* rows, const int32_t* cols,
                         const float* eps, float* next, const int64_t* n_edges, int64_t e_cap, int epoch,
                         const Params& p, int neg_rate, uint64_t seed, bool neg5, bool first, cudaStream_t stream) {
  const bool five = neg_rate == 5 && neg5;
  const unsigned grid = epoch_grid(e_cap, five ? kEpochBlocksPerSM5 : kEpochBlocksPerSM);
  const int chunks = pass_chunks(e_cap, grid);
  launch_overlapping(five ? epoch_kernel<DIM, 5>(chunks) : epoch_kernel<DIM, 0>(chunks), grid, !first, stream, Y, l.dY, n,
                     rows, cols, eps, next, n_edges, epoch, p, neg_rate, (uint32_t)seed, (uint32_t)(seed >> 32));
  const int64_t m = n * DIM;
  const unsigned gb = (unsigned)(ceil_div(m, 4 * kBlock) < num_sms() * 8 ? ceil_div(m, 4 * kBlock) : num_sms() * 8);
  launch_overlapping(apply_kernel, gb, true, stream, Y, l.dY, m);
}
static void launch_epoch_wide(const Layout& l, float* Y, int64_t n, int dim, const int32_t* rows,
                              const int32_t* cols, const float* eps, float* next, const int64_t* n_edges,
                              int64_t e_cap, int epoch, const Params& p, int neg_rate, uint64_t seed,
                              cudaStream_t stream) {
  const int64_t want = ceil_div(e_cap > 0 ? e_cap : 1, kBlock);
  const int64_t cap = (int64_t)num_sms() * 8;
  sgd_epoch_wide_kernel<<<(unsigned)(want < cap ? want : cap), kBlock, 0, stream>>>(
      Y, l.dY, (int)n, dim, rows, cols, eps, next, n_edges, epoch, p, neg_rate, (uint32_t)seed,
      (uint32_t)(seed >> 32));
  const int64_t m = n * dim;
  const unsigned gb = (unsigned)(ceil_div(m, kBlock) < num_sms() * 8 ? ceil_div(m, kBlock) : num_sms() * 8);
  apply_kernel<<<gb, kBlock, 0, stream>>>(Y, l.dY, m);
}

template <int DIM>
static void launch_injected(const Layout& l, float* Y, int64_t n, const int32_t* rows, const int32_t* cols,
                            const float* eps, float* next, const int64_t* n_edges, int64_t e_cap, int epoch,
                            const Params& p, int neg_rate, const int32_t* neg_to, cudaStream_t stream) {
  const unsigned nb = (unsigned)ceil_div(e_cap > 0 ? e_cap : 1, kEdgesPerBlock);
  sgd_injected_kernel<DIM><<<nb, kBlock, 0, stream>>>(Y, l.dY, rows, cols, eps, next, n_edges, epoch, p, neg_rate,
                                                      neg_to, l.block_counts, l.total);
  const int64_t m = n * DIM;
  apply_kernel<<<(unsigned)ceil_div(m, kBlock), kBlock, 0, stream>>>(Y, l.dY, m);
}

// Enqueues epochs [begin, end) on a resident grid, one CTA per SM at most and at least 256
// edges each (a smaller barrier); false: as launch_cluster.
template <int DIM, int NEG>
static bool launch_grid(ClusterArgs a, int64_t e_cap, cudaStream_t stream) {
  static std::mutex mu;
  static int known[64] = {0};  // 1: cooperative launches of the kernel work on this device; -1: not
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return false;
  const void* kernel = (const void*)layout_cluster_kernel<DIM, NEG, true>;
  {
    std::lock_guard<std::mutex> lock(mu);
    if (known[dev] == 0) {
      int coop = 0, per_sm = 0;
      known[dev] = cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev) == cudaSuccess && coop &&
                           cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                (int)kClusterSmem) == cudaSuccess &&
                           cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, kClusterThreads,
                                                                         kClusterSmem) == cudaSuccess &&
                           per_sm > 0
                       ? 1
                       : -1;
      cudaGetLastError();
    }
    if (known[dev] < 0) return false;
  }
  int64_t ctas = ceil_div(e_cap > 0 ? e_cap : 1, 256);
  if (ctas > num_sms()) ctas = num_sms();
  a.rows_per = (int)ceil_div(a.n, ctas);
  a.cap = (int)ceil_div(e_cap, ctas);
  const size_t smem = cluster_smem(a.n, DIM, a.cap);
  if (smem > kClusterSmem || a.cap > 65535) return false;
  if (cudaMemsetAsync(a.bar, 0, sizeof(unsigned), stream) != cudaSuccess) {  // umapb_layout_prepare clears the status
    cudaGetLastError();
    return false;
  }
  void* args[] = {&a};
  if (cudaLaunchCooperativeKernel(kernel, dim3((unsigned)ctas), dim3(kClusterThreads), args, smem, stream) !=
      cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  return true;
}

// Enqueues epochs [begin, end) on one cluster; false: the problem does not fit one, or the
// device cannot schedule one (the launches serve it then).
template <int DIM, int NEG>
static bool launch_cluster(ClusterArgs a, int64_t e_cap, cudaStream_t stream) {
  static std::mutex mu;
  static int known[64] = {0};  // CTAs per cluster on this device; 0 unknown, -1 none
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return false;
  const auto kernel = layout_cluster_kernel<DIM, NEG, false>;
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.blockDim = dim3(kClusterThreads, 1, 1);
  cfg.stream = stream;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  {
    std::lock_guard<std::mutex> lock(mu);
    if (known[dev] == 0) {
      known[dev] = -1;
      if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kClusterSmem) == cudaSuccess &&
          cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess) {
        for (int c = kClusterMax; c >= 8 && known[dev] < 0; c /= 2) {
          attr[0].val.clusterDim.x = c;
          cfg.gridDim = dim3(c, 1, 1);
          cfg.dynamicSmemBytes = kClusterSmem;
          int clusters = 0;
          if (cudaOccupancyMaxActiveClusters(&clusters, kernel, &cfg) == cudaSuccess && clusters > 0) known[dev] = c;
        }
      }
      cudaGetLastError();
    }
  }
  const int ctas = known[dev];
  if (ctas < 0) return false;
  a.rows_per = (int)ceil_div(a.n, ctas);
  a.cap = (int)ceil_div(e_cap, ctas);
  cfg.dynamicSmemBytes = cluster_smem(a.n, DIM, a.cap);
  if (cfg.dynamicSmemBytes > kClusterSmem) return false;
  attr[0].val.clusterDim.x = ctas;
  cfg.gridDim = dim3(ctas, 1, 1);
  if (cudaLaunchKernelEx(&cfg, kernel, a) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  return true;
}

// UMAPB_LAYOUT_ONE_LAUNCH in the environment (read per call): 0 runs few rows by launches as well,
// grid runs few edges on the grid that devices without such clusters use.
static bool one_launch_is(const char* what) {
  const char* e = getenv("UMAPB_LAYOUT_ONE_LAUNCH");
  return e && strcmp(e, what) == 0;
}

template <int DIM, int NEG>
static bool launch_resident(const ClusterArgs& a, int64_t e_cap, cudaStream_t stream) {
  return (e_cap <= kClusterEdges && !one_launch_is("grid") && launch_cluster<DIM, NEG>(a, e_cap, stream)) ||
         launch_grid<DIM, NEG>(a, e_cap, stream);
}

}  // namespace layout
}  // namespace umapb

using namespace umapb;

extern "C" int umapb_layout_workspace(int64_t n, int32_t dim, int64_t e_cap, size_t* bytes) {
  clear_error();
  UMAPB_REQUIRE(bytes, "bytes is null");
  UMAPB_REQUIRE(n >= 1 && dim >= 1 && dim <= 32 && e_cap >= 0, "layout: need n >= 1, 1 <= dim <= 32, e_cap >= 0");
  *bytes = layout::carve(nullptr, n, dim, e_cap).bytes;
  return UMAPB_OK;
}

extern "C" int umapb_layout_prepare(const float* vals, const int64_t* n_edges, int64_t e_cap, int32_t n_epochs,
                                    float* eps, float* next, void* workspace, size_t workspace_bytes,
                                    umapb_stream_t stream_) {
  clear_error();
  cudaStream_t stream = reinterpret_cast<cudaStream_t>(stream_);
  UMAPB_REQUIRE(vals && n_edges && eps && next, "layout_prepare: null array argument");
  UMAPB_REQUIRE(n_epochs >= 1, "layout_prepare: n_epochs must be >= 1");
  UMAPB_REQUIRE(workspace && workspace_bytes >= 512, "layout_prepare: workspace too small");
  layout::Layout l = layout::carve(workspace, 1, 1, 1);  // status and wmax sit at fixed offsets
  UMAPB_CUDA_TRY(cudaMemsetAsync(l.status, 0, reinterpret_cast<char*>(l.wmax + 1) - reinterpret_cast<char*>(l.status),
                                 stream),
                 "layout_prepare: reset");
  const unsigned g = layout::edge_grid(e_cap);
  layout::max_kernel<<<g, layout::kBlock, 0, stream>>>(vals, n_edges, l.wmax);
  layout::eps_kernel<<<g, layout::kBlock, 0, stream>>>(vals, n_edges, l.wmax, n_epochs, eps, next);
  UMAPB_LAUNCH_CHECK("layout_prepare kernels");
  count_launches(2);
  return UMAPB_OK;
}

static int check_epochs(const float* Y, int64_t n, int32_t dim, const int32_t* rows, const int32_t* cols,
                        const float* eps, const float* next, const int64_t* n_edges, int64_t e_cap,
                        int32_t epoch_begin, int32_t epoch_end, int32_t n_epochs, int32_t neg_rate,
                        const void* workspace, size_t workspace_bytes) {
  UMAPB_REQUIRE(Y && rows && cols && eps && next && n_edges, "layout_epochs: null array argument");
  UMAPB_REQUIRE(n >= 1 && n < ((int64_t)1 << 31), "layout_epochs: need 1 <= n < 2^31");
  UMAPB_REQUIRE(dim >= 1 && dim <= 32, "layout_epochs: dim must be in [1, 32]");
  UMAPB_REQUIRE(neg_rate >= 0, "layout_epochs: negative_sample_rate must be >= 0");
  UMAPB_REQUIRE(0 <= epoch_begin && epoch_begin <= epoch_end && epoch_end <= n_epochs,
                "layout_epochs: need 0 <= epoch_begin <= epoch_end <= n_epochs");
  const layout::Layout l = layout::carve(nullptr, n, dim, e_cap);
  if (!workspace || workspace_bytes < l.bytes)
    return set_error(UMAPB_ERR_WORKSPACE, "layout: workspace of %zu bytes, need %zu", workspace_bytes, l.bytes);
  return UMAPB_OK;
}

// The cluster form, where the checked arguments allow it.
static bool enqueue_cluster(float* Y, int64_t n, int32_t dim, const int32_t* rows, const int32_t* cols,
                            const float* eps, float* next, const int64_t* n_edges, int64_t e_cap, int32_t epoch_begin,
                            int32_t epoch_end, int32_t n_epochs, float a, float b, float learning_rate,
                            int32_t neg_rate, uint64_t seed, void* workspace, cudaStream_t stream) {
  // below four epochs the load of the edges and the store of their schedule cost more than the
  // launches (a callback after every epoch runs them one by one)
  // (above a million epochs the barrier's count would run into its top bit)
  if (!layout::resident_rows(n, dim) || epoch_end - epoch_begin < 4 ||
      epoch_end - epoch_begin > 1000000 || layout::one_launch_is("0"))
    return false;
  const layout::Params p = layout::make_params(a, b, learning_rate, 0, n_epochs);
  layout::ClusterArgs c = {};
  const layout::Layout l = layout::carve(workspace, n, dim, e_cap);
  c.Y = Y;
  c.dY = l.dY;
  c.status = l.status;
  c.bar = reinterpret_cast<unsigned*>(l.status + 32);
  c.limit_ns = wait_limit_ns();
  c.rows = rows;
  c.cols = cols;
  c.eps = eps;
  c.next = next;
  c.n_edges = n_edges;
  c.n = (int)n;
  c.epoch_begin = epoch_begin;
  c.epoch_end = epoch_end;
  c.n_epochs = n_epochs;
  c.neg_rate = neg_rate;
  c.a = p.a;
  c.b = p.b;
  c.m2ab = p.m2ab;
  c.two_b = p.two_b;
  c.lr = learning_rate;
  c.k0 = (uint32_t)seed;
  c.k1 = (uint32_t)(seed >> 32);
  const bool five = neg_rate == 5 && layout::neg5_kernel_enabled();
  bool ok = false;
  switch (dim) {
    case 1: ok = layout::launch_resident<1, 0>(c, e_cap, stream); break;
    case 2: ok = five ? layout::launch_resident<2, 5>(c, e_cap, stream) : layout::launch_resident<2, 0>(c, e_cap, stream); break;
    case 3: ok = five ? layout::launch_resident<3, 5>(c, e_cap, stream) : layout::launch_resident<3, 0>(c, e_cap, stream); break;
    default: ok = layout::launch_resident<4, 0>(c, e_cap, stream); break;
  }
  if (ok) count_launches(1);
  return ok;
}

static int enqueue_epochs(float* Y, int64_t n, int32_t dim, const int32_t* rows, const int32_t* cols,
                          const float* eps, float* next, const int64_t* n_edges, int64_t e_cap, int32_t epoch_begin,
                          int32_t epoch_end, int32_t n_epochs, float a, float b, float learning_rate,
                          int32_t neg_rate, uint64_t seed, void* workspace, size_t workspace_bytes,
                          cudaStream_t stream) {
  layout::Layout l = layout::carve(nullptr, n, dim, e_cap);
  if (!workspace || workspace_bytes < l.bytes)
    return set_error(UMAPB_ERR_WORKSPACE, "layout: workspace of %zu bytes, need %zu", workspace_bytes, l.bytes);
  l = layout::carve(workspace, n, dim, e_cap);
  UMAPB_CUDA_TRY(cudaMemsetAsync(l.dY, 0, sizeof(float) * n * dim, stream), "layout_epochs: reset");
  const bool neg5 = layout::neg5_kernel_enabled();
  for (int ep = epoch_begin; ep < epoch_end; ++ep) {
    const layout::Params p = layout::make_params(a, b, learning_rate, ep, n_epochs);
    switch (dim) {
      case 1: layout::launch_epoch<1>(l, Y, n, rows, cols, eps, next, n_edges, e_cap, ep, p, neg_rate, seed, neg5, ep == epoch_begin, stream); break;
      case 2: layout::launch_epoch<2>(l, Y, n, rows, cols, eps, next, n_edges, e_cap, ep, p, neg_rate, seed, neg5, ep == epoch_begin, stream); break;
      case 3: layout::launch_epoch<3>(l, Y, n, rows, cols, eps, next, n_edges, e_cap, ep, p, neg_rate, seed, neg5, ep == epoch_begin, stream); break;
      case 4: layout::launch_epoch<4>(l, Y, n, rows, cols, eps, next, n_edges, e_cap, ep, p, neg_rate, seed, neg5, ep == epoch_begin, stream); break;
      default:
        layout::launch_epoch_wide(l, Y, n, dim, rows, cols, eps, next, n_edges, e_cap, ep, p, neg_rate, seed, stream);
        break;
    }
  }
  UMAPB_LAUNCH_CHECK("layout_epochs kernels");
  count_launches(2 * (epoch_end - epoch_begin));
  return UMAPB_OK;
}

extern "C" int umapb_layout_epochs(float* Y, int64_t n, int32_t dim, const int32_t* rows, const int32_t* cols,
                                   const float* eps, float* next, const int64_t* n_edges, int64_t e_cap,
                                   int32_t epoch_begin, int32_t epoch_end, int32_t n_epochs, float a, float b,
                                   float learning_rate, int32_t neg_rate, uint64_t seed, void* workspace,
                                   size_t workspace_bytes, umapb_stream_t stream_) {
  clear_error();
  if (const int rc = check_epochs(Y, n, dim, rows, cols, eps, next, n_edges, e_cap, epoch_begin, epoch_end, n_epochs,
                                  neg_rate, workspace, workspace_bytes))
    return rc;
  if (enqueue_cluster(Y, n, dim, rows, cols, eps, next, n_edges, e_cap, epoch_begin, epoch_end, n_epochs, a, b,
                      learning_rate, neg_rate, seed, workspace, reinterpret_cast<cudaStream_t>(stream_)))
    return UMAPB_OK;
  return enqueue_epochs(Y, n, dim, rows, cols, eps, next, n_edges, e_cap, epoch_begin, epoch_end, n_epochs, a, b,
                        learning_rate, neg_rate, seed, workspace, workspace_bytes,
                        reinterpret_cast<cudaStream_t>(stream_));
}

// One executable graph per device, reused across calls: each call records its
// launches (stream capture, thread-local mode, on a private non-blocking stream:
// the caller's stream may be the legacy default stream, which cannot be captured),
// updates the cached executable with the new parameters (cudaGraphExecUpdate; same
// topology for the same epoch count) or instantiates a new one, and launches it on
// the caller's stream.  Updates affect later launches only, so a replay still in
// flight keeps its parameters.
namespace {
std::mutex g_graph_mu;
cudaGraphExec_t g_graph_exec[64] = {};
cudaStream_t g_capture_stream[64] = {};
}  // namespace

extern "C" int umapb_layout_epochs_graph(float* Y, int64_t n, int32_t dim, const int32_t* rows,
                                         const int32_t* cols, const float* eps, float* next, const int64_t* n_edges,
                                         int64_t e_cap, int32_t epoch_begin, int32_t epoch_end, int32_t n_epochs,
                                         float a, float b, float learning_rate, int32_t neg_rate, uint64_t seed,
                                         void* workspace, size_t workspace_bytes, umapb_stream_t stream_) {
  clear_error();
  cudaStream_t stream = reinterpret_cast<cudaStream_t>(stream_);
  int dev = 0;
  UMAPB_CUDA_TRY(cudaGetDevice(&dev), "layout_epochs_graph: device");
  UMAPB_REQUIRE(dev >= 0 && dev < 64, "layout_epochs_graph: device index out of range");
  cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
  UMAPB_CUDA_TRY(cudaStreamIsCapturing(stream, &cs), "layout_epochs_graph: capture query");
  UMAPB_REQUIRE(cs == cudaStreamCaptureStatusNone, "layout_epochs_graph: the stream is already being captured");
  if (const int rc = check_epochs(Y, n, dim, rows, cols, eps, next, n_edges, e_cap, epoch_begin, epoch_end, n_epochs,
                                  neg_rate, workspace, workspace_bytes))
    return rc;
  if (enqueue_cluster(Y, n, dim, rows, cols, eps, next, n_edges, e_cap, epoch_begin, epoch_end, n_epochs, a, b,
                      learning_rate, neg_rate, seed, workspace, stream))
    return UMAPB_OK;  // one launch: nothing to record
  std::lock_guard<std::mutex> lock(g_graph_mu);
  cudaStream_t& cap = g_capture_stream[dev];
  if (!cap) UMAPB_CUDA_TRY(cudaStreamCreateWithFlags(&cap, cudaStreamNonBlocking), "layout_epochs_graph: stream");
  UMAPB_CUDA_TRY(cudaStreamBeginCapture(cap, cudaStreamCaptureModeThreadLocal), "layout_epochs_graph: capture");
  const int rc = enqueue_epochs(Y, n, dim, rows, cols, eps, next, n_edges, e_cap, epoch_begin, epoch_end, n_epochs, a,
                                b, learning_rate, neg_rate, seed, workspace, workspace_bytes, cap);
  cudaGraph_t graph = nullptr;
  const cudaError_t ce = cudaStreamEndCapture(cap, &graph);
  if (rc != UMAPB_OK || ce != cudaSuccess) {
    if (graph) cudaGraphDestroy(graph);
    if (rc != UMAPB_OK) return rc;
    return set_error(UMAPB_ERR_CUDA, "layout_epochs_graph: end of capture: %s", cudaGetErrorString(ce));
  }
  cudaGraphExec_t& exec = g_graph_exec[dev];
  if (exec) {
    cudaGraphExecUpdateResultInfo info;
    if (cudaGraphExecUpdate(exec, graph, &info) != cudaSuccess) {
      cudaGetLastError();  // a topology change: instantiate anew
      cudaGraphExecDestroy(exec);
      exec = nullptr;
    }
  }
  cudaError_t e = cudaSuccess;
  if (!exec) e = cudaGraphInstantiate(&exec, graph, 0);
  cudaGraphDestroy(graph);
  if (e != cudaSuccess) {
    exec = nullptr;
    return set_error(UMAPB_ERR_CUDA, "layout_epochs_graph: instantiate: %s", cudaGetErrorString(e));
  }
  UMAPB_CUDA_TRY(cudaGraphLaunch(exec, stream), "layout_epochs_graph: launch");
  return UMAPB_OK;
}

extern "C" int umapb_layout_count_active(const float* next, const int64_t* n_edges, int64_t n, int32_t dim,
                                         int64_t e_cap, int32_t epoch, int64_t* count, void* workspace,
                                         size_t workspace_bytes, umapb_stream_t stream_) {
  clear_error();
  cudaStream_t stream = reinterpret_cast<cudaStream_t>(stream_);
  UMAPB_REQUIRE(next && n_edges && count, "layout_count_active: null array argument");
  UMAPB_REQUIRE(n >= 1 && dim >= 1 && dim <= 32, "layout_count_active: need n >= 1 and 1 <= dim <= 32");
  layout::Layout l = layout::carve(nullptr, n, dim, e_cap);
  if (!workspace || workspace_bytes < l.bytes)
    return set_error(UMAPB_ERR_WORKSPACE, "layout: workspace of %zu bytes, need %zu", workspace_bytes, l.bytes);
  l = layout::carve(workspace, n, dim, e_cap);
  const int64_t nb = ceil_div(e_cap > 0 ? e_cap : 1, layout::kEdgesPerBlock);
  layout::count_active_kernel<<<(unsigned)nb, layout::kBlock, 0, stream>>>(next, n_edges, epoch, l.block_counts);
  scan_exclusive(l.block_counts, nb, count, l.scan_ws, stream);
  UMAPB_LAUNCH_CHECK("layout_count_active kernels");
  count_launches(2);
  return UMAPB_OK;
}

extern "C" int umapb_layout_epoch_injected(float* Y, int64_t n, int32_t dim, const int32_t* rows,
                                           const int32_t* cols, const float* eps, float* next,
                                           const int64_t* n_edges, int64_t e_cap, int32_t epoch, int32_t n_epochs,
                                           float a, float b, float learning_rate, int32_t neg_rate,
                                           const int32_t* neg_to, int64_t neg_count, void* workspace,
                                           size_t workspace_bytes, umapb_stream_t stream_) {
  clear_error();
  cudaStream_t stream = reinterpret_cast<cudaStream_t>(stream_);
  UMAPB_REQUIRE(Y && rows && cols && eps && next && n_edges, "layout_epoch_injected: null array argument");
  UMAPB_REQUIRE(dim >= 1 && dim <= 32, "layout_epoch_injected: dim must be in [1, 32]");
  UMAPB_REQUIRE(0 <= epoch && epoch < n_epochs, "layout_epoch_injected: epoch out of range");
  UMAPB_REQUIRE(neg_rate >= 0 && neg_count >= 0, "layout_epoch_injected: negative counts must be >= 0");
  UMAPB_REQUIRE(neg_to || neg_count == 0, "layout_epoch_injected: neg_to is null");
  layout::Layout l = layout::carve(nullptr, n, dim, e_cap);
  if (!workspace || workspace_bytes < l.bytes)
    return set_error(UMAPB_ERR_WORKSPACE, "layout: workspace of %zu bytes, need %zu", workspace_bytes, l.bytes);
  l = layout::carve(workspace, n, dim, e_cap);
  UMAPB_CUDA_TRY(cudaMemsetAsync(l.dY, 0, sizeof(float) * n * dim, stream), "layout_epoch_injected: reset");
  const unsigned nb = (unsigned)ceil_div(e_cap > 0 ? e_cap : 1, layout::kEdgesPerBlock);
  layout::count_active_kernel<<<nb, layout::kBlock, 0, stream>>>(next, n_edges, epoch, l.block_counts);
  scan_exclusive(l.block_counts, (int64_t)nb, l.total, l.scan_ws, stream);
  UMAPB_LAUNCH_CHECK("layout_epoch_injected: active count");
  int64_t active = 0;
  UMAPB_CUDA_TRY(cudaMemcpyAsync(&active, l.total, sizeof(active), cudaMemcpyDeviceToHost, stream),
                 "layout_epoch_injected: count readback");
  UMAPB_CUDA_TRY(cudaStreamSynchronize(stream), "layout_epoch_injected: sync");
  if (active * neg_rate != neg_count)
    return set_error(UMAPB_ERR_ARG, "layout_epoch_injected: epoch %d has %lld active edges, so %lld negatives are "
                     "needed (got %lld)", epoch, (long long)active, (long long)(active * neg_rate),
                     (long long)neg_count);
  const layout::Params p = layout::make_params(a, b, learning_rate, epoch, n_epochs);
  switch (dim) {
    case 1: layout::launch_injected<1>(l, Y, n, rows, cols, eps, next, n_edges, e_cap, epoch, p, neg_rate, neg_to, stream); break;
    case 2: layout::launch_injected<2>(l, Y, n, rows, cols, eps, next, n_edges, e_cap, epoch, p, neg_rate, neg_to, stream); break;
    case 3: layout::launch_injected<3>(l, Y, n, rows, cols, eps, next, n_edges, e_cap, epoch, p, neg_rate, neg_to, stream); break;
    case 4: layout::launch_injected<4>(l, Y, n, rows, cols, eps, next, n_edges, e_cap, epoch, p, neg_rate, neg_to, stream); break;
    default: {
      const unsigned nb = (unsigned)ceil_div(e_cap > 0 ? e_cap : 1, layout::kEdgesPerBlock);
      layout::sgd_injected_wide_kernel<<<nb, layout::kBlock, 0, stream>>>(Y, l.dY, (int)n, dim, rows, cols, eps, next,
                                                                          n_edges, epoch, p, neg_rate, neg_to,
                                                                          l.block_counts, l.total);
      const int64_t m = n * dim;
      layout::apply_kernel<<<(unsigned)ceil_div(m, layout::kBlock), layout::kBlock, 0, stream>>>(Y, l.dY, m);
      break;
    }
  }
  UMAPB_LAUNCH_CHECK("layout_epoch_injected kernels");
  count_launches(4);
  return UMAPB_OK;
}
