// NNDescent row update from the blocked join's distances — the candidate handling of a
// full-path iteration (nndescent.py:241-280, 439-486), one warp per row.
//
// A row's candidates are [current k | first j_nn neighbours of each of its k
// neighbours | reverse k], the first occurrence of an id counts and the k smallest
// (distance, id) stay.  The join has computed every distance already, so the row works
// from the distances to the ids instead of the other way round: the current list,
// sorted, bounds what can enter; of the other candidates (in registers, 32 per
// register) those at or below the bound are taken in bands of at most 32 by ascending
// distance (a bisection finds the band), and only for these the ids are read,
// duplicates dropped and the list updated.  The bound falls with each band, so two
// or three bands settle a row even when all its candidates are new.
//
// The reverse candidates are the row's own bucket of the join (which rows list it, at
// what distance): its k smallest ids, as the reference's slots hold them, and row 0 for
// empty slots (its zero padding), whose distance comes from a per-space array.
//
// What bounds it: instructions (a few hundred per row); ids of rejected candidates are
// never read.  Against collecting every id and removing duplicates through a hash table
// first (and a separate kernel for the reverse slots), B200, row updates of the full
// path: 70000 x 784, k = 15 7 x 415 -> 7 x 125 us; 1000000 x 128, k = 15 7 x 5.2 -> 7 x
// 1.73 ms; 30001 x 50, k = 30 4 x 1500 -> 4 x 340 us.
#include <math.h>

#include "common.cuh"
#include "nnd_select.cuh"
#include "nnd_sort.cuh"

namespace umapb {
namespace nnd {

constexpr int kSelWarps = 4;
constexpr unsigned kAll = 0xffffffffu;
// mark of a candidate that is absent or taken: a NaN, neither below nor at any distance
__device__ __forceinline__ float gone() { return __int_as_float(0x7fffffff); }

// NCH: registers of 32 nn-of-nn candidates (k * j_nn <= 32 NCH)
template <int NCH>
__global__ void __launch_bounds__(kSelWarps * 32) select_rows_kernel(SelectArgs a) {
  __shared__ float s_d[kSelWarps][32];
  __shared__ int s_c[kSelWarps][32];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int64_t pos = (int64_t)blockIdx.x * kSelWarps + warp;
  if (pos >= a.n) return;
  const int64_t row = a.order ? (int64_t)a.order[pos] : pos;
  const int k = a.k, nn_cols = k * a.j_nn;
  const unsigned below = (1u << lane) - 1u;

  const int my_old = lane < k ? a.idx_old[row * k + lane] : -1;
  const float my_d = lane < k ? (a.curd ? a.curd : a.dist_old)[row * k + lane] : 0.f;
  float d[NCH];  // nn-of-nn candidates; gone(): absent or taken
  const float* nn = a.nnbuf + row * nn_cols;
#pragma unroll
  for (int u = 0; u < NCH; ++u) d[u] = u * 32 + lane < nn_cols ? nn[u * 32 + lane] : gone();

  // reverse candidates, one per lane: id rid at distance rd
  int rid = -1, pads = 0;  // pads: empty slots
  float rd = gone();
  if (a.off) {
    const int o = a.off[row], cnt = a.off[row + 1] - o;
    pads = cnt < k ? k - cnt : 0;
    if (cnt <= 32) {
      if (lane < cnt) {
        rid = a.entries[o + lane] >> 5;
        rd = a.entd[o + lane];
      }
      if (cnt > k) {  // the k smallest ids
        int rank = 0;
        for (int t = 0; t < cnt; ++t) {
          const int id = __shfl_sync(kAll, rid, t);
          rank += id < rid || (id == rid && t < lane) ? 1 : 0;
        }
        if (rank >= k) rid = -1, rd = gone();
      } else if (lane == cnt && pads) {
        rid = 0;
        rd = a.d0[row];
      }
    } else {
      // a hub: its k smallest ids in one pass, as a list of (id, entry) over the lanes in which
      // earlier copies of an id come first; the ids arrive nearly ascending, so few enter
      // (bisecting the ids took 17 passes, and one row listed by thousands held up the grid: 100,000 x
      // 51, k = 2 420 -> 142 us)
      int hid = 0x7fffffff, he = 0, worst = 0x7fffffff;
      for (int e0 = 0; e0 < cnt; e0 += 128) {
        int v[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const int e = e0 + 32 * u + lane;
          v[u] = e < cnt ? a.entries[o + e] >> 5 : 0x7fffffff;
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          unsigned b = __ballot_sync(kAll, v[u] < worst);
          while (b) {
            const int s = __ffs(b) - 1;
            const int id = __shfl_sync(kAll, v[u], s);
            const int at = __popc(__ballot_sync(kAll, lane < k && hid <= id));
            const int up_id = __shfl_up_sync(kAll, hid, 1), up_e = __shfl_up_sync(kAll, he, 1);
            if (lane < k && lane >= at) {
              hid = lane == at ? id : up_id;
              he = lane == at ? e0 + 32 * u + s : up_e;
            }
            worst = __shfl_sync(kAll, hid, k - 1);
            b &= b - 1u;
            b &= __ballot_sync(kAll, v[u] < worst);
          }
        }
      }
      if (lane < k) {  // more entries than k, so the list is full
        rid = hid;
        rd = a.entd[o + he];
      }
    }
  }

  // the current list, sorted; later copies of an id and the row itself count as dropped
  float lv = kSent;
  int li = 0x7fffffff;
  {
    const unsigned same = __match_any_sync(kAll, lane < k ? my_old : -2 - lane);
    if (lane < k) {
      lv = (__ffs(same) - 1 == lane && my_old != (int)row) ? my_d : kBig;
      li = my_old;
    }
    const float nv = __shfl_down_sync(kAll, lv, 1);
    const int ni = __shfl_down_sync(kAll, li, 1);
    if (__any_sync(kAll, lane < 31 && key_lt(nv, ni, lv, li))) warp_sort_keys(lv, li, lane);
  }
  float tau = __shfl_sync(kAll, lv, k - 1);
  int tau_i = __shfl_sync(kAll, li, k - 1);

  // gone() is not <= tau, whatever tau is: a turn counts untaken candidates only and takes at least
  // one of them
  while (true) {
    int c = rd <= tau ? 1 : 0;
#pragma unroll
    for (int u = 0; u < NCH; ++u) c += d[u] <= tau ? 1 : 0;
    c = __reduce_add_sync(kAll, c);
    if (c == 0) break;
    float T = tau;
    // a band of at least kBandMin candidates where possible: a step costs NCH compares, a short
    // band may leave the list to be settled by another one (B200, earlier form, 1,000,000 rows, k = 15:
    // 1.96 ms at 12, 1.85 at 20, 1.86 at 26; 30,000 rows, k = 30: 351 us at 12, 362 at 20, 432 at 26)
    constexpr int kBandMin = NCH <= 8 ? 20 : 12;
    if (c > 32) {  // the bits of non-negative floats (and of gone()) order like the values
      uint32_t mn = __float_as_uint(rd);
#pragma unroll
      for (int u = 0; u < NCH; ++u) mn = min(mn, __float_as_uint(d[u]));
      uint32_t lo = __reduce_min_sync(kAll, mn), hi = __float_as_uint(tau);
      bool got = false;
      while (lo < hi) {
        const uint32_t mid = lo + (hi - lo) / 2;
        const float m = __uint_as_float(mid);
        int x = rd <= m ? 1 : 0;
#pragma unroll
        for (int u = 0; u < NCH; ++u) x += d[u] <= m ? 1 : 0;
        x = __reduce_add_sync(kAll, x);
        if (x > 32) {
          hi = mid;
        } else {
          T = m;
          got = true;
          if (x >= kBandMin) break;
          lo = mid + 1u;
        }
      }
      if (!got) T = __uint_as_float(hi);  // more than 32 at the smallest distance: the first of them
    }
    int base = 0;
#pragma unroll
    for (int u = 0; u < NCH; ++u) {
      const bool take = d[u] <= T;
      const unsigned b = __ballot_sync(kAll, take);
      const int p = base + __popc(b & below);
      if (take && p < 32) {
        s_d[warp][p] = d[u];
        s_c[warp][p] = u * 32 + lane;
        d[u] = gone();
      }
      base += __popc(b);
    }
    {
      const bool take = rd <= T;
      const unsigned b = __ballot_sync(kAll, take);
      const int p = base + __popc(b & below);
      if (take && p < 32) {
        s_d[warp][p] = rd;
        s_c[warp][p] = NCH * 32 + lane;
        rd = gone();
      }
      base += __popc(b);
    }
    __syncwarp();
    const int m = base < 32 ? base : 32;
    float cd = lane < m ? s_d[warp][lane] : kSent;
    const int col = lane < m ? s_c[warp][lane] : 0;
    __syncwarp();
    const int p = (int)(((uint32_t)col * a.magic) >> 20);
    const int src = __shfl_sync(kAll, my_old, p & 31);
    int id = __shfl_sync(kAll, rid, col & 31);
    if (lane < m && col < NCH * 32) id = a.idx_old[(int64_t)src * k + (col - p * a.j_nn)];
    bool ok = lane < m && id != (int)row && key_lt(cd, id, tau, tau_i);
    const unsigned same = __match_any_sync(kAll, ok ? id : -2 - lane);
    ok = ok && __ffs(same) - 1 == lane;  // lanes are in column order
    bool dup = false;
    for (int t = 0; t < k; ++t) {
      const int in_list = __shfl_sync(kAll, li, t);  // every lane takes part, whatever dup is
      dup = dup || id == in_list;
    }
    ok = ok && !dup;
    unsigned b = __ballot_sync(kAll, ok);
    if (__popc(b) > 6) {
      if (!ok) {
        cd = kSent;
        id = 0x7fffffff;
      }
      warp_sort_keys(cd, id, lane);
      const float od = __shfl_sync(kAll, cd, 31 - lane);
      const int oi = __shfl_sync(kAll, id, 31 - lane);
      if (key_lt(od, oi, lv, li)) {
        lv = od;
        li = oi;
      }
      warp_bitonic_clean(lv, li, lane);
      if (lane >= k) {
        lv = kSent;
        li = 0x7fffffff;
      }
    } else {
      while (b) {
        const int s = __ffs(b) - 1;
        b &= b - 1u;
        list_insert(lv, li, __shfl_sync(kAll, cd, s), __shfl_sync(kAll, id, s), k, lane);
      }
    }
    tau = __shfl_sync(kAll, lv, k - 1);
    tau_i = __shfl_sync(kAll, li, k - 1);
  }

  if (key_lt(kBig, 0, tau, tau_i)) {
    // Fewer than k candidates nearer than 1e30 (small n, or infinite distances): the dropped
    // columns (the row itself, later copies of an id) count as 1e30, by id.  Those of the
    // current list are in the list already.
    const int total = nn_cols + (a.off ? 32 + pads : 0);
    auto column = [&](int t) {  // the id in column t (behind the current list), -1: none; all lanes call
      const int p = (int)(((uint32_t)(t < nn_cols ? t : 0) * a.magic) >> 20);
      const int src = __shfl_sync(kAll, my_old, p & 31);
      const int r = __shfl_sync(kAll, rid, (t - nn_cols) & 31);
      if (t < nn_cols) return (int)a.idx_old[(int64_t)src * k + (t - p * a.j_nn)];
      if (t < nn_cols + 32) return a.off ? r : -1;  // the slots (the first empty one among them)
      return t < total - 1 ? 0 : -1;                // the other empty slots
    };
    for (int t0 = 0; t0 < total; t0 += 32) {
      const int id = column(t0 + lane);
      const unsigned same = __match_any_sync(kAll, id >= 0 ? id : -2 - lane);
      bool drop = id >= 0 && (id == (int)row || __ffs(same) - 1 != lane);
      for (int t = 0; t < k; ++t) {
        const int other = __shfl_sync(kAll, my_old, t);
        drop = drop || (id >= 0 && id == other);
      }
      for (int e0 = 0; e0 < t0; e0 += 32) {  // an earlier column with the same id
        if (!__any_sync(kAll, id >= 0 && !drop && key_lt(kBig, id, tau, tau_i))) break;
        const int before = column(e0 + lane);
        for (int t = 0; t < 32; ++t) {
          const int other = __shfl_sync(kAll, before, t);
          drop = drop || (id >= 0 && id == other);
        }
      }
      for (unsigned todo = __ballot_sync(kAll, drop); todo; todo &= todo - 1u) {
        const int si = __shfl_sync(kAll, id, __ffs(todo) - 1);
        if (key_lt(kBig, si, tau, tau_i)) {
          list_insert(lv, li, kBig, si, k, lane);
          tau = __shfl_sync(kAll, lv, k - 1);
          tau_i = __shfl_sync(kAll, li, k - 1);
        }
      }
    }
  }

  if (lane < k) {
    a.idx_new[row * k + lane] = li;
    a.dist_new[row * k + lane] = lv;
    a.flags_new[row * k + lane] = li != my_old ? 1 : 0;
  }
  const int nch = __popc(__ballot_sync(kAll, lane < k && li != my_old));
  if (lane == 0 && nch) atomicAdd(a.changed, (unsigned long long)nch);
}

int select_rows(const SelectArgs& a, cudaStream_t stream) {
  const unsigned blocks = (unsigned)ceil_div(a.n, kSelWarps);
  const int cols = a.k * a.j_nn;
  if (cols <= 8 * 32)
    select_rows_kernel<8><<<blocks, kSelWarps * 32, 0, stream>>>(a);
  else if (cols <= 16 * 32)
    select_rows_kernel<16><<<blocks, kSelWarps * 32, 0, stream>>>(a);
  else
    select_rows_kernel<32><<<blocks, kSelWarps * 32, 0, stream>>>(a);
  UMAPB_LAUNCH_CHECK("nnd_select kernel");
  count_launches(1);
  return UMAPB_OK;
}

}  // namespace nnd
}  // namespace umapb
