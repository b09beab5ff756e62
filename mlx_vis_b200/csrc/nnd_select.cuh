// The row update of a full-path NNDescent iteration from the blocked join's distances
// (nnd_select.cu), called by nndescent.cu.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

namespace umapb {
namespace nnd {

struct SelectArgs {
  const int32_t* idx_old;   // (n, k)
  const float* dist_old;    // (n, k): stored distances, read unless curd is given
  const float* curd;        // nullable: recomputed distances of the current lists (n, k)
  const int32_t* order;     // nullable: row handled by warp slot r
  const float* nnbuf;       // (n, k * j_nn)
  const int32_t* off;       // nullable (no reverse candidates): n + 1 bucket offsets by source
  const int32_t* entries;   // i * 32 + p, bucketed by source
  const float* entd;        // distance of entry (i, p) to its source, in bucket order
  const float* d0;          // (n): distance to row 0 (the reference's zero padding)
  int64_t n;
  int k, j_nn;
  uint32_t magic;           // 2^20 / j_nn + 1: column / j_nn by a multiply
  int32_t* idx_new;
  float* dist_new;
  uint8_t* flags_new;
  unsigned long long* changed;
};

// Enqueues the update of all rows (k <= 32).
int select_rows(const SelectArgs& a, cudaStream_t stream);

}  // namespace nnd
}  // namespace umapb
