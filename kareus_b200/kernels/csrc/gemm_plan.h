// Tile width and K split of the two-SM GEMM (gemm_pair_sm100.cu), chosen on the host.
#pragma once
#include <cuda_runtime.h>

namespace kb {

struct PairPlan {
  int bn;            // tile width: 64, 128, 192 or 256
  int ks;            // K parts of each split tile (accumulating outputs only; 1: no split)
  int split_tiles;   // tiles that are split: the ones left over after the full waves
  double cost;       // modelled time, for comparing widths
  bool ordered;      // the parts of a tile are added in a fixed order (through a workspace), not as they come
  // fp32 partial sums that the parts after the first leave
  long scratch_floats() const { return ordered ? (long)split_tiles * (ks - 1) * 256 * bn : 0; }
};

// `work` holds pl.scratch_floats() floats (16-byte aligned; unused where that is 0).
int gemm_pair_dispatch(const void* A, const void* B, void* C, int M, int N, int K, int a_mn, int lda, int b_mn, int ldb,
                       int ldc, int out_f32, int accumulate, const PairPlan& pl, int pairs, float* work, int* status,
                       cudaStream_t stream);

}  // namespace kb
