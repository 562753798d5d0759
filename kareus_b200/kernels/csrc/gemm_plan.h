// Tile width and K split of the two-SM GEMM (gemm_pair_sm100.cu), chosen on the host.
#pragma once
#include <cuda_runtime.h>

namespace kb {

struct PairPlan {
  int bn;            // tile width: 64, 128, 192 or 256
  int ks;            // K parts of each split tile (1: no split)
  int split_tiles;   // tiles that are split: the ones left over after the full waves
  double cost;       // modelled time, for comparing widths
  bool ordered;      // the parts of a tile are added in a fixed order (through a workspace), not as they come
  // fp32 partial sums in the workspace: of an accumulating output those of the parts after the first, of a bf16 output all
  long scratch_floats() const { return ordered ? (long)split_tiles * (ks - 1) * 256 * bn : 0; }
  long bf16_scratch_floats() const { return ks > 1 ? (long)split_tiles * ks * 256 * bn : 0; }
};

// `work` holds pl.scratch_floats() floats, for a bf16 output pl.bf16_scratch_floats() (16-byte aligned; unused where that is 0).
int gemm_pair_dispatch(const void* A, const void* B, void* C, int M, int N, int K, int a_mn, int lda, int b_mn, int ldb,
                       int ldc, int out_f32, int accumulate, const PairPlan& pl, int pairs, float* work, int* status,
                       cudaStream_t stream);

// bf16 C = A * B^T (both K-major; null: the product is not stored) and the softmax statistics of its rows, see RowStats in
// gemm_pair_sm100.cu.  `part`: row_stats_floats() floats, 16-byte aligned.  With `weight` ([M]) *loss becomes the
// sum of weight * (max + log(sum) - target).
inline long row_stats_floats(int M, int N, int bn) { return 4L * ((N + bn - 1) / bn) * M + (M + 31) / 32; }
int gemm_pair_row_stats(const void* A, const void* B, void* C, int M, int N, int K, int lda, int ldb, const PairPlan& pl,
                        int pairs, const long* targets, long first_col, float* part, float* omax, float* osum, float* otgt,
                        const float* weight, float* loss, int* status, cudaStream_t stream);

// H [M, features] = silu(gate) * up of [gate | up] = A [M, K] * B [2 * features, K]^T, which goes to X ([M, 2 * features]) unless X
// is null.
int gemm_pair_swiglu(const void* A, const void* B, void* X, void* H, int M, int features, int K, int lda, int ldb, int pairs,
                     int* status, cudaStream_t stream);
// dX [M, 2 * features] = gradient of X = [gate | up] when that of silu(gate) * up is A [M, K] * B [K, features].
int gemm_pair_swiglu_bwd(const void* A, const void* B, const void* X, void* dX, int M, int features, int K, int lda, int ldb,
                         const PairPlan& pl, int pairs, int* status, cudaStream_t stream);

}  // namespace kb
