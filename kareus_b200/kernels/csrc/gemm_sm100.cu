// bf16 GEMM for sm_100a: C[M,N] (+)= A[M,K] * B[N,K]^T with fp32 accumulation in tensor memory.
//
// Persistent, warp-specialised kernel, one CTA per SM:
//   warp 0      TMA producer   (cp.async.bulk.tensor into a 4-stage, 128B-swizzled smem ring)
//   warp 1      MMA issuer     (tcgen05.mma 128xBNx16, one thread; TMEM allocation)
//   warps 2..5  epilogue       (tcgen05.ld of the accumulator, convert, store / accumulate)
// Two accumulator buffers in TMEM let the epilogue of tile i overlap the main loop of tile i+1.
//
// Both operands may be K-major (row = output index, K contiguous) or MN-major (row = K, output
// index contiguous), which covers fprop (x·Wᵀ), dgrad (dy·W) and wgrad (dyᵀ·x) without
// transposing anything in memory.  This is the role of the reference's cuBLASLt wrapper
// (3rdparty/TransformerEngine/transformer_engine/common/gemm/cublaslt_gemm.cu; layouts TN/NN/NT
// at kareus/transformer_engine/pytorch/ops/basic/basic_linear.py:572-582,848-859,899-909).
#include "sm100.cuh"
#include "launch.h"
#include "pdl.cuh"
#include "host_utils.h"
#include "native_calls.h"
#include "gemm_plan.h"
#include <stdlib.h>

namespace kb {

constexpr int GEMM_BM = 128;
constexpr int GEMM_BK = 64;
constexpr int GEMM_STAGES = 4;
constexpr int GEMM_THREADS = 192;

template <int BN>
struct GemmSmem {
  static constexpr int A_BYTES = GEMM_BM * GEMM_BK * 2;
  static constexpr int B_BYTES = BN * GEMM_BK * 2;
  static constexpr int STAGE_BYTES = A_BYTES + B_BYTES;
  static constexpr int TILE_BYTES = STAGE_BYTES * GEMM_STAGES;
  static constexpr int BAR_BYTES = 256;
  static constexpr int TOTAL = TILE_BYTES + BAR_BYTES + 4 * 4096 + 1024;  // + epilogue staging + alignment slack
};

// Tile rasterisation: m-tiles are taken in groups of `group_m`; inside a group the m index runs
// fastest.  The 148 tiles in flight then cover a near-square patch of C whose A and B panels fit in
// L2 together, instead of streaming the whole of A once per wave.
__device__ __forceinline__ void tile_coords(int t, int tiles_m, int tiles_n, int group_m, int& tm, int& tn) {
  const int per_group = group_m * tiles_n;
  const int g = t / per_group;
  const int first_m = g * group_m;
  const int gsz = min(group_m, tiles_m - first_m);
  const int r = t - g * per_group;
  tm = first_m + r % gsz;
  tn = r / gsz;
}

// Optional epilogue on the fp32 accumulator before it is stored: + bias[col] (bf16, per output
// feature) and then an activation (1: GELU, tanh approximation).  This is the fused forward of
// Linear + Bias (+ activation) of the reference's operator set
// (kareus/transformer_engine/pytorch/ops/basic/basic_linear_bias.py:34-315,
// ops/fused/forward_linear_bias_activation.py:37-213); Llama layers have no bias and pass null.
struct Epilogue {
  const __nv_bfloat16* bias;
  int act;
};
__device__ __forceinline__ void apply_epilogue(uint32_t (&v)[32], const Epilogue& ep, int col0, int N) {
  if (ep.bias == nullptr && ep.act == 0) return;
#pragma unroll
  for (int j = 0; j < 32; ++j) {
    float x = __uint_as_float(v[j]);
    if (ep.bias != nullptr && col0 + j < N) x += __bfloat162float(ep.bias[col0 + j]);
    if (ep.act == 1) x = 0.5f * x * (1.f + tanhf(0.7978845608028654f * x * (1.f + 0.044715f * x * x)));
    v[j] = __float_as_uint(x);
  }
}

// `vec_out`: base and rows of C are 16-byte aligned, so that the epilogue may use 16-byte accesses.
template <int BN, bool A_MN, bool B_MN, bool OUT_F32, bool ACCUM>
__global__ void __launch_bounds__(GEMM_THREADS, 1)
gemm_bf16_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
                 void* __restrict__ Cout, int M, int N, int K, int ldc, bool vec_out, int group_m, int ks, int* status,
                 Epilogue ep) {
  using S = GemmSmem<BN>;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + S::TILE_BYTES);
  uint64_t* empty = full + GEMM_STAGES;
  uint64_t* tfull = empty + GEMM_STAGES;
  uint64_t* tempty = tfull + 2;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(tempty + 2);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const int tiles_m = (M + GEMM_BM - 1) / GEMM_BM;
  const int tiles_n = (N + BN - 1) / BN;
  const int num_tiles = tiles_m * tiles_n;
  const int nk = (K + GEMM_BK - 1) / GEMM_BK;
  // split-K (accumulating outputs only): unit u = (tile u / ks, K part u % ks); every part adds its
  // partial sum to C with reductions, so parts of one tile may run on different SMs at once
  const int num_units = num_tiles * ks;
  constexpr uint32_t TMEM_COLS = (2 * BN <= 32) ? 32 : 2 * BN;

  if (threadIdx.x == 0) {
    for (int i = 0; i < GEMM_STAGES; ++i) {
      mbar_init(&full[i], 1);
      mbar_init(&empty[i], 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(&tfull[i], 1);
      mbar_init(&tempty[i], 4);   // one arrival per epilogue warp
    }
    *abort_flag = 0;
    mbar_fence_init();
  }
  if (warp == 1) tmem_alloc(tmem_slot, TMEM_COLS);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  pdl_begin();

  if (warp == 0) {
    // ------------------------------------------------------------------ producer
    if (elect_one()) {
      prefetch_tmap(&tmA);
      prefetch_tmap(&tmB);
      uint32_t it = 0;
      bool ok = true;
      for (int u = blockIdx.x; u < num_units && ok; u += gridDim.x) {
        int tm, tn;
        tile_coords(u / ks, tiles_m, tiles_n, group_m, tm, tn);
        const int m0 = tm * GEMM_BM;
        const int n0 = tn * BN;
        const int kb0 = split_begin(nk, ks, u % ks), kb1 = split_begin(nk, ks, u % ks + 1);
        for (int kb_ = kb0; kb_ < kb1; ++kb_, ++it) {
          const int s = it % GEMM_STAGES;
          const uint32_t ph = (it / GEMM_STAGES) & 1u;
          if (!mbar_wait(&empty[s], ph ^ 1u, abort_flag, status, ST_TIMEOUT_EMPTY)) { ok = false; break; }
          uint8_t* a_dst = smem + s * S::STAGE_BYTES;
          uint8_t* b_dst = a_dst + S::A_BYTES;
          mbar_expect_tx(&full[s], S::STAGE_BYTES);
          const int k0 = kb_ * GEMM_BK;
          if constexpr (!A_MN) {
            tma_load_2d(a_dst, &tmA, &full[s], k0, m0);
          } else {
#pragma unroll
            for (int j = 0; j < GEMM_BM / 64; ++j) tma_load_2d(a_dst + j * 8192, &tmA, &full[s], m0 + 64 * j, k0);
          }
          if constexpr (!B_MN) {
            tma_load_2d(b_dst, &tmB, &full[s], k0, n0);
          } else {
#pragma unroll
            for (int j = 0; j < BN / 64; ++j) tma_load_2d(b_dst + j * 8192, &tmB, &full[s], n0 + 64 * j, k0);
          }
        }
      }
      if (!ok) {
        // leave no copy in flight: tile loads land within microseconds, give them 200 us
        const uint64_t t0 = globaltimer_ns();
        while (globaltimer_ns() - t0 < 200000ull) {}
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------------ MMA issuer
    constexpr uint32_t idesc = make_idesc_bf16(GEMM_BM, BN, A_MN, B_MN);
    uint32_t it = 0;
    uint32_t tile_i = 0;
    bool ok = true;
    if (elect_one())             // one thread runs the role, see elect_one()
    for (int u = blockIdx.x; u < num_units && ok; u += gridDim.x, ++tile_i) {
      const uint32_t buf = tile_i & 1u;
      const uint32_t bph = (tile_i >> 1) & 1u;
      if (!mbar_wait(&tempty[buf], bph ^ 1u, abort_flag, status, ST_TIMEOUT_TMEM_EMPTY)) { ok = false; break; }
      tc_fence_after();
      const uint32_t d_tmem = tmem_base + buf * BN;
      const int kb0 = split_begin(nk, ks, u % ks), kb1 = split_begin(nk, ks, u % ks + 1);
      for (int kb_ = kb0; kb_ < kb1; ++kb_, ++it) {
        const int s = it % GEMM_STAGES;
        const uint32_t ph = (it / GEMM_STAGES) & 1u;
        if (!mbar_wait(&full[s], ph, abort_flag, status, ST_TIMEOUT_FULL)) { ok = false; break; }
        tc_fence_after();
        const uint32_t a_addr = smem_u32(smem + s * S::STAGE_BYTES);
        const uint32_t b_addr = a_addr + S::A_BYTES;
#pragma unroll
        for (int k = 0; k < GEMM_BK / 16; ++k) {
          const uint64_t ad = A_MN ? make_smem_desc(a_addr + k * 2048, 8192, 1024)
                                   : make_smem_desc(a_addr + k * 32, 16, 1024);
          const uint64_t bd = B_MN ? make_smem_desc(b_addr + k * 2048, 8192, 1024)
                                   : make_smem_desc(b_addr + k * 32, 16, 1024);
          umma_ss(d_tmem, ad, bd, idesc, (kb_ > kb0 || k > 0) ? 1u : 0u);
        }
        umma_commit(&empty[s]);                       // stage reusable once these MMAs retire
        if (kb_ == kb1 - 1) umma_commit(&tfull[buf]); // accumulator complete
      }
    }
    __syncwarp();
  } else {
    // ------------------------------------------------------------------ epilogue (warps 2..5)
    const int q = warp & 3;                 // TMEM lane quarter this warp may read
    uint32_t tile_i = 0;
    bool ok = true;
    for (int u = blockIdx.x; u < num_units && ok; u += gridDim.x, ++tile_i) {
      const uint32_t buf = tile_i & 1u;
      const uint32_t bph = (tile_i >> 1) & 1u;
      int tm, tn;
      tile_coords(u / ks, tiles_m, tiles_n, group_m, tm, tn);
      const int m0 = tm * GEMM_BM;
      const int n0 = tn * BN;
      uint8_t* stg = smem + S::TILE_BYTES + S::BAR_BYTES + q * 4096;     // this warp's staging
      if (!mbar_wait_warp(&tfull[buf], bph, abort_flag, status, ST_TIMEOUT_TMEM_FULL)) { ok = false; break; }
      tc_fence_after();
      const int row = m0 + q * 32 + lane;
      const uint32_t taddr = tmem_base + buf * BN + (static_cast<uint32_t>(q * 32) << 16);
      if constexpr (!OUT_F32) {
        // bf16 output with 16-byte aligned rows: go through this warp's 4 KB of shared memory (32 rows
        // x 128 B, 16-byte units XOR-swizzled by row) so every store instruction writes four full
        // 128-byte row segments instead of 32 scattered 16-byte pieces
        if (vec_out && (N & 7) == 0) {
          __nv_bfloat16* cbase = reinterpret_cast<__nv_bfloat16*>(Cout) + static_cast<size_t>(m0 + q * 32) * ldc;
#pragma unroll 1
          for (int cp = 0; cp < BN / 64; ++cp) {
#pragma unroll
            for (int half = 0; half < 2; ++half) {
              uint32_t v[32];
              tmem_ld_32x32(taddr + (cp * 2 + half) * 32, v);
              tmem_ld_wait();
              apply_epilogue(v, ep, n0 + cp * 64 + half * 32, N);
#pragma unroll
              for (int j = 0; j < 4; ++j) {
                uint4 o;
                o.x = pack_bf16x2(__uint_as_float(v[8 * j + 0]), __uint_as_float(v[8 * j + 1]));
                o.y = pack_bf16x2(__uint_as_float(v[8 * j + 2]), __uint_as_float(v[8 * j + 3]));
                o.z = pack_bf16x2(__uint_as_float(v[8 * j + 4]), __uint_as_float(v[8 * j + 5]));
                o.w = pack_bf16x2(__uint_as_float(v[8 * j + 6]), __uint_as_float(v[8 * j + 7]));
                const int unit = half * 4 + j;
                *reinterpret_cast<uint4*>(stg + lane * 128 + ((unit ^ (lane & 7)) << 4)) = o;
              }
            }
            __syncwarp();
            const int u = lane & 7;
            const int col = n0 + cp * 64 + u * 8;
#pragma unroll
            for (int it4 = 0; it4 < 8; ++it4) {
              const int r = it4 * 4 + (lane >> 3);
              const uint4 o = *reinterpret_cast<const uint4*>(stg + r * 128 + ((u ^ (r & 7)) << 4));
              if (m0 + q * 32 + r < M && col + 8 <= N)
                *reinterpret_cast<uint4*>(cbase + static_cast<size_t>(r) * ldc + col) = o;
            }
            __syncwarp();
          }
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(&tempty[buf]);
          continue;
        }
      }
#pragma unroll 1
      for (int c = 0; c < BN / 32; ++c) {
        uint32_t v[32];
        __syncwarp();                       // rows past the edge store nothing: the warp reads TMEM as a whole again
        tmem_ld_32x32(taddr + c * 32, v);
        tmem_ld_wait();
        const int col = n0 + c * 32;
        if constexpr (!ACCUM) apply_epilogue(v, ep, col, N);
        if (!(col + 32 <= N && vec_out)) {
          // rows that are not 16-byte aligned, or the edge: through the staging buffer (columns XOR-swizzled by row), so
          // that an access takes 32 neighbouring columns of a row and not one column of 32 rows (4096 x 50257 x 3072: fp32
          // 2.03 -> 1.23 ms, with accumulation 5.46 -> 1.54 ms)
          float* st = reinterpret_cast<float*>(stg);
#pragma unroll
          for (int j = 0; j < 32; ++j) st[lane * 32 + (j ^ lane)] = __uint_as_float(v[j]);
          __syncwarp();
          const int rows = min(32, M - (m0 + q * 32));
          if (!OUT_F32 && col + lane < N) {
            __nv_bfloat16* cc = reinterpret_cast<__nv_bfloat16*>(Cout) + static_cast<size_t>(m0 + q * 32) * ldc + col + lane;
#pragma unroll 4
            for (int r = 0; r < rows; ++r) cc[static_cast<long>(r) * ldc] = __float2bfloat16(st[r * 32 + (lane ^ r)]);
          } else if (col + lane < N) {
            float* cc = reinterpret_cast<float*>(Cout) + static_cast<size_t>(m0 + q * 32) * ldc + col + lane;
#pragma unroll 1
            for (int r0 = 0; r0 < rows; r0 += 8, cc += 8L * ldc) {
              float old[8];
              if (ACCUM && ks == 1) {
#pragma unroll
                for (int r = 0; r < 8; ++r)
                  if (r0 + r < rows) old[r] = cc[static_cast<long>(r) * ldc];
              }
#pragma unroll
              for (int r = 0; r < 8; ++r) {
                if (r0 + r >= rows) break;
                const float o = st[(r0 + r) * 32 + (lane ^ (r0 + r))];
                float* p = cc + static_cast<long>(r) * ldc;
                if (ACCUM && ks > 1) atomicAdd(p, o);
                else *p = ACCUM ? old[r] + o : o;
              }
            }
          }
          __syncwarp();
        } else if (row < M && col < N) {
          if constexpr (OUT_F32) {
            float* crow = reinterpret_cast<float*>(Cout) + static_cast<size_t>(row) * ldc + col;
#pragma unroll
            for (int j = 0; j < 8; ++j) {
              float4 o = make_float4(__uint_as_float(v[4 * j]), __uint_as_float(v[4 * j + 1]),
                                     __uint_as_float(v[4 * j + 2]), __uint_as_float(v[4 * j + 3]));
              float4* p = reinterpret_cast<float4*>(crow) + j;
              if constexpr (ACCUM) {
                if (ks > 1) { red_add_f32x4(p, o); continue; }
                float4 old = *p;
                o.x += old.x; o.y += old.y; o.z += old.z; o.w += old.w;
              }
              *p = o;
            }
          } else {
            __nv_bfloat16* crow = reinterpret_cast<__nv_bfloat16*>(Cout) + static_cast<size_t>(row) * ldc + col;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              uint4 o;
              o.x = pack_bf16x2(__uint_as_float(v[8 * j + 0]), __uint_as_float(v[8 * j + 1]));
              o.y = pack_bf16x2(__uint_as_float(v[8 * j + 2]), __uint_as_float(v[8 * j + 3]));
              o.z = pack_bf16x2(__uint_as_float(v[8 * j + 4]), __uint_as_float(v[8 * j + 5]));
              o.w = pack_bf16x2(__uint_as_float(v[8 * j + 6]), __uint_as_float(v[8 * j + 7]));
              reinterpret_cast<uint4*>(crow)[j] = o;
            }
          }
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&tempty[buf]);
    }
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, TMEM_COLS);
  }
}

// ----------------------------------------------------------------------------- host side
// Base and rows of an output that are 16-byte aligned.
static bool aligned_rows(const void* C, int ldc, int out_f32) {
  return (reinterpret_cast<uintptr_t>(C) & 15) == 0 && (ldc & (out_f32 ? 3 : 7)) == 0;
}

template <int BN, bool A_MN, bool B_MN, bool OUT_F32, bool ACCUM>
static int launch_gemm(const void* A, const void* B, void* C, int M, int N, int K, int lda, int ldb, int ldc,
                       int num_sms, int ks, int* status, cudaStream_t stream, Epilogue ep) {
  CUtensorMap tmA, tmB;
  int rc;
  // K-major operand: dims (K, rows), box (64, tile rows).  MN-major: dims (rows, K), box (64, 64).
  if (!A_MN) rc = make_tmap_2d_bf16(&tmA, A, K, M, lda, GEMM_BK, GEMM_BM);
  else       rc = make_tmap_2d_bf16(&tmA, A, M, K, lda, 64, GEMM_BK);
  if (rc) return rc;
  if (!B_MN) rc = make_tmap_2d_bf16(&tmB, B, K, N, ldb, GEMM_BK, BN);
  else       rc = make_tmap_2d_bf16(&tmB, B, N, K, ldb, 64, GEMM_BK);
  if (rc) return rc;
  auto kern = gemm_bf16_kernel<BN, A_MN, B_MN, OUT_F32, ACCUM>;
  constexpr int smem = GemmSmem<BN>::TOTAL;
  static bool configured = false;
  if (!configured) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) return 1000 + static_cast<int>(e);
    configured = true;
  }
  if (!ACCUM || ks < 1) ks = 1;
  const int tiles = ((M + GEMM_BM - 1) / GEMM_BM) * ((N + BN - 1) / BN) * ks;
  int grid = tiles < num_sms ? tiles : num_sms;
  if (grid < 1) grid = 1;
  // m-tiles per group: keep the group's A panel near 40 MB so A and B panels share the 126 MB L2
  int tiles_m = (M + GEMM_BM - 1) / GEMM_BM;
  long panel = (long)GEMM_BM * K * 2;
  int group_m = (int)((40L << 20) / (panel > 0 ? panel : 1));
  if (group_m < 4) group_m = 4;
  if (group_m > tiles_m) group_m = tiles_m;
  KB_LAUNCH_PDL(kern, grid, GEMM_THREADS, smem, stream, tmA, tmB, C, M, N, K, ldc, aligned_rows(C, ldc, OUT_F32), group_m, ks,
            status, ep);
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? 0 : 2000 + static_cast<int>(e);
}

template <int BN, bool A_MN, bool B_MN>
static int dispatch_out(const void* A, const void* B, void* C, int M, int N, int K, int lda, int ldb, int ldc,
                        int out_f32, int accumulate, int num_sms, int ks, int* status, cudaStream_t stream,
                        Epilogue ep) {
  if (out_f32 && accumulate)
    return launch_gemm<BN, A_MN, B_MN, true, true>(A, B, C, M, N, K, lda, ldb, ldc, num_sms, ks, status, stream, ep);
  if (out_f32)
    return launch_gemm<BN, A_MN, B_MN, true, false>(A, B, C, M, N, K, lda, ldb, ldc, num_sms, 1, status, stream, ep);
  if (accumulate) return ST_BAD_ARG;
  return launch_gemm<BN, A_MN, B_MN, false, false>(A, B, C, M, N, K, lda, ldb, ldc, num_sms, 1, status, stream, ep);
}

// ----------------------------------------------------------------------------- tile and split choice
static int g_force_bn = 0, g_force_ks = 0, g_force_single = 0;   // measurement and test overrides, see below

static bool split_allowed() {
  static const bool allow = [] { const char* e = getenv("KB_GEMM_SPLITK"); return !(e && e[0] == '0'); }();
  return allow;
}

// Modelled time of the two-SM kernel at tile width `bn`, in 64-deep K steps of a 256 x 256 tile.
static PairPlan plan_pair_width(int M, int N, int K, int pairs, int bn, bool may_split, bool b_mn = false) {
  // Measured per step: a step moves 16 KB of A and bn / 256 x 16 KB of B into each SM, so narrow tiles are bound by the
  // bytes in flight and not by the tensor pipe (16384 x 6144 x 3072, us per step: 0.41 at 256 columns, 0.30 at 192, 0.23 at
  // 128, 0.17 at 64; with six stages at every width 0.32, 0.24 and 0.175).  MN-major B comes in 64-wide chunks, 192 columns
  // move as much of it as 256 (2048 x 8192 x 3072: 76.6 us at 192 columns, 70.9 at 256).
  static const double step_cost[2][5] = {{0, 0.45, 0.57, 0.75, 1.0}, {0, 0.55, 0.61, 0.83, 1.0}};
  const int nk = (K + GEMM_BK - 1) / GEMM_BK;
  const double step = step_cost[b_mn][bn / 64], fixed = 3.0;
  const long tiles = (long)((M + 255) / 256) * ((N + bn - 1) / bn);
  const long full_waves = tiles / pairs, rest = tiles - full_waves * pairs;
  const double base = full_waves * (nk * step + fixed);
  PairPlan best{bn, 1, 0, base + (rest ? nk * step + fixed : 0.0) + 4.0, false};
  if (may_split && rest)
    for (int ks = 2; ks <= 8 && nk / ks >= 8; ++ks) {
      const long waves = (rest * ks + pairs - 1) / pairs;
      const double t = base + waves * ((nk + ks - 1) / ks * step + fixed) + 4.0;
      if (t < best.cost * 0.97) best = PairPlan{bn, ks, (int)rest, t, false};   // a split must pay for its extra additions
    }
  return best;
}

// The same for `C +=` with parts added in order, in us.  Fitted to 73 weight gradients of 144..16384 x 184..8192, 560 to
// 19152 tokens (within 10 %; the plans it picks take 0.2 % longer than the best width and split of each).  Both operands
// are MN-major there and B comes in 64-wide chunks, which makes 64 and 192 columns dearer than above.  The second launch
// costs 3.8 us and 0.29 us per MB that it moves.
static PairPlan plan_ordered_width(int M, int N, int K, int pairs, int bn, bool may_split) {
  static const double step_us[5] = {0, 0.206, 0.225, 0.298, 0.341}, fixed_us[5] = {0, 0.15, 1.0, 1.85, 2.5};
  const int nk = (K + GEMM_BK - 1) / GEMM_BK;
  const double step = step_us[bn / 64], fixed = fixed_us[bn / 64];
  const long tiles = (long)((M + 255) / 256) * ((N + bn - 1) / bn);
  const long full_waves = tiles / pairs, rest = tiles - full_waves * pairs;
  const double base = full_waves * (nk * step + fixed);
  PairPlan best{bn, 1, 0, base + (rest ? nk * step + fixed : 0.0), true};
  if (may_split && rest)
    for (int ks = 2; ks <= 8 && nk / ks >= 8; ++ks) {
      const long waves = (rest * ks + pairs - 1) / pairs;
      const double mb = rest * 256e-6 * bn * 4 * (ks + 1);
      const double t = base + waves * ((nk + ks - 1) / ks * step + fixed) + 3.8 + 0.29 * mb;
      if (t < best.cost * 0.97) best = PairPlan{bn, ks, (int)rest, t, true};
    }
  return best;
}

// K split of the one-SM kernel, which accumulating outputs take whose rows TMA cannot store: modelled time in 64-deep K
// steps of a 128 x 256 tile (0.6 of it at 128 columns), with 14 + 2 ks steps of fill and epilogue a unit (weight gradients
// of a 3B layer at tensor-parallel sizes 1, 2 and 8).  1000 x 1001 over 8192 tokens: 165 us in one part, 34 in the picked
// number; 640 x 3070 over 16384: 217 and 64.
static int split_single(int M, int N, int K, int num_sms, bool narrow) {
  const int nk = (K + GEMM_BK - 1) / GEMM_BK, bn = narrow ? 128 : 256;
  const long tiles = (long)((M + GEMM_BM - 1) / GEMM_BM) * ((N + bn - 1) / bn);
  auto time = [&](int ks) {
    return (tiles * ks + num_sms - 1) / num_sms * ((nk + ks - 1) / ks * (narrow ? 0.6 : 1.0) + 14.0 + 2.0 * ks);
  };
  int best = 1;
  if (split_allowed())
    for (int ks = 2; ks <= 8 && nk / ks >= 8; ++ks)
      if (time(ks) < 0.97 * time(best)) best = ks;
  return best;
}

// Narrow outputs waste less of the last wave with the 128-wide tile of the one-SM kernel.
static bool narrow_single(int N) { return N <= 128 || (N % 256 != 0 && N % 256 <= 128); }

template <typename F>
static PairPlan best_width(F plan) {
  PairPlan best = plan(g_force_bn ? g_force_bn : 256);
  for (int bn = 192; bn >= 64 && !g_force_bn; bn -= 64) {
    const PairPlan p = plan(bn);
    if (p.cost < best.cost) best = p;
  }
  return best;
}

static PairPlan plan_pair(int M, int N, int K, int pairs, bool b_mn) {
  return best_width([&](int bn) { return plan_pair_width(M, N, K, pairs, bn, false, b_mn); });
}

// Tile width of the one-SM kernel for a plain bf16 output where that is the faster one (0: it is not), from the modelled
// us of both kernels (fitted to 284 forward and input-gradient calls of 64..20000 rows; rms error 8 to 15 %).  Without a
// cluster to start it is 1 us quicker to its first product, and 128-row tiles waste less of a short last wave; per step it
// takes 10 % longer.  776 x 5120 x 3072: 27.7 us on pairs (two waves), 20.7 here (one); 4096 x 1024 x 128: 7.4 and 6.0.  Up to
// two steps of K it was the faster one whatever the number of waves (15720 x 4344 x 128: 52.3 and 44.1).
static const double pair_us[5][3] = {{}, {0.16, 1.0, 4.4}, {0.179, 1.4, 4.3}, {0.245, 1.85, 4.0}, {0.304, 1.95, 4.6}};   // step, wave, call
struct PlainTimes { double pair, w128, w256; };
static PlainTimes plain_times(int M, int N, int K, bool b_mn, int num_sms, int pair_bn) {
  const int nk = (K + GEMM_BK - 1) / GEMM_BK;
  auto waves = [](int M_, int N_, int bm, int bn, int slots) {
    return (long)(((long)((M_ + bm - 1) / bm) * ((N_ + bn - 1) / bn) + slots - 1) / slots);
  };
  const double* c = pair_us[pair_bn / 64];
  // an MN-major B comes in 64-wide chunks, of which 64-wide tiles use half
  return {c[2] + (b_mn && pair_bn == 64 ? 0.6 : 0.0) + waves(M, N, 256, pair_bn, num_sms / 2) * (nk * c[0] + c[1]),
          3.5 + waves(M, N, 128, 128, num_sms) * (nk * 0.275 + 0.95), 3.2 + waves(M, N, 128, 256, num_sms) * (nk * 0.337 + 2.2)};
}
static int single_width(int M, int N, int K, bool b_mn, int num_sms, int pair_bn) {
  const PlainTimes t = plain_times(M, N, K, b_mn, num_sms, pair_bn);
  if ((K + GEMM_BK - 1) / GEMM_BK > 2 && (t.w128 < t.w256 ? t.w128 : t.w256) >= 0.97 * t.pair) return 0;
  return t.w128 < t.w256 ? 128 : 256;
}

static int g_force_swiglu = 0;      // measurement and test aid, see kb_gemm_swiglu_force
static const double long_us[2][6][3] = {   // step, wave, call of 64, 128, 192, 256 columns on pairs, 128 and 256 on one SM
    {{0.186, 0.6, 11.8}, {0.242, 0.99, 3.4}, {0.309, 1.33, 3.0}, {0.385, 1.62, 1.9}, {0.331, 0.53, 14.0}, {0.471, 1.29, 7.5}},
    {{0.215, 1.0, 13.6}, {0.232, 1.26, 9.7}, {0.33, 1.61, 8.3}, {0.368, 1.93, 5.6}, {0.339, 0.69, 12.1}, {0.478, 1.66, 9.0}}};
// Kernel and width of a plain bf16 output: the width (64..256) of pairs, or negative that (128, 256) of the one-SM kernel; `us`:
// modelled time.  The table above was fitted to calls of up to about 50 us; longer ones run at lower clocks, and wide tiles,
// which move fewer bytes for a product, lose less: fitted again to 133 calls of 45 to 700 us (rms 9 to 20 %) the picks take
// 1.1 % longer than the best kernel and width of each, by the first table 3.6 % (3934 x 14264 x 5640: one-SM 668, pairs of 256
// columns 521; input gradient 11384 x 2072 x 2584: 192 columns 137, 256 columns 120).
static int plain_choice(int M, int N, int K, bool b_mn, int num_sms, double* us) {
  const int pairs = num_sms / 2, bn = plan_pair(M, N, K, pairs, b_mn).bn, nk = (K + GEMM_BK - 1) / GEMM_BK;
  const PlainTimes t = plain_times(M, N, K, b_mn, num_sms, bn);
  const int one = N % 8 ? 0 : single_width(M, N, K, b_mn, num_sms, bn);
  *us = one == 128 ? t.w128 : one ? t.w256 : t.pair;
  if (*us < 50.0 || nk <= 2 || g_force_bn) return one ? -one : bn;
  int best = 0;
  for (int i = 0; i < (N % 8 ? 4 : 6); ++i) {
    const int width = i < 4 ? 64 * (i + 1) : 128 * (i - 3), rows = i < 4 ? 256 : 128, slots = i < 4 ? pairs : num_sms;
    const long waves = ((long)((M + rows - 1) / rows) * ((N + width - 1) / width) + slots - 1) / slots;
    const double* c = long_us[b_mn][i];
    const double x = waves * (nk * c[0] + c[1]) + c[2];
    if (!best || x < *us) {
      *us = x;
      best = i < 4 ? width : -width;
    }
  }
  return best;
}

static int g_force_parts = 0, g_force_parts_bn = 0;   // measurement and test aid, see kb_gemm_parts_force
// Plan of a bf16 output with a workspace: the tiles after the last full wave in K parts that a second kernel adds in order, where
// the model says that this is faster than the best unsplit plan.  Two kinds of shapes gain: long sums over few tiles (203 x 504 x
// 15384 85 → 24 us, 128 x 1024 x 8192 28 → 18) and long sums whose last wave is short (3800 x 2048 x 12288 154 → 136; the
// 4096 x 3072 input gradient of a 128256-word vocabulary 2233 → 2062).  Us per step, wave and MB of partial sums (written once, read
// once) fitted to 3400 calls of 160 shapes (64..20000 rows, 1024..96000 deep; rms 8 to 13 %); unsplit times below 50 us are
// 10 % too short there.  Over those shapes the picks take 0.82 of the unsplit time, the best ones 0.79, the worst 1.04 of it
// (`route_sweep` of kernels/profile_cases.py times every kernel, width and a range of parts for drawn layers).
static PairPlan plan_parts(int M, int N, int K, bool b_mn, int num_sms) {
  static const double cost[2][5][3] = {{{}, {0.187, 1.39, 0.11}, {0.22, 2.6, 0.05}, {0.288, 2.1, 0.14}, {0.361, 2.06, 0.164}},
                                       {{}, {0.222, 0.0, 0.45}, {0.227, 0.44, 0.32}, {0.31, 1.16, 0.28}, {0.344, 1.6, 0.21}}};
  const int nk = (K + GEMM_BK - 1) / GEMM_BK, pairs = num_sms / 2;
  double plain;
  const int choice = plain_choice(M, N, K, b_mn, num_sms, &plain);
  PairPlan best{choice > 0 ? choice : 256, 1, 0, (plain < 50.0 ? 1.1 : 1.0) * plain, false};        // unsplit: the caller picks by plain_choice
  double best_us = 0.95 * best.cost;
  // callers without room for 16 steps of 64 do not ask for a workspace
  if (K < 1024 || !split_allowed() || g_force_parts == 1 || g_force_bn || g_force_single) return best;
  for (int bn = 256; bn >= 64; bn -= 64) {
    if (g_force_parts_bn && bn != g_force_parts_bn) continue;
    const double* c = cost[b_mn][bn / 64];
    const long tiles = (long)((M + 255) / 256) * ((N + bn - 1) / bn), full = tiles / pairs, rest = tiles - full * pairs;
    for (int ks = 2; rest && ks <= 16 && nk / ks >= 4; ++ks) {
      const PairPlan plan{bn, ks, (int)rest, 0.0, true};
      if (g_force_parts > 1 && ks == g_force_parts) return plan;
      const double mb = plan.bf16_scratch_floats() * 4e-6;
      if (mb > 64.0) break;
      const long waves = (rest * ks + pairs - 1) / pairs;
      const double us = 7.0 + full * (nk * c[0] + c[1]) + waves * ((nk + ks - 1) / ks * c[0] + c[1]) + c[2] * mb;
      if (us < best_us) {
        best_us = us;
        best = plan;
        best.cost = us;
      }
    }
  }
  return best;
}

// Is the activation in the epilogue faster than the product followed by a kernel of its own?  The product is taken as it would run:
// plain_choice, or in K parts, which the epilogue cannot have; both sides by the same table.  A 256-column tile's epilogue takes
// 4.2 us forward and 12 backward (memory latency; it has eight warps) and runs under the main loop of the next tile, the last one
// alone.  The other constants are fitted to 376 calls of 64..17000 rows of the configured layers and their shards (`swiglu_sweep` of
// kernels/profile_cases.py): the picks take 0.3 % longer than the faster of the two, 13 of them more than 3 %; by unsplit times of
// short calls, as this rule was, 1.6 % forward and 0.5 % backward, 42 of them more than 3 % (on 72 layers drawn later the picks
// take 1.5 and 0.3 % longer; up to 120 rows the forward epilogue would be up to 20 % faster where the rule says no).  Measured, us
// of two kernels / one: forward 324 x 512 → 2 x 1024 7.6 / 9.0, 427 x 3072 → 2 x 4096 28.5 / 23.4, 3798 x 2048 → 2 x 3072 101 / 73;
// backward 148 x 2048 → 3072 12.8 / 14.1, 904 x 4096 → 14336 128 / 135 (in K parts), 4074 x 2048 → 1536 36.1 / 38.5, 7784 x 2048 →
// 3072 127 / 114, 16646 x 2048 → 6144 516 / 390.
// Forward passes with and without storing the product (a recomputing step has both) get one answer: they agree bit for bit.
static bool swiglu_pays(int M, int features, int K, bool backward, int num_sms) {
  if (g_force_swiglu) return g_force_swiglu == 1 || (g_force_swiglu == 2 && !backward);
  const int nk = (K + GEMM_BK - 1) / GEMM_BK, N = backward ? features : 2 * features, pairs = num_sms / 2;
  const PairPlan two = plan_parts(M, N, K, backward, num_sms);
  const int fbn = backward ? plan_pair(M, N, K, pairs, true).bn : 256;
  double us;
  const bool is_long = plain_choice(M, N, K, backward, num_sms, &us) != 0 && us >= 50.0 && nk > 2;
  const double* c = is_long ? long_us[backward][fbn / 64 - 1] : pair_us[fbn / 64];
  const long waves = ((long)((M + 255) / 256) * ((N + fbn - 1) / fbn) + pairs - 1) / pairs;
  const double main_loop = nk * c[0] + c[1], epilogue = (backward ? 12.0 : 4.2) * fbn / 256, last = (backward ? 18.0 : 2.0) * fbn / 256;
  const double fused = c[2] + waves * (main_loop > epilogue ? main_loop : epilogue) + last;
  return (us < 50.0 ? 1.1 : 1.0) * fused < two.cost + (backward ? 1.0 : 3.5) + (backward ? 12.0 : 9.0) * M * features / 5.5e6;
}

// `C +=`.  Where 128-row tiles would not fill the chip once and be split even so, the parts add in L2 as they come: the
// second launch of an ordered sum costs such calls up to a third (1024 x 128 over 4096 rows: 8.4 us, ordered 11.3; 640 x 3072
// over 16384 rows: 55 and 60).  Everything larger repeats bit for bit, which costs 0 to 17 % of a call (16384 x 3072 over
// 16384 rows: 0; 5120 x 3072 over 2048 rows: 9; 2120 x 584 over 5912 rows: 17).  Without a workspace an ordered sum is not
// split, and over fewer than 16 steps nothing is: widths are then picked as for other outputs (3072 x 8192 over 64 rows:
// 27 us, 38 with the fit to long sums).
static PairPlan plan_accumulate(int M, int N, int K, int num_sms, bool workspace) {
  const bool narrow = narrow_single(N);
  const long tiles = (long)((M + GEMM_BM - 1) / GEMM_BM) * ((N + (narrow ? 127 : 255)) / (narrow ? 128 : 256));
  const bool few = tiles <= num_sms && split_single(M, N, K, num_sms, narrow) > 1;
  const int pairs = num_sms / 2;
  PairPlan best = best_width([&](int bn) {
    return few || K <= 15 * GEMM_BK ? plan_pair_width(M, N, K, pairs, bn, few)
               : plan_ordered_width(M, N, K, pairs, bn, workspace && split_allowed());
  });
  best.ordered = !few;
  if (g_force_ks > 0 && (few || workspace)) {
    const int nk = (K + GEMM_BK - 1) / GEMM_BK;
    best.ks = g_force_ks <= nk ? g_force_ks : nk;
    best.split_tiles = ((M + 255) / 256) * ((N + best.bn - 1) / best.bn);
  }
  return best;
}

}  // namespace kb

// Tile width, K split and number of split tiles (those after the last full wave) of the two-SM kernel for an
// accumulating fp32 output of this shape.
extern "C" void kb_gemm_accum_plan(int M, int N, int K, int num_sms, int* bn, int* ks, int* split_tiles) {
  const kb::PairPlan pl = kb::plan_accumulate(M, N, K, num_sms, true);
  *bn = pl.bn;
  *ks = pl.ks;
  *split_tiles = pl.split_tiles;
}

// Tile width that kb_gemm_bf16 uses for a bf16 output of this shape (rows 16-byte aligned): positive on the two-SM kernel,
// negative on the one-SM kernel.
extern "C" int kb_gemm_plan(int M, int N, int K, int b_mn, int num_sms) {
  double us;
  return kb::plain_choice(M, N, K, b_mn != 0, num_sms, &us);
}

// Floats of workspace that kb_gemm_accum_bf16 needs for an output of this shape (0: it splits nothing).
extern "C" long kb_gemm_accum_scratch_floats(int M, int N, int K, int num_sms) {
  using namespace kb;
  if (num_sms <= 0) num_sms = device_sm_count();
  if (M <= 0 || N <= 0 || K <= 0 || num_sms < 2 || g_force_single) return 0;
  return plan_accumulate(M, N, K, num_sms, true).scratch_floats();
}

// Measurement aid: force the tile rows (128 / 256) and K split of accumulating GEMMs; ks = 0 returns to the model.
extern "C" void kb_gemm_accum_force(int tile_rows, int ks) {
  kb::g_force_single = ks > 0 && tile_rows == 128 ? 256 : 0;
  kb::g_force_ks = ks;
}

// Measurement aid: force the tile width of the two-SM kernel (64..256), or with a negative width the one-SM
// kernel (-128 / -256); 0 returns to the model.
extern "C" void kb_gemm_force_width(int bn) {
  kb::g_force_bn = bn > 0 ? bn : 0;
  kb::g_force_single = bn < 0 ? -bn : 0;
}

// C[M,N] (+)= op(A) * op(B)^T.
//   a_mn = 0: A is [M, K] row-major (lda = row stride in elements); a_mn = 1: A is stored [K, M].
//   b_mn = 0: B is [N, K] row-major;                                b_mn = 1: B is stored [K, N].
//   out_f32: C is fp32 (else bf16); accumulate: C += (fp32 only).  num_sms limits the grid.
// Strides must be multiples of 8 elements and base pointers 16-byte aligned (TMA rules).
// kb_gemm_bias_act_bf16 adds the epilogue: bias (bf16 [N], may be null) and act (0 none, 1 GELU); it is not
// available together with accumulate.  kb_gemm_accum_bf16 is C += with a workspace of kb_gemm_accum_scratch_floats()
// floats (16-byte aligned, may be null if that is 0) for the parts of K; kb_gemm_bf16 has none and splits K less often.
namespace kb {
static int gemm_run(const void* A, const void* B, void* C, int M, int N, int K, int a_mn, int lda, int b_mn, int ldb, int ldc,
                    int out_f32, int accumulate, int num_sms, const void* bias, int act, float* work, int* status,
                    cudaStream_t stream, bool parts = false) {
  if (M <= 0 || N <= 0 || K <= 0) return ST_BAD_ARG;
  if ((bias != nullptr || act != 0) && accumulate) return ST_BAD_ARG;
  if (act < 0 || act > 1) return ST_BAD_ARG;
  const Epilogue ep{reinterpret_cast<const __nv_bfloat16*>(bias), act};
  const bool plain = bias == nullptr && act == 0;
  if ((lda & 7) || (ldb & 7) || (reinterpret_cast<uintptr_t>(A) & 15) || (reinterpret_cast<uintptr_t>(B) & 15))
    return ST_BAD_ARG;
  if (num_sms <= 0) num_sms = device_sm_count();
  if (accumulate && !out_f32) return ST_BAD_ARG;
  // The two-SM kernel stores through TMA: 16-byte aligned output rows.
  int single = g_force_single;
  if (plain && aligned_rows(C, ldc, out_f32) && N >= 8 && num_sms >= 2 && !single) {
    const int pairs = num_sms / 2;
    PairPlan pl = accumulate ? plan_accumulate(M, N, K, num_sms, work != nullptr)
                  : parts    ? plan_parts(M, N, K, b_mn != 0, num_sms)
                             : plan_pair(M, N, K, pairs, b_mn != 0);
    if (!out_f32 && !g_force_bn && !(parts && pl.ks > 1)) {
      double us;
      const int choice = plain_choice(M, N, K, b_mn != 0, num_sms, &us);
      if (choice < 0) single = -choice;
      else pl = PairPlan{choice, 1, 0, us, false};
    }
    if (!single)
      return gemm_pair_dispatch(A, B, C, M, N, K, a_mn, lda, b_mn, ldb, ldc, out_f32, accumulate, pl, pairs, work, status,
                                stream);
  }
  const bool narrow = single ? single == 128 : narrow_single(N);
  int ks = accumulate ? split_single(M, N, K, num_sms, narrow) : 1;
  if (g_force_ks > 0 && accumulate) ks = g_force_ks <= (K + GEMM_BK - 1) / GEMM_BK ? g_force_ks : (K + GEMM_BK - 1) / GEMM_BK;
#define KB_GO(BN_)                                                                                         \
  do {                                                                                                     \
    if (!a_mn && !b_mn) return dispatch_out<BN_, false, false>(A, B, C, M, N, K, lda, ldb, ldc, out_f32, accumulate, num_sms, ks, status, stream, ep); \
    if (!a_mn && b_mn) return dispatch_out<BN_, false, true>(A, B, C, M, N, K, lda, ldb, ldc, out_f32, accumulate, num_sms, ks, status, stream, ep);   \
    if (a_mn && !b_mn) return dispatch_out<BN_, true, false>(A, B, C, M, N, K, lda, ldb, ldc, out_f32, accumulate, num_sms, ks, status, stream, ep);   \
    return dispatch_out<BN_, true, true>(A, B, C, M, N, K, lda, ldb, ldc, out_f32, accumulate, num_sms, ks, status, stream, ep);                       \
  } while (0)
  if (narrow) KB_GO(128);
  KB_GO(256);
#undef KB_GO
}
}  // namespace kb

extern "C" int kb_gemm_bias_act_bf16(const void* A, const void* B, void* C, int M, int N, int K, int a_mn, int lda,
                                     int b_mn, int ldb, int ldc, int out_f32, int accumulate, int num_sms,
                                     const void* bias, int act, int* status, cudaStream_t stream) {
  return kb::gemm_run(A, B, C, M, N, K, a_mn, lda, b_mn, ldb, ldc, out_f32, accumulate, num_sms, bias, act, nullptr, status,
                      stream);
}

extern "C" int kb_gemm_accum_bf16(const void* A, const void* B, float* C, int M, int N, int K, int a_mn, int lda, int b_mn,
                                  int ldb, int ldc, int num_sms, float* work, int* status, cudaStream_t stream) {
  return kb::gemm_run(A, B, C, M, N, K, a_mn, lda, b_mn, ldb, ldc, 1, 1, num_sms, nullptr, 0, work, status, stream);
}

// bf16 output with a workspace of kb_gemm_scratch_floats() floats (16-byte aligned; none where that is 0) for the K parts of its
// last tiles.
extern "C" long kb_gemm_scratch_floats(int M, int N, int K, int b_mn, int num_sms) {
  using namespace kb;
  if (num_sms <= 0) num_sms = device_sm_count();
  if (M <= 0 || N <= 0 || K <= 0 || num_sms < 2) return 0;
  return plan_parts(M, N, K, b_mn != 0, num_sms).bf16_scratch_floats();
}
extern "C" int kb_gemm_work_bf16(const void* A, const void* B, void* C, int M, int N, int K, int a_mn, int lda, int b_mn, int ldb,
                                 int ldc, int num_sms, float* work, int* status, cudaStream_t stream) {
  return kb::gemm_run(A, B, C, M, N, K, a_mn, lda, b_mn, ldb, ldc, 0, 0, num_sms, nullptr, 0, work, status, stream, work != nullptr);
}
// Measurement and test aid: K parts of the last tiles of bf16 outputs (1: none, 0: by the model) and their width (0: any).
extern "C" void kb_gemm_parts_force(int ks, int bn) {
  kb::g_force_parts = ks;
  kb::g_force_parts_bn = bn;
}

extern "C" int kb_gemm_bf16(const void* A, const void* B, void* C, int M, int N, int K, int a_mn, int lda,
                            int b_mn, int ldb, int ldc, int out_f32, int accumulate, int num_sms, int* status,
                            cudaStream_t stream) {
  return kb::gemm_run(A, B, C, M, N, K, a_mn, lda, b_mn, ldb, ldc, out_f32, accumulate, num_sms, nullptr, 0, nullptr, status,
                      stream);
}

// Logits of a vocabulary shard and the statistics of their rows that a cross entropy needs: maximum, sum of exponentials and
// target logit, in the epilogue of the product (see RowStats in gemm_pair_sm100.cu).  A [M, K], B [N, K], C [M, N] contiguous
// (N a multiple of 8) or null; targets are columns plus vocab_start.  With `weight` *loss is the weighted sum of the rows'
// losses (statistics of the whole vocabulary only).  `part` holds kb_gemm_row_stats_floats() floats.
extern "C" long kb_gemm_row_stats_floats(int M, int N, int K) {
  using namespace kb;
  return M <= 0 || N <= 0 || K <= 0 ? 0 : row_stats_floats(M, N, plan_pair(M, N, K, device_sm_count() / 2, false).bn);
}
extern "C" int kb_gemm_row_stats(const void* A, const void* B, void* C, int M, int N, int K, int lda, int ldb,
                                 const long* targets, long vocab_start, float* part, float* omax, float* osum, float* otgt,
                                 const float* weight, float* loss, int* status, cudaStream_t stream) {
  using namespace kb;
  if (M <= 0 || N <= 0 || K <= 0 || (N & 7) || (lda & 7) || (ldb & 7)) return ST_BAD_ARG;
  if ((reinterpret_cast<uintptr_t>(A) | reinterpret_cast<uintptr_t>(B) | reinterpret_cast<uintptr_t>(C) |
       reinterpret_cast<uintptr_t>(part)) & 15)
    return ST_BAD_ARG;
  const int pairs = device_sm_count() / 2;
  return gemm_pair_row_stats(A, B, C, M, N, K, lda, ldb, plan_pair(M, N, K, pairs, false), pairs, targets, vocab_start, part, omax,
                             osum, otgt, weight, loss, status, stream);
}

// SwiGLU in the epilogue of the GEMM beside it (see SwigluOut in gemm_pair_sm100.cu).  A [M, K], B [2 * features, K], X [M, 2 *
// features] (or null), H [M, features]; backward: A [M, K], B [K, features], X and dX [M, 2 * features].  X, H and dX are
// contiguous, features a multiple of 8.  kb_gemm_swiglu_pays: is that the faster way?
extern "C" int kb_gemm_swiglu_pays(int M, int features, int K, int backward) {
  using namespace kb;
  if (M <= 0 || features <= 0 || K <= 0 || (features & 7) || features > (1 << 29)) return 0;
  return swiglu_pays(M, features, K, backward != 0, device_sm_count()) ? 1 : 0;
}
// Measurement and test aid: 0 by the rule, 1 the epilogue for every shape, 2 forward only, 3 never.
extern "C" void kb_gemm_swiglu_force(int how) { kb::g_force_swiglu = how; }

static bool swiglu_args_ok(int M, int features, int K, int lda, int ldb, const void* A, const void* B, const void* X, const void* Y) {
  return M > 0 && features > 0 && K > 0 && features <= (1 << 29) && !((features | lda | ldb) & 7) &&
         !((reinterpret_cast<uintptr_t>(A) | reinterpret_cast<uintptr_t>(B) | reinterpret_cast<uintptr_t>(X) |
            reinterpret_cast<uintptr_t>(Y)) & 15);
}
extern "C" int kb_gemm_swiglu(const void* A, const void* B, void* X, void* H, int M, int features, int K, int lda, int ldb, int* status,
                              cudaStream_t stream) {
  using namespace kb;
  if (!swiglu_args_ok(M, features, K, lda, ldb, A, B, X, H) || !H) return ST_BAD_ARG;
  return gemm_pair_swiglu(A, B, X, H, M, features, K, lda, ldb, device_sm_count() / 2, status, stream);
}
extern "C" int kb_gemm_swiglu_bwd(const void* A, const void* B, const void* X, void* dX, int M, int features, int K, int lda, int ldb,
                                  int* status, cudaStream_t stream) {
  using namespace kb;
  if (!swiglu_args_ok(M, features, K, lda, ldb, A, B, X, dX) || !X || !dX) return ST_BAD_ARG;
  const int pairs = device_sm_count() / 2;
  return gemm_pair_swiglu_bwd(A, B, X, dX, M, features, K, lda, ldb, plan_pair(M, features, K, pairs, true), pairs, status, stream);
}
