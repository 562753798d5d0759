// bf16 GEMM on pairs of SMs: one 256 x BN output tile per two-CTA cluster (tcgen05 cta_group::2).
//
// Both CTAs of a cluster work on one instruction stream: the leader (even rank) issues M = 256 MMAs
// whose A rows 0..127 / 128..255 and B rows 0..BN/2-1 / BN/2..BN-1 come from the shared memory of
// CTA 0 / CTA 1, and each CTA keeps its 128 rows of the accumulator in its own TMEM.  Per SM and
// 64-deep K step that is 16 KB of A and at most 16 KB of B through L2 and shared memory for
// 512 tensor clocks, half of the B traffic of a 128x256 tile on one SM, which leaves room in TMEM
// for two accumulators (the epilogue of a tile runs under the main loop of the next) and in shared
// memory for six stages, up to nine at narrower tiles.
//
//   warp 0      TMA producer of this CTA's halves (both CTAs count on the leader's `full` barriers)
//   warp 1      MMA issuer (leader CTA only); allocates TMEM in both CTAs
//   warps 2..9  epilogue: TMEM → registers → 4 KB of swizzled shared memory per warp → TMA store
//               (bf16 / fp32 output) or TMA reduce-add (fp32 `C +=`: the addition happens in L2, so
//               nobody waits for the old value)
//
// K parts of a tile.  A bf16 output sums them from a workspace in a second small kernel, in order (EPI_PARTS).  `C +=`, ordered: the
// first part adds to C, the others store their sums to a workspace, which a second small kernel adds part by part, so that every
// run gives the same bits.  Not ordered: all parts add in L2 as they come; this is for outputs of few tiles, where the second launch
// would cost a third of the time (see gemm_sm100.cu).
//
// BN is a run-time multiple of 64 (64..256): the launcher picks the width whose last wave is fullest.
// Loads use no multicast: every CTA fetches its own halves.
//
// What bounds it: at 256 columns the tensor pipe (519 clocks per 64-deep step of 512 needed) and with it the
// power limit; below that the 64 B per clock that reach an SM.  bf16, us before (one-SM 128x256 and 256x256
// tiles) / now, one B200 in a loop: 16384 x 16384 x 3072 forward 1180 / 1023, input gradient 1282 / 1154,
// weight gradient 1523 / 1093; weight gradients 5120 x 3072 488 / 344, 12288 x 2048 (7600 tokens) 502 / 263,
// 128256 x 3072 (4096 tokens) 4479 / 2335; 640-wide QKV shard 117 / 68 forward.
#include "sm100.cuh"
#include "launch.h"
#include "pdl.cuh"
#include "host_utils.h"
#include "gemm_plan.h"

namespace kb {

constexpr int GP_BM = 256;                     // rows of a tile (128 per CTA)
constexpr int GP_BK = 64;
constexpr int GP_MAX_STAGES = 9;
constexpr int GP_EPI_WARPS = 8;                // 4 TMEM lane quarters x 2 sets of column slabs
constexpr int GP_THREADS = (2 + GP_EPI_WARPS) * 32;
constexpr int GP_A_BYTES = 128 * GP_BK * 2;    // 16 KB: this CTA's rows of A
constexpr int GP_TILE_BYTES = 6 * (GP_A_BYTES + 128 * GP_BK * 2);   // ring: six stages at BN = 256, more at narrower tiles
// This CTA's rows of B (BN / 2 of them); MN-major B comes in whole 64-wide chunks.
__host__ __device__ constexpr int gp_b_bytes(int bn, bool b_mn) {
  return b_mn ? ((bn / 2 + 63) / 64) * 64 * GP_BK * 2 : bn / 2 * GP_BK * 2;
}
constexpr int GP_STG_BYTES = GP_EPI_WARPS * 4096;
constexpr int GP_SMEM = GP_TILE_BYTES + GP_STG_BYTES + 256 + 1024;
static_assert(GP_SMEM <= 227 * 1024, "shared memory per CTA");

// Work unit u of a launch → tile and K range.  The first `whole` units are whole tiles; the remaining
// tiles are cut into `ks` K parts each, part-major (all tiles of part 0, then part 1, ...), so that the
// clusters that run side by side walk the same K range of neighbouring tiles and share operands in L2.
struct PairWork {
  int tiles_m, tiles_n, group_m, nk, whole, split_tiles, ks;
  bool ordered;
  __device__ __forceinline__ int units() const { return whole + split_tiles * ks; }
  // slab of the workspace (256 x bn floats) that unit u stores to, negative if it goes to C
  __device__ __forceinline__ int slab(int u) const { return ordered ? u - whole - split_tiles : -1; }
  __device__ __forceinline__ void decode(int u, int& tm, int& tn, int& kb0, int& kb1) const {
    int t;
    if (u < whole) {
      t = u;
      kb0 = 0;
      kb1 = nk;
    } else {
      const int r = u - whole;
      const int part = r / split_tiles;
      t = whole + r - part * split_tiles;
      kb0 = split_begin(nk, ks, part);
      kb1 = split_begin(nk, ks, part + 1);
    }
    coords(t, tm, tn);
  }
  __device__ __forceinline__ void coords(int t, int& tm, int& tn) const {
    // m-tiles are taken in groups of `group_m`; inside a group the m index runs fastest, so the tiles in
    // flight cover a near-square patch of C
    const int per_group = group_m * tiles_n;
    const int g = t / per_group;
    const int first_m = g * group_m;
    const int gsz = min(group_m, tiles_m - first_m);
    const int r = t - g * per_group;
    tm = first_m + r % gsz;
    tn = r / gsz;
  }
};

// What the epilogue does besides storing the product.
enum PairEpilogue : int {
  EPI_NONE = 0,
  EPI_ROW_STATS = 1,    // maximum and sum of exponentials of the row pieces that it stores (see RowStats)
  EPI_SWIGLU = 2,       // silu(gate) * up of a [gate | up] product (see SwigluOut)
  EPI_SWIGLU_BWD = 3,   // from the gradient of silu(gate) * up, which is the product, that of [gate | up]
  EPI_PARTS = 4,        // the tiles after the last full wave are split in K: their parts go to a workspace as fp32 sums
};

// Row statistics of the bf16 product for a softmax over its columns.  A thread of the epilogue has a row of its tile in
// registers, so this costs it arithmetic that hides under the main loop, in place of a pass over the product in
// memory: the maximum and the sum of exp(x - maximum) over the 64-column slabs of this thread go to
// part[2 * column tile + slab parity][row].  x is the product rounded to bf16, as it is stored.  4096 x 128256 x 3072: the product
// takes 2.18 ms with or without them, the pass over it took 229 us; 8997 x 32768 x 2048 without storing it: 134 us of
// statistics and 90 us of stores less.
struct RowStats {
  float2* part;          // [2 * column tiles][M]
  const long* targets;   // [M]: column (plus first_col) whose value goes to `target`, which holds 0 otherwise
  float* target;         // [M]
  long first_col;
  bool store;            // false: the product itself is not wanted
};

// EPI_SWIGLU: a tile has 128 gate columns (B rows that CTA 0 loads) and the up columns of the same features (CTA 1), so
// a thread of the epilogue holds both and stores their activation; the product itself leaves only if it is wanted
// for a backward pass (as halves of a [M, 2 * features] matrix).
// EPI_SWIGLU_BWD: the epilogue fetches gate and up of its columns and stores both gradients; the gradient of the
// activation never reaches memory.
// Everything is rounded to bf16 where the separate kernels store it.  One B200, us with kernels of their own / in the epilogue:
// forward 16384 x 3072 → 2 x 8192 1176 / 1059 (1002 without the product), 3800 x 2048 → 2 x 6144 146 / 123 (117); backward
// 16384 x 3072 → 8192 741 / 604, 3800 x 2048 → 6144 111 / 91.
struct SwigluOut {
  CUtensorMap gate, up;     // boxes of 32 rows x 64 columns
  int features;
  bool store;               // the product is wanted
};
struct SwigluGrad {
  const __nv_bfloat16* x;   // [gate | up] of the forward pass, [M, 2 * features]
  __nv_bfloat16* dx;        // its gradient
};
template <int EPI> struct EpiArgs { struct type {}; };
template <> struct EpiArgs<EPI_ROW_STATS> { using type = RowStats; };
template <> struct EpiArgs<EPI_SWIGLU> { using type = SwigluOut; };
template <> struct EpiArgs<EPI_SWIGLU_BWD> { using type = SwigluGrad; };

__device__ __forceinline__ float2 bf16_pair(uint32_t v) {
  return make_float2(__uint_as_float(v << 16), __uint_as_float(v & 0xffff0000u));
}

__device__ __forceinline__ float ex2_approx(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// 64 accumulator columns of a thread's row as packed bf16 pairs.
__device__ __forceinline__ void pack_row(const uint32_t (&v0)[32], const uint32_t (&v1)[32], uint32_t (&o)[32]) {
#pragma unroll
  for (int j = 0; j < 16; ++j) {
    o[j] = pack_bf16x2(__uint_as_float(v0[2 * j]), __uint_as_float(v0[2 * j + 1]));
    o[16 + j] = pack_bf16x2(__uint_as_float(v1[2 * j]), __uint_as_float(v1[2 * j + 1]));
  }
}

// A warp's slab (32 rows x 128 bytes, a row per thread) into its staging buffer, 16-byte units swizzled by row as the tensor maps
// expect, once the store before it has read the buffer.
__device__ __forceinline__ void put_slab(const uint32_t (&o)[32], uint32_t stg_row, int lane) {
  if (lane == 0) tma_store_wait_read<0>();
  __syncwarp();
#pragma unroll
  for (int j = 0; j < 8; ++j) st_shared_v4(stg_row + ((j ^ (lane & 7)) << 4), o[4 * j], o[4 * j + 1], o[4 * j + 2], o[4 * j + 3]);
  fence_proxy_async_smem();
  __syncwarp();
}

// 32 rows x 64 columns of a matrix, whole 128-byte row segments per access; rows past M and columns past N (a multiple of 8) read
// as zero.
__device__ __forceinline__ void load_slab(const __nv_bfloat16* x, int ld, int row0, int M, int col, int N, int lane, uint4 (&v)[8]) {
  const int unit = lane & 7;
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int r = row0 + i * 4 + (lane >> 3);
    v[i] = make_uint4(0u, 0u, 0u, 0u);
    if (r < M && col + unit * 8 < N) v[i] = *reinterpret_cast<const uint4*>(x + static_cast<size_t>(r) * ld + col + unit * 8);
  }
}
// What load_slab returned into a (free) 4 KB buffer, 16-byte units swizzled by row, and such a buffer out to a matrix.
__device__ __forceinline__ void slab_to_smem(const uint4 (&v)[8], uint8_t* buf, int lane) {
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int r = i * 4 + (lane >> 3);
    *reinterpret_cast<uint4*>(buf + r * 128 + (((lane & 7) ^ (r & 7)) << 4)) = v[i];
  }
}
__device__ __forceinline__ void slab_from_smem(const uint8_t* buf, __nv_bfloat16* x, int ld, int row0, int M, int col, int N, int lane) {
  const int unit = lane & 7;
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int r = i * 4 + (lane >> 3);
    const uint4 v = *reinterpret_cast<const uint4*>(buf + r * 128 + ((unit ^ (r & 7)) << 4));
    if (row0 + r < M && col + unit * 8 < N) *reinterpret_cast<uint4*>(x + static_cast<size_t>(row0 + r) * ld + col + unit * 8) = v;
  }
}

// 1 / (1 + e^-a) of two values.
__device__ __forceinline__ float2 sigmoid2(float2 a) {
  constexpr float L2E = 1.4426950408889634f;
  float2 e = __fmul2_rn(a, make_float2(-L2E, -L2E));
  e = __fadd2_rn(make_float2(ex2_approx(e.x), ex2_approx(e.y)), make_float2(1.f, 1.f));
  float2 r;                                          // keeps subnormal results, unlike a quick division
  asm("rcp.approx.f32 %0, %1;" : "=f"(r.x) : "f"(e.x));
  asm("rcp.approx.f32 %0, %1;" : "=f"(r.y) : "f"(e.y));
  return r;
}

// Adds 64 columns of a row (packed bf16 pairs, the first `valid` of them count) to a running maximum and sum.
__device__ __forceinline__ void add_row_stats(const uint32_t (&o)[32], int valid, float& m, float& s) {
  constexpr float L2E = 1.4426950408889634f;
  float x[64];
#pragma unroll
  for (int j = 0; j < 32; ++j) {
    x[2 * j] = __uint_as_float(o[j] << 16);
    x[2 * j + 1] = __uint_as_float(o[j] & 0xffff0000u);
  }
  if (valid < 64) {
#pragma unroll
    for (int j = 0; j < 64; ++j)
      if (j >= valid) x[j] = -INFINITY;
  }
  float mx[4] = {m, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
  for (int j = 0; j < 64; j += 8)
#pragma unroll
    for (int h = 0; h < 4; ++h) mx[h] = fmaxf(mx[h], fmaxf(x[j + 2 * h], x[j + 2 * h + 1]));
  const float nm = fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3]));
  const float base = nm == -INFINITY ? 0.f : nm;
  float2 acc[2] = {make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
#pragma unroll
  for (int j = 0; j < 32; ++j) {
    float2 e = __fmul2_rn(__fadd2_rn(make_float2(x[2 * j], x[2 * j + 1]), make_float2(-base, -base)), make_float2(L2E, L2E));
    e.x = ex2_approx(e.x);
    e.y = ex2_approx(e.y);
    acc[j & 1] = __fadd2_rn(acc[j & 1], e);
  }
  s = s * ex2_approx((m - base) * L2E) + ((acc[0].x + acc[0].y) + (acc[1].x + acc[1].y));
  m = nm;
}

template <bool A_MN, bool B_MN, bool OUT_F32, bool ACCUM, int EPI>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(GP_THREADS, 1)
gemm_pair_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
                 const __grid_constant__ CUtensorMap tmC, const __grid_constant__ CUtensorMap tmW, const PairWork w,
                 const int M, const int N, const int bn, void* const C, const int ldc, int* status,
                 const __grid_constant__ typename EpiArgs<EPI>::type epi) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + GP_TILE_BYTES + GP_STG_BYTES);   // used in the leader
  uint64_t* empty = full + GP_MAX_STAGES;
  uint64_t* tfull = empty + GP_MAX_STAGES;  // [2]
  uint64_t* tempty = tfull + 2;             // [2] used in the leader
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(tempty + 2);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int rank = blockIdx.x & 1;          // rank in the cluster (clusters are consecutive pairs of CTAs)
  const int first = blockIdx.x >> 1, step = gridDim.x >> 1;
  const int num_units = w.units();
  const int half_n = bn >> 1;
  // What a narrow tile waits for is latency times bytes in flight, so it gets all the stages that fit
  const int b_bytes = gp_b_bytes(bn, B_MN), stage_bytes = GP_A_BYTES + b_bytes;
  // one stage less where the epilogue works on two slabs a warp
  constexpr int RING = GP_TILE_BYTES - (EPI == EPI_SWIGLU_BWD ? GP_EPI_WARPS * 4096 : 0);
  const int stages = min(GP_MAX_STAGES, RING / stage_bytes);

  if (threadIdx.x == 0) {
    for (int i = 0; i < GP_MAX_STAGES; ++i) {
      mbar_init(&full[i], 1);
      mbar_init(&empty[i], 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(&tfull[i], 1);
      mbar_init(&tempty[i], 2 * GP_EPI_WARPS);
    }
    *abort_flag = 0;
    mbar_fence_init();
  }
  if (warp == 1) tmem_alloc_pair(tmem_slot, 512);
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();                       // the peer's barriers exist before anything arrives on them
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  pdl_begin();

  if (warp == 0) {
    // ------------------------------------------------------------------ producer (each CTA: its own halves)
    if (elect_one()) {
      prefetch_tmap(&tmA);
      prefetch_tmap(&tmB);
      const int b_chunks = (half_n + 63) >> 6;
      const uint32_t stage_tx = 2u * stage_bytes;     // bytes of both CTAs, counted on the leader's barrier
      const uint32_t full0 = cluster_addr(full, 0);
      int s = 0;
      uint32_t ph = 1;
      bool ok = true;
      for (int u = first; u < num_units && ok; u += step) {
        int tm, tn, kb0, kb1;
        w.decode(u, tm, tn, kb0, kb1);
        const int m0 = tm * GP_BM + rank * 128;
        int n0 = tn * bn + rank * half_n;
        if constexpr (EPI == EPI_SWIGLU) n0 = tn * 128 + rank * epi.features;
        for (int kb_ = kb0; kb_ < kb1; ++kb_) {
          if (!mbar_wait(&empty[s], ph, abort_flag, status, ST_TIMEOUT_EMPTY)) { ok = false; break; }
          uint8_t* a_dst = smem + s * stage_bytes;
          uint8_t* b_dst = a_dst + GP_A_BYTES;
          const uint32_t bar = full0 + s * 8;
          if (rank == 0) mbar_expect_tx(&full[s], stage_tx);
          const int k0 = kb_ * GP_BK;
          if constexpr (!A_MN) {
            tma_load_2d_pair(a_dst, &tmA, bar, k0, m0);
          } else {
            tma_load_2d_pair(a_dst, &tmA, bar, m0, k0);
            tma_load_2d_pair(a_dst + 8192, &tmA, bar, m0 + 64, k0);
          }
          if constexpr (!B_MN) {
            tma_load_2d_pair(b_dst, &tmB, bar, k0, n0);
          } else {
            tma_load_2d_pair(b_dst, &tmB, bar, n0, k0);
            if (b_chunks > 1) tma_load_2d_pair(b_dst + 8192, &tmB, bar, n0 + 64, k0);
          }
          if (++s == stages) { s = 0; ph ^= 1u; }
        }
      }
      if (!ok) {
        // leave no copy in flight: tile loads land within microseconds, give them 200 us
        const uint64_t t0 = globaltimer_ns();
        while (globaltimer_ns() - t0 < 200000ull) {}
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    // ------------------------------------------------------------------ MMA issuer (leader)
    // One thread chosen by elect.sync runs the whole role: with `lane == 0` in its place the four MMAs of
    // a step took 605 clocks at every tile width (512 at 256 columns and 128 at 64 is what they need),
    // because the compiler then cannot keep descriptors and addresses in uniform registers.
    if (rank == 0 && elect_one()) {
      const uint32_t idesc = make_idesc_bf16(GP_BM, bn, A_MN, B_MN);
      const uint32_t smem0 = smem_u32(smem);
      const uint64_t ad0 = A_MN ? make_smem_desc(smem0, 8192, 1024) : make_smem_desc(smem0, 16, 1024);
      const uint64_t bd0 = B_MN ? make_smem_desc(smem0 + GP_A_BYTES, 8192, 1024)
                                : make_smem_desc(smem0 + GP_A_BYTES, 16, 1024);
      constexpr uint64_t ka = (A_MN ? 2048 : 32) >> 4, kb = (B_MN ? 2048 : 32) >> 4;   // descriptor step of 16 in K
      uint32_t tile_i = 0;
      int s = 0;
      uint32_t ph = 0;
      bool ok = true;
      for (int u = first; u < num_units && ok; u += step, ++tile_i) {
        int tm, tn, kb0, kb1;
        w.decode(u, tm, tn, kb0, kb1);
        const uint32_t buf = tile_i & 1u;
        if (!mbar_wait(&tempty[buf], ((tile_i >> 1) & 1u) ^ 1u, abort_flag, status, ST_TIMEOUT_TMEM_EMPTY)) break;
        tc_fence_after();
        const uint32_t d_tmem = tmem_base + buf * 256;
        for (int kb_ = kb0; kb_ < kb1; ++kb_) {
          if (!mbar_wait(&full[s], ph, abort_flag, status, ST_TIMEOUT_FULL)) { ok = false; break; }
          tc_fence_after();
          const uint64_t ad = ad0 + static_cast<uint64_t>(s * (stage_bytes >> 4));
          const uint64_t bd = bd0 + static_cast<uint64_t>(s * (stage_bytes >> 4));
#pragma unroll
          for (int k = 0; k < GP_BK / 16; ++k)
            umma_ss_pair(d_tmem, ad + k * ka, bd + k * kb, idesc, (kb_ > kb0 || k > 0) ? 1u : 0u);
          umma_commit_pair(&empty[s]);                              // both CTAs may refill the stage
          if (kb_ == kb1 - 1) umma_commit_pair(&tfull[buf]);        // both CTAs' halves are complete
          if (++s == stages) { s = 0; ph ^= 1u; }
        }
      }
    }
    __syncwarp();
  } else {
    // ------------------------------------------------------------------ epilogue
    const int q = warp & 3;                   // TMEM lane quarter
    const int h = (warp - 2) >> 2;            // this warp takes the column slabs h, h + 2, ...
    uint8_t* stg = smem + RING + (warp - 2) * (EPI == EPI_SWIGLU_BWD ? 8192 : 4096);
    constexpr int SLAB = OUT_F32 ? 32 : 64;   // output columns of one 128-byte wide slab
    const int slabs = bn / SLAB;
    const uint32_t stg_row = smem_u32(stg) + lane * 128;
    uint32_t tile_i = 0;
    if constexpr (EPI == EPI_SWIGLU_BWD) {
      // Gate and up of the next slab, of this tile or the next, are on their way while one is worked on and while the
      // accumulator is waited for; the gradients take their place in shared memory, a row per thread.
      uint4 vg[8], vu[8];
      auto fetch = [&](int u, int c) {
        int tm, tn, kb0, kb1;
        w.decode(u, tm, tn, kb0, kb1);
        const int row0 = tm * GP_BM + rank * 128 + q * 32, col = tn * bn + c * SLAB;
        load_slab(epi.x, 2 * N, row0, M, col, N, lane, vg);
        load_slab(epi.x + N, 2 * N, row0, M, col, N, lane, vu);
      };
      if (first < num_units && h < slabs) fetch(first, h);
      for (int u = first; u < num_units; u += step, ++tile_i) {
        int tm, tn, kb0, kb1;
        w.decode(u, tm, tn, kb0, kb1);
        const uint32_t buf = tile_i & 1u;
        const int row0 = tm * GP_BM + rank * 128 + q * 32;
        if (!mbar_wait_warp(&tfull[buf], (tile_i >> 1) & 1u, abort_flag, status, ST_TIMEOUT_TMEM_FULL)) break;
        tc_fence_after();
        const uint32_t taddr = tmem_base + buf * 256 + (static_cast<uint32_t>(q * 32) << 16);
#pragma unroll 1
        for (int c = h; c < slabs; c += 2) {
          slab_to_smem(vg, stg, lane);
          slab_to_smem(vu, stg + 4096, lane);
          __syncwarp();
          if (c + 2 < slabs) fetch(u, c + 2);
          else if (u + step < num_units) fetch(u + step, h);
          __syncwarp();                               // rows and columns past the edge are left out lane by lane
          const float2 one = make_float2(1.f, 1.f);
#pragma unroll
          for (int half = 0; half < 2; ++half) {
            uint32_t v[32];
            tmem_ld_32x32(taddr + c * 64 + half * 32, v);
            tmem_ld_wait();
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              uint4* pg = reinterpret_cast<uint4*>(stg + lane * 128 + (((half * 4 + j) ^ (lane & 7)) << 4));
              uint4* pu = reinterpret_cast<uint4*>(reinterpret_cast<uint8_t*>(pg) + 4096);
              uint4 g4 = *pg, u4 = *pu;
              uint32_t* g = reinterpret_cast<uint32_t*>(&g4);
              uint32_t* up = reinterpret_cast<uint32_t*>(&u4);
#pragma unroll
              for (int i = 0; i < 4; ++i) {
                const float2 d = bf16_pair(pack_bf16x2(__uint_as_float(v[8 * j + 2 * i]), __uint_as_float(v[8 * j + 2 * i + 1])));
                const float2 a = bf16_pair(g[i]), sg = sigmoid2(a), ds = __fmul2_rn(d, sg);
                const float2 t = __ffma2_rn(a, __fadd2_rn(one, make_float2(-sg.x, -sg.y)), one);      // 1 + a (1 - sigmoid)
                const float2 da = __fmul2_rn(__fmul2_rn(ds, bf16_pair(up[i])), t), db = __fmul2_rn(ds, a);
                g[i] = pack_bf16x2(da.x, da.y);
                up[i] = pack_bf16x2(db.x, db.y);
              }
              *pg = g4;
              *pu = u4;
            }
          }
          if (c + 2 >= slabs) tc_fence_before();
          __syncwarp();
          if (c + 2 >= slabs && lane == 0) mbar_arrive_cluster(cluster_addr(&tempty[buf], 0));
          const int col = tn * bn + c * SLAB;
          slab_from_smem(stg, epi.dx, 2 * N, row0, M, col, N, lane);
          slab_from_smem(stg + 4096, epi.dx + N, 2 * N, row0, M, col, N, lane);
          __syncwarp();
        }
        if (slabs <= h) {                             // no slab for this warp (narrow tile): release all the same
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive_cluster(cluster_addr(&tempty[buf], 0));
        }
      }
    } else
    for (int u = first; u < num_units; u += step, ++tile_i) {
      int tm, tn, kb0, kb1;
      w.decode(u, tm, tn, kb0, kb1);
      const uint32_t buf = tile_i & 1u;
      const int row0 = tm * GP_BM + rank * 128 + q * 32;
      if (!mbar_wait_warp(&tfull[buf], (tile_i >> 1) & 1u, abort_flag, status, ST_TIMEOUT_TMEM_FULL)) break;
      tc_fence_after();
      const uint32_t taddr = tmem_base + buf * 256 + (static_cast<uint32_t>(q * 32) << 16);
      if constexpr (EPI == EPI_PARTS) {
        if (u >= w.whole) {                           // a K part: 32-column slabs of the workspace
#pragma unroll 1
          for (int c = h; c < bn / 32; c += 2) {
            uint32_t v[32];
            __syncwarp();
            tmem_ld_32x32(taddr + c * 32, v);
            tmem_ld_wait();
            if (c + 2 >= bn / 32) {
              tc_fence_before();
              __syncwarp();
              if (lane == 0) mbar_arrive_cluster(cluster_addr(&tempty[buf], 0));
            }
            put_slab(v, stg_row, lane);
            if (lane == 0) {
              tma_store_2d(&tmW, stg, c * 32, (u - w.whole) * GP_BM + rank * 128 + q * 32);
              tma_store_commit();
            }
          }
          continue;
        }
      }
      if constexpr (EPI == EPI_SWIGLU) {
        // this warp's 64 features: gate at column 64 h of the accumulator, up at 128 + 64 h
        uint32_t g[32], u[32];
        {
          uint32_t v0[32], v1[32];
          tmem_ld_32x32(taddr + h * 64, v0);
          tmem_ld_32x32(taddr + h * 64 + 32, v1);
          tmem_ld_wait();
          pack_row(v0, v1, g);
          tmem_ld_32x32(taddr + 128 + h * 64, v0);
          tmem_ld_32x32(taddr + 128 + h * 64 + 32, v1);
          tmem_ld_wait();
          pack_row(v0, v1, u);
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive_cluster(cluster_addr(&tempty[buf], 0));
        const int col = tn * 128 + h * 64;
        const bool here = row0 < M && col < N;
        if (epi.store) {
          put_slab(g, stg_row, lane);
          if (lane == 0 && here) tma_store_2d(&epi.gate, stg, col, row0);
          if (lane == 0) tma_store_commit();
          put_slab(u, stg_row, lane);
          if (lane == 0 && here) tma_store_2d(&epi.up, stg, col, row0);
          if (lane == 0) tma_store_commit();
        }
#pragma unroll
        for (int j = 0; j < 32; ++j) {
          const float2 a = bf16_pair(g[j]), y = __fmul2_rn(__fmul2_rn(a, sigmoid2(a)), bf16_pair(u[j]));
          g[j] = pack_bf16x2(y.x, y.y);
        }
        put_slab(g, stg_row, lane);
        if (lane == 0 && here) tma_store_2d(&tmC, stg, col, row0);
        if (lane == 0) tma_store_commit();
        continue;
      }
      const int row = row0 + lane;
      float row_max = -INFINITY, row_sum = 0.f;
      long target = -1;                               // column of this tile that holds the row's target
      if constexpr (EPI == EPI_ROW_STATS) {
        if (row < M) target = epi.targets[row] - epi.first_col;
        target = target >= 0 && target < N ? target - tn * bn : -1;
      }
#pragma unroll 1
      for (int c = h; c < slabs; c += 2) {
        uint32_t o[32];
        // TMEM is read by whole warps: what lanes did on their own before (a row's target, the stores of the slab before) ends here
        __syncwarp();
        if constexpr (OUT_F32) {
          tmem_ld_32x32(taddr + c * 32, o);
          tmem_ld_wait();
        } else {
          uint32_t v0[32], v1[32];
          tmem_ld_32x32(taddr + c * 64, v0);
          tmem_ld_32x32(taddr + c * 64 + 32, v1);
          tmem_ld_wait();
          pack_row(v0, v1, o);
        }
        if (c + 2 >= slabs) {
          // this warp's last read of the accumulator: hand it back before the stores go out
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive_cluster(cluster_addr(&tempty[buf], 0));
        }
        if constexpr (EPI == EPI_ROW_STATS) {
          const int col0 = tn * bn + c * SLAB;
          if (col0 < N) add_row_stats(o, min(64, N - col0), row_max, row_sum);
          const long t = target - c * SLAB;
          if (t >= 0 && t < SLAB) {
            uint32_t pick[16];                        // halves by the bits of t: an index would put o into local memory
#pragma unroll
            for (int j = 0; j < 16; ++j) pick[j] = t & 32 ? o[16 + j] : o[j];
#pragma unroll
            for (int n = 8; n > 0; n >>= 1)
#pragma unroll
              for (int j = 0; j < n; ++j) pick[j] = t & (2 * n) ? pick[n + j] : pick[j];
            const uint32_t pair = pick[0];
            epi.target[row] = __uint_as_float(t & 1 ? pair & 0xffff0000u : pair << 16);
          }
          if (!epi.store) continue;
        }
        if (lane == 0) tma_store_wait_read<0>();      // the previous slab has left the staging buffer
        __syncwarp();
#pragma unroll
        for (int j = 0; j < 8; ++j)
          st_shared_v4(stg_row + ((j ^ (lane & 7)) << 4), o[4 * j], o[4 * j + 1], o[4 * j + 2], o[4 * j + 3]);
        fence_proxy_async_smem();
        __syncwarp();
        const int col = tn * bn + c * SLAB;
        // A TMA store ends on a 16-byte boundary: the map of a plain output holds whole units, and the columns after the last
        // one are stored one by one from the staging buffer (what lies behind them may be someone else's).
        const int whole = ACCUM ? N : N & ~(OUT_F32 ? 3 : 7);
        if (!ACCUM && whole < N && whole >= col && whole < col + SLAB && row0 + lane < M) {
          const int unit = (whole - col) / (OUT_F32 ? 4 : 8);
          const uint8_t* src = stg + lane * 128 + ((unit ^ (lane & 7)) << 4);
          for (int j = 0; whole + j < N; ++j) {
            const size_t at = static_cast<size_t>(row0 + lane) * ldc + whole + j;
            if constexpr (OUT_F32) static_cast<float*>(C)[at] = reinterpret_cast<const float*>(src)[j];
            else static_cast<__nv_bfloat16*>(C)[at] = reinterpret_cast<const __nv_bfloat16*>(src)[j];
          }
        }
        if (lane == 0 && row0 < M && col < whole) {   // the tensor map clips what crosses the edge
          if (ACCUM && w.slab(u) >= 0) tma_store_2d(&tmW, stg, c * SLAB, w.slab(u) * GP_BM + rank * 128 + q * 32);
          else if constexpr (ACCUM) tma_reduce_add_2d(&tmC, stg, col, row0);
          else tma_store_2d(&tmC, stg, col, row0);
          tma_store_commit();
        }
      }
      if constexpr (EPI == EPI_ROW_STATS) {
        if (row < M) epi.part[static_cast<size_t>(2 * tn + h) * M + row] = make_float2(row_max, row_sum);
      }
      if (slabs <= h) {                               // no slab for this warp (narrow tile): release all the same
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive_cluster(cluster_addr(&tempty[buf], 0));
      }
    }
    if (lane == 0) tma_store_wait<0>();               // nothing in flight out of shared memory at exit
  }

  tc_fence_before();
  __syncthreads();
  cluster_sync_all();                                 // the peer's MMAs and arrivals no longer touch this CTA
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc_pair(tmem_base, 512);
  }
}

// Row statistics from their pieces: maximum, sum of exponentials, target value (0 where no column of this matrix is the
// target); 32 rows a block, eight threads a row, in a fixed order.  With `weight`, block b also leaves the sum of
// weight * (max + log(sum) - target) over its rows in loss[b].
__global__ void __launch_bounds__(256)
row_stats_kernel(const RowStats st, int pieces, int M, int N, float* __restrict__ omax, float* __restrict__ osum,
                 const float* __restrict__ weight, float* __restrict__ loss) {
  pdl_begin();
  __shared__ float2 sh[8][32];
  const int lane = threadIdx.x & 31, seg = threadIdx.x >> 5, row = blockIdx.x * 32 + lane;
  float m = -INFINITY, s = 0.f;
  if (row < M) {
#pragma unroll 4
    for (int p = seg; p < pieces; p += 8) {
      const float2 v = st.part[static_cast<size_t>(p) * M + row];
      const float nm = fmaxf(m, v.x), base = nm == -INFINITY ? 0.f : nm;
      s = s * __expf(m - base) + v.y * __expf(v.x - base);
      m = nm;
    }
  }
  sh[seg][lane] = make_float2(m, s);
  __syncthreads();
  if (seg) return;
  float gm = -INFINITY, gs = 0.f;
#pragma unroll
  for (int i = 0; i < 8; ++i) gm = fmaxf(gm, sh[i][lane].x);
#pragma unroll
  for (int i = 0; i < 8; ++i) gs += sh[i][lane].y == 0.f ? 0.f : sh[i][lane].y * __expf(sh[i][lane].x - gm);
  float l = 0.f;
  if (row < M) {
    const long t = st.targets[row] - st.first_col;
    const bool here = t >= 0 && t < N;
    const float tv = here ? st.target[row] : 0.f;
    if (!here) st.target[row] = 0.f;
    omax[row] = gm;
    osum[row] = gs;
    if (weight) l = (gm + logf(gs) - tv) * weight[row];
  }
  if (!weight) return;
#pragma unroll
  for (int i = 16; i > 0; i >>= 1) l += __shfl_xor_sync(0xffffffffu, l, i);
  if (lane == 0) loss[blockIdx.x] = l;
}

// out = the sum of n values, by one block in a fixed order.
__global__ void __launch_bounds__(256)
sum_kernel(const float* __restrict__ x, int n, float* __restrict__ out) {
  pdl_begin();
  __shared__ float sh[8];
  float s = 0.f;
  for (int i = threadIdx.x; i < n; i += 256) s += x[i];
#pragma unroll
  for (int i = 16; i > 0; i >>= 1) s += __shfl_xor_sync(0xffffffffu, s, i);
  if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x == 0) *out = ((sh[0] + sh[1]) + (sh[2] + sh[3])) + ((sh[4] + sh[5]) + (sh[6] + sh[7]));
}

// C += the sums that K parts 1 .. ks - 1 of the split tiles left in the workspace, part by part: four columns a thread.
__global__ void __launch_bounds__(256)
gemm_add_parts_kernel(float* __restrict__ C, int ldc, int M, int N, const float* __restrict__ work, const PairWork w, int bn) {
  pdl_begin();
  const int vecs = bn >> 2, per_tile = GP_BM * vecs, total = w.split_tiles * per_tile;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < total; i += gridDim.x * blockDim.x) {
    const int tile = i / per_tile, rest = i - tile * per_tile, r = rest / vecs, c = (rest - r * vecs) * 4;
    int tm, tn;
    w.coords(w.whole + tile, tm, tn);
    const int row = tm * GP_BM + r, col = tn * bn + c;
    if (row >= M || col >= N) continue;
    float* dst = C + static_cast<size_t>(row) * ldc + col;
    const float* src = work + (static_cast<size_t>(tile) * GP_BM + r) * bn + c;
    const size_t part = static_cast<size_t>(w.split_tiles) * GP_BM * bn;
    if (col + 4 <= N) {
      float4 v = *reinterpret_cast<const float4*>(dst);
      for (int p = 1; p < w.ks; ++p, src += part) {
        const float4 a = *reinterpret_cast<const float4*>(src);
        v.x += a.x; v.y += a.y; v.z += a.z; v.w += a.w;
      }
      *reinterpret_cast<float4*>(dst) = v;
    } else {
      for (int j = 0; col + j < N; ++j) {
        float v = dst[j];
        for (int p = 1; p < w.ks; ++p) v += src[(p - 1) * part + j];
        dst[j] = v;
      }
    }
  }
}

// C (bf16) = the sum of the K parts of the split tiles, in order: eight columns a thread.
__global__ void __launch_bounds__(256)
gemm_sum_parts_kernel(__nv_bfloat16* __restrict__ C, int ldc, int M, int N, const float* __restrict__ work, const PairWork w, int bn) {
  pdl_begin();
  const int vecs = bn >> 3, per_tile = GP_BM * vecs, total = w.split_tiles * per_tile;
  const size_t part = static_cast<size_t>(w.split_tiles) * GP_BM * bn;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < total; i += gridDim.x * blockDim.x) {
    const int tile = i / per_tile, rest = i - tile * per_tile, r = rest / vecs, c = (rest - r * vecs) * 8;
    int tm, tn;
    w.coords(w.whole + tile, tm, tn);
    const int row = tm * GP_BM + r, col = tn * bn + c;
    if (row >= M || col >= N) continue;
    const float4* src = reinterpret_cast<const float4*>(work + (static_cast<size_t>(tile) * GP_BM + r) * bn + c);
    float4 a = src[0], b = src[1];
#pragma unroll 4
    for (int p = 1; p < w.ks; ++p) {
      src += part / 4;
      const float4 x = src[0], y = src[1];
      a.x += x.x; a.y += x.y; a.z += x.z; a.w += x.w;
      b.x += y.x; b.y += y.y; b.z += y.z; b.w += y.w;
    }
    const uint4 o = make_uint4(pack_bf16x2(a.x, a.y), pack_bf16x2(a.z, a.w), pack_bf16x2(b.x, b.y), pack_bf16x2(b.z, b.w));
    __nv_bfloat16* dst = C + static_cast<size_t>(row) * ldc + col;
    if (col + 8 <= N) {
      *reinterpret_cast<uint4*>(dst) = o;
    } else {
      const uint32_t v[4] = {o.x, o.y, o.z, o.w};
#pragma unroll
      for (int j = 0; j < 8; ++j)
        if (col + j < N) dst[j] = __ushort_as_bfloat16(static_cast<unsigned short>(v[j >> 1] >> (j & 1 ? 16 : 0)));
    }
  }
}

template <bool A_MN, bool B_MN, bool OUT_F32, bool ACCUM, int EPI = EPI_NONE>
static int launch_pair(const void* A, const void* B, void* C, int M, int N, int K, int lda, int ldb, int ldc,
                       const PairPlan& pl, int pairs, float* work, int* status, cudaStream_t stream,
                       const typename EpiArgs<EPI>::type& epi = {}) {
  CUtensorMap tmA, tmB, tmC, tmW;
  int rc;
  if (!A_MN) rc = make_tmap_2d_bf16(&tmA, A, K, M, lda, GP_BK, 128);
  else       rc = make_tmap_2d_bf16(&tmA, A, M, K, lda, 64, GP_BK);
  if (rc) return rc;
  if (!B_MN) rc = make_tmap_2d_bf16(&tmB, B, K, EPI == EPI_SWIGLU ? 2 * N : N, ldb, GP_BK, pl.bn / 2);
  else       rc = make_tmap_2d_bf16(&tmB, B, N, K, ldb, 64, GP_BK);
  if (rc) return rc;
  {
    const uint64_t dims[2] = {(uint64_t)(ACCUM ? N : N & ~(OUT_F32 ? 3 : 7)), (uint64_t)M};
    const uint64_t str[1] = {(uint64_t)ldc * (OUT_F32 ? 4 : 2)};
    const uint32_t box[2] = {OUT_F32 ? 32u : 64u, 32u};
    rc = make_tmap(&tmC, C, OUT_F32 ? 4 : 2, 2, dims, str, box, 3);
    if (rc) return rc;
  }
  const bool split = (ACCUM || EPI == EPI_PARTS) && pl.ks > 1 && pl.split_tiles > 0, ordered = split && pl.ordered;
  tmW = tmC;
  if (ordered) {
    const uint64_t dims[2] = {(uint64_t)pl.bn, (uint64_t)pl.split_tiles * (EPI == EPI_PARTS ? pl.ks : pl.ks - 1) * GP_BM};
    const uint64_t str[1] = {(uint64_t)pl.bn * 4};
    const uint32_t box[2] = {32u, 32u};
    rc = make_tmap(&tmW, work, 4, 2, dims, str, box, 3);
    if (rc) return rc;
  }
  auto kern = gemm_pair_kernel<A_MN, B_MN, OUT_F32, ACCUM, EPI>;
  static bool configured = false;
  if (!configured) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, GP_SMEM);
    if (e != cudaSuccess) return 1000 + static_cast<int>(e);
    configured = true;
  }
  PairWork w;
  w.tiles_m = (M + GP_BM - 1) / GP_BM;
  w.tiles_n = EPI == EPI_SWIGLU ? (N + 127) / 128 : (N + pl.bn - 1) / pl.bn;
  w.nk = (K + GP_BK - 1) / GP_BK;
  w.ks = split ? pl.ks : 1;
  w.ordered = ordered;
  const int tiles = w.tiles_m * w.tiles_n;
  w.split_tiles = split ? pl.split_tiles : 0;
  w.whole = tiles - w.split_tiles;
  // m-tiles per group: about 24 MB of A rows, at most 16 tiles
  const long panel = (long)GP_BM * K * 2;
  long gm = (24L << 20) / panel;
  gm = gm < 8 ? 8 : gm > 16 ? 16 : gm;
  w.group_m = gm < w.tiles_m ? (int)gm : w.tiles_m;
  const int units = w.whole + w.split_tiles * w.ks;
  const int grid = 2 * (units < pairs ? units : pairs);
  KB_LAUNCH_PDL(kern, grid, GP_THREADS, GP_SMEM, stream, tmA, tmB, tmC, tmW, w, M, N, pl.bn, C, ldc, status, epi);
  if constexpr (EPI == EPI_PARTS) {
    const int blocks = w.split_tiles * (GP_BM * pl.bn / 8 / 256);
    KB_LAUNCH_PDL(gemm_sum_parts_kernel, blocks, 256, 0, stream, static_cast<__nv_bfloat16*>(C), ldc, M, N, (const float*)work, w,
                  pl.bn);
  } else if (ordered) {
    const int blocks = w.split_tiles * (GP_BM * pl.bn / 4 / 256);
    KB_LAUNCH_PDL(gemm_add_parts_kernel, blocks, 256, 0, stream, static_cast<float*>(C), ldc, M, N, (const float*)work, w, pl.bn);
  }
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? 0 : 2000 + static_cast<int>(e);
}

int gemm_pair_dispatch(const void* A, const void* B, void* C, int M, int N, int K, int a_mn, int lda, int b_mn, int ldb,
                       int ldc, int out_f32, int accumulate, const PairPlan& pl, int pairs, float* work, int* status,
                       cudaStream_t stream) {
#define GP_GO(AM, BM_)                                                                                         \
  do {                                                                                                         \
    if (out_f32 && accumulate) return launch_pair<AM, BM_, true, true>(A, B, C, M, N, K, lda, ldb, ldc, pl, pairs, work, status, stream);\
    if (out_f32) return launch_pair<AM, BM_, true, false>(A, B, C, M, N, K, lda, ldb, ldc, pl, pairs, work, status, stream);             \
    if (pl.ks > 1 && pl.split_tiles > 0)                                                                                                 \
      return launch_pair<AM, BM_, false, false, EPI_PARTS>(A, B, C, M, N, K, lda, ldb, ldc, pl, pairs, work, status, stream);            \
    return launch_pair<AM, BM_, false, false>(A, B, C, M, N, K, lda, ldb, ldc, pl, pairs, work, status, stream);                         \
  } while (0)
  if (!a_mn && !b_mn) GP_GO(false, false);
  if (!a_mn && b_mn) GP_GO(false, true);
  if (a_mn && !b_mn) GP_GO(true, false);
  GP_GO(true, true);
#undef GP_GO
}

int gemm_pair_row_stats(const void* A, const void* B, void* C, int M, int N, int K, int lda, int ldb, const PairPlan& pl,
                        int pairs, const long* targets, long first_col, float* part, float* omax, float* osum, float* otgt,
                        const float* weight, float* loss, int* status, cudaStream_t stream) {
  const RowStats st{reinterpret_cast<float2*>(part), targets, otgt, first_col, C != nullptr};
  // without a product to store its tensor map is never used; it still needs an address
  const int rc = launch_pair<false, false, false, false, EPI_ROW_STATS>(A, B, C ? C : part, M, N, K, lda, ldb, N, pl, pairs, nullptr,
                                                                        status, stream, st);
  if (rc) return rc;
  const int blocks = (M + 31) / 32, pieces = 2 * ((N + pl.bn - 1) / pl.bn);
  float* block_loss = part + 2L * pieces * M;
  KB_LAUNCH_PDL(row_stats_kernel, blocks, 256, 0, stream, st, pieces, M, N, omax, osum, weight, block_loss);
  if (weight) KB_LAUNCH_PDL(sum_kernel, 1, 256, 0, stream, (const float*)block_loss, blocks, loss);
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? 0 : 2000 + static_cast<int>(e);
}

static int swiglu_maps(SwigluOut* e, const void* x, int M, int features) {
  const uint64_t dims[2] = {(uint64_t)features, (uint64_t)M};
  const uint64_t str[1] = {(uint64_t)features * 4};
  const uint32_t box[2] = {64u, 32u};
  const int rc = make_tmap(&e->gate, x, 2, 2, dims, str, box, 3);
  return rc ? rc : make_tmap(&e->up, reinterpret_cast<const __nv_bfloat16*>(x) + features, 2, 2, dims, str, box, 3);
}

int gemm_pair_swiglu(const void* A, const void* B, void* X, void* H, int M, int features, int K, int lda, int ldb, int pairs,
                     int* status, cudaStream_t stream) {
  SwigluOut e;
  e.features = features;
  e.store = X != nullptr;
  // without a product to store its tensor maps are never used; they still need an address
  const int rc = swiglu_maps(&e, X ? X : H, M, features);
  if (rc) return rc;
  return launch_pair<false, false, false, false, EPI_SWIGLU>(A, B, H, M, features, K, lda, ldb, features, PairPlan{256, 1, 0, 0.0, false},
                                                             pairs, nullptr, status, stream, e);
}

int gemm_pair_swiglu_bwd(const void* A, const void* B, const void* X, void* dX, int M, int features, int K, int lda, int ldb,
                         const PairPlan& pl, int pairs, int* status, cudaStream_t stream) {
  const SwigluGrad e{reinterpret_cast<const __nv_bfloat16*>(X), reinterpret_cast<__nv_bfloat16*>(dX)};
  return launch_pair<false, true, false, false, EPI_SWIGLU_BWD>(A, B, dX, M, features, K, lda, ldb, 2 * features, pl, pairs, nullptr,
                                                                status, stream, e);
}

}  // namespace kb
