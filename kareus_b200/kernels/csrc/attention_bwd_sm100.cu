// Causal GQA flash-attention backward for sm_100a (head dim 128, bf16, fp32 accumulation).
//
// One CTA owns 128 keys of one (batch, KV group) and walks the query tiles that can see them.  Scores are
// kept transposed (rows = keys), so that P leaves the registers as the TMEM operand of dV:
//   warps 0..15  32 keys x 32 query columns each, as matrix fragments (a thread meets 8 columns on 4 rows): Pᵀ = exp2(Sᵀ·c − lse) as soon as Sᵀ is there,
//                bf16 into the TMEM columns the scores came from; then dSᵀ = Pᵀ∘(dPᵀ − δ) once dPᵀ is there, bf16
//                into swizzled shared memory.  lse and δ of a query tile are staged next to its Q; with a key row
//                per thread every thread would read all of its columns' statistics, which cost the shared-memory
//                pipe more than the operands of two products
//   warps 16..19 dQ from TMEM → 8 KB of shared memory per warp → TMA reduce-add into the fp32 accumulator in
//                global memory, 32 rows x 32 columns at a time, no barrier between the warps
//   warp 20      TMA producer: K and V once, then per query tile Q and its row statistics (two buffers) and dO
//   warp 21      MMA issuer (tcgen05, accumulators in TMEM), per query tile i in this order:
//                  dPᵀ = V·dOᵀ,  dV += Pᵀ·dO,  Sᵀ(i+1) = K·Qᵀ,  dQ = dS·K,  dK += dSᵀ·Q
// The order is what makes it a pipeline: Pᵀ(i+1) is computed under dQ and dK of tile i, dSᵀ under dV and the next
// scores, and dQ of tile i leaves TMEM under dK.  dSᵀ is stored once ([key][query], queries contiguous) and serves
// as K-major operand (dK) and, through an MN-major descriptor, as transposed operand of dQ.  The softmax scale goes into dS
// before its rounding to bf16 (δ comes scaled, the scale of dPᵀ rides on the subtraction): it is not a power of two, so that
// rounding first and scaling dQ and dK where they leave would round other values (0.3 % of the gradients as a norm).
// TMEM: Sᵀ|Pᵀ + dPᵀ|dQ + dV + dK = 512 columns.  dK/dV stay in TMEM across the whole walk.
// A CTA walks all query heads of its KV group one after the other and writes dK and dV itself.  Where that leaves
// SMs idle (merge_heads), every query head gets its own CTA and dK/dV are added up in fp32 accumulators.  Starting
// and ending a CTA costs about as much as three query tiles, and accumulators have to be zeroed and converted.
// Shared memory: K, V, Q x 2, dO, dS, dQ staging = 7 tiles of 32 KB.
// What bounds it: the chain dQ → its columns read → dP → dS → dQ, about 3900 clocks per tile for 2560 of MMA; without the
// dQ reductions a tile took 13 % less, without the exponentials 3 %.  One B200, 4 x 4096 tokens, 24 / 8 heads:
// 1850 → 957 us (0.56 → 1.08 PFLOP/s); 4096 queries against 16 k keys, 6 heads: 690 → 408 us.
//
// Chunked keys and queries (context parallelism, see attention_chunks.h): K/V tiles may come from
// several source buffers (other GPUs' shards through their peer mappings, plain TMA loads), query
// tiles carry per-chunk absolute positions, and the bf16 conversion can scatter dK/dV chunk by chunk
// into the input buffer of a reduce-scatter.
//
// Replaces the FlashAttention-2 backward the reference calls through its wheel
// (kareus/flash_attn/flash_attn_interface.py:147-199).
#include "sm100.cuh"
#include "launch.h"
#include "pdl.cuh"
#include "host_utils.h"
#include "native_calls.h"
#include "attention_chunks.h"
#include <string.h>

namespace kb {

constexpr int FB_T = 128;                      // tile edge (queries, keys) and head dim
constexpr int FB_TILE = FB_T * FB_T * 2;       // 32 KB bf16 tile as two 64-wide swizzled chunks
constexpr int FB_CHUNK = 16384;
constexpr int FB_SOFTMAX_WARPS = 16;             // 4 TMEM lane quarters x 4 chunks of 32 query columns
constexpr int FB_DQ_WARP = FB_SOFTMAX_WARPS;     // first of the four dQ warps
constexpr int FB_TMA_WARP = FB_DQ_WARP + 4, FB_MMA_WARP = FB_DQ_WARP + 5;
constexpr int FB_THREADS = (FB_SOFTMAX_WARPS + 8) * 32;   // six warpgroups; the last two warps only fill theirs
// Registers a thread: what the block is launched with, and after the dQ warps have taken some from the last warpgroup
constexpr int FB_REGS = 80, FB_REGS_DQ = 120, FB_REGS_AUX = 40;
static_assert(FB_REGS_DQ + FB_REGS_AUX <= 2 * FB_REGS, "the shares must not exceed the registers at launch");
constexpr int FB_STATS = 2 * FB_T;               // floats of row statistics per query tile: −lse·log2(e), then −δ·scale

// Destinations, strides in elements.
struct RowMap {
  int chunk_rows;                    // 0: rows map to themselves
  int base[MAX_KV_CHUNKS];
  __device__ __forceinline__ long at(long row) const {
    if (chunk_rows == 0) return row;
    const int c = static_cast<int>(row / chunk_rows);
    return base[c] + (row - static_cast<long>(c) * chunk_rows);
  }
};
struct BwdOut {
  void* dq; long dqs_s, dqs_b, dqs_g, dqs_r;
  void* dk; long dks_s, dks_b, dks_g;
  void* dv; long dvs_s, dvs_b, dvs_g;
  RowMap dk_rows, dv_rows;
};

struct BwdParams {
  const float* stats;    // [b, hq, query tiles, 2, 128], see attn_stats_kernel
  float* dk_acc;         // [skv, b, g, d]  (one query head per CTA)
  float* dv_acc;         // [skv, b, g, d]
  int heads;             // query heads of a CTA: rep (the CTA writes dK and dV) or 1
  BwdOut out;
  int sq, skv, b, hq, rep, q_offset, causal;
  float scale, scale_log2;
  int* status;
  ChunkGeom geom;
};

// Can any query of tile `qt` see key tile starting at k0?  (Suffix rule per query chunk.)
__device__ __forceinline__ bool q_tile_sees(const BwdParams& p, int qt, int k0) {
  if (!p.causal) return true;
  const int q0 = qt * FB_T;
  return p.geom.q_offset_of(q0, p.q_offset) + q0 + FB_T - 1 >= k0;
}

// The query tiles of heads head0, head0 + 1, ... that see a key tile, in order.
struct QTiles {
  int n_q, first, qt, head;
  // first query tile worth looking at: exact for one query chunk, where visible tiles are a suffix
  static __device__ __forceinline__ int first_tile(const BwdParams& p, int n_q, int k0) {
    return p.causal && p.geom.q_chunk_rows == 0 ? min(n_q, max(0, k0 - p.q_offset) / FB_T) : 0;
  }
  static __device__ __forceinline__ int count(const BwdParams& p, int n_q, int k0) {
    const int f = first_tile(p, n_q, k0);
    if (!p.causal || p.geom.q_chunk_rows == 0) return n_q - f;
    int n = 0;
    for (int qt = f; qt < n_q; ++qt) n += q_tile_sees(p, qt, k0) ? 1 : 0;
    return n;
  }
  __device__ __forceinline__ QTiles(const BwdParams& p, int n, int k0, int head0)
      : n_q(n), first(first_tile(p, n, k0)), qt(first - 1), head(head0) {}
  __device__ __forceinline__ bool next(const BwdParams& p, int k0, int head1) {
    for (;;) {
      if (++qt >= n_q) {
        qt = first;
        if (++head >= head1 || first >= n_q) return false;
      }
      if (p.geom.q_chunk_rows == 0 || q_tile_sees(p, qt, k0)) return true;
    }
  }
};

struct FbSmem {
  // Q_OFF: two consecutive tiles (buffer = iteration & 1)
  static constexpr int K_OFF = 0, V_OFF = FB_TILE, Q_OFF = 2 * FB_TILE, DO_OFF = 4 * FB_TILE, DS_OFF = 5 * FB_TILE,
                       STG_OFF = 6 * FB_TILE, STAT_OFF = 7 * FB_TILE, BAR_OFF = STAT_OFF + 2 * FB_STATS * 4;
  // what is left of 227 KB aligns the tiles to 1024 bytes; the kernel checks that it suffices
  static constexpr int USED = BAR_OFF + 256, TOTAL = 227 * 1024;
  static_assert(USED <= TOTAL, "shared memory per CTA");
};

__device__ __forceinline__ float bwd_exp2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ void red_add_v4(float* p, float a, float b, float c, float d) {
  asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(p), "f"(a), "f"(b), "f"(c), "f"(d) : "memory");
}

__global__ void __launch_bounds__(FB_THREADS, 1)
flash_attn_bwd_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ KvMaps kv,
                      const __grid_constant__ CUtensorMap tmDO, const __grid_constant__ CUtensorMap tmDQ,
                      const BwdParams p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  if (smem - smem_raw + FbSmem::USED > FbSmem::TOTAL) {   // the same for all threads
    pdl_wait();
    if (threadIdx.x == 0) atomicCAS(p.status, 0, ST_BAD_ARG);
    return;
  }
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + FbSmem::BAR_OFF);
  uint64_t* kv_full = bars + 0;
  uint64_t* q_full = bars + 1;      // [2] Q and statistics of iteration i are in buffer i & 1
  uint64_t* q_empty = bars + 3;     // [2] the MMAs that read that buffer have retired
  uint64_t* do_full = bars + 5;
  uint64_t* do_empty = bars + 6;    // dPᵀ and dV of this iteration have retired
  uint64_t* s_full = bars + 7;      // Sᵀ is in TMEM
  uint64_t* p_full = bars + 8;      // Pᵀ is in TMEM, Sᵀ has been read (one arrival per warp)
  uint64_t* dp_full = bars + 9;     // dPᵀ is in TMEM
  uint64_t* ds_full = bars + 10;    // dSᵀ is in shared memory, dPᵀ has been read (one arrival per warp)
  uint64_t* ds_empty = bars + 11;   // dQ and dK of this iteration have retired
  uint64_t* dq_full = bars + 12;    // dQ is in TMEM
  uint64_t* dq_empty = bars + 13;   // dQ has been read out of TMEM (one arrival per dQ warp)
  uint64_t* all_done = bars + 14;   // every MMA of the walk has retired
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 15);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // key tile 0 is seen by the most queries: its CTAs go first, over all heads and batches, so that the short ones fill
  // the end.  The CTAs of neighbouring key tiles of a head walk the same queries at the same time, which keeps L2 useful.
  const int units = p.hq / p.heads;
  const int kt = static_cast<int>(blockIdx.x) / (units * p.b), bu = static_cast<int>(blockIdx.x) % (units * p.b);
  const int batch = bu / units;
  const int head0 = (bu - batch * units) * p.heads, head1 = head0 + p.heads;
  const int g = head0 / p.rep;
  const int k0 = kt * FB_T;
  const int n_q = (p.sq + FB_T - 1) / FB_T;
  const int n_it = QTiles::count(p, n_q, k0) * p.heads;   // query tiles that see this key tile, over all heads

  if (threadIdx.x == 0) {
    for (int i = 0; i < 15; ++i)
      mbar_init(&bars[i], &bars[i] == p_full || &bars[i] == ds_full ? FB_SOFTMAX_WARPS : &bars[i] == dq_empty ? 4 : 1);
    *abort_flag = 0;
    mbar_fence_init();
  }
  if (warp == FB_MMA_WARP) tmem_alloc(tmem_slot, 512);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  pdl_begin();
  // Pᵀ of query chunk c goes into the first 16 of the 32 columns of its scores.  dQ of a tile goes where its dPᵀ
  // was: that has been read by then.
  const uint32_t t_s = tmem_base, t_dp = tmem_base + 128, t_dv = tmem_base + 256, t_dk = tmem_base + 384;
  const uint32_t t_dq = t_dp;

  if (warp >= FB_TMA_WARP) {
    regs_dec<FB_REGS_AUX>();
    if (warp == FB_TMA_WARP) {
      if (n_it > 0 && elect_one()) {
        int src, srow;
        p.geom.locate(k0, src, srow);
        prefetch_tmap(&tmQ); prefetch_tmap(&kv.k[src]); prefetch_tmap(&kv.v[src]); prefetch_tmap(&tmDO);
        const float* stats = p.stats + static_cast<size_t>(batch) * p.hq * n_q * FB_STATS;
        mbar_expect_tx(kv_full, 2 * FB_TILE);
        tma_load_4d(smem + FbSmem::K_OFF, &kv.k[src], kv_full, 0, g, batch, srow);
        tma_load_4d(smem + FbSmem::K_OFF + FB_CHUNK, &kv.k[src], kv_full, 64, g, batch, srow);
        tma_load_4d(smem + FbSmem::V_OFF, &kv.v[src], kv_full, 0, g, batch, srow);
        tma_load_4d(smem + FbSmem::V_OFF + FB_CHUNK, &kv.v[src], kv_full, 64, g, batch, srow);
        // per visible tile: Q(it) into buffer it & 1 (released by dK of tile it-2), then dO(it) (released by dV of
        // tile it-1): Q(it+1) goes out right behind dO(it), one tile ahead of the MMAs
        int it = 0;
        QTiles tiles(p, n_q, k0, head0);
        while (tiles.next(p, k0, head1)) {
          const int qt = tiles.qt, head = tiles.head, r = head - g * p.rep;
          const int qb = it & 1;
          const int q0 = qt * FB_T;
          if (!mbar_wait(&q_empty[qb], ((it >> 1) & 1u) ^ 1u, abort_flag, p.status, ST_TIMEOUT_EMPTY)) break;
          uint8_t* qdst = smem + FbSmem::Q_OFF + qb * FB_TILE;
          mbar_expect_tx(&q_full[qb], FB_TILE + FB_STATS * 4);
          tma_load_5d(qdst, &tmQ, &q_full[qb], 0, r, g, batch, q0);
          tma_load_5d(qdst + FB_CHUNK, &tmQ, &q_full[qb], 64, r, g, batch, q0);
          bulk_load(smem + FbSmem::STAT_OFF + qb * FB_STATS * 4, stats + (static_cast<size_t>(head) * n_q + qt) * FB_STATS,
                    FB_STATS * 4, &q_full[qb]);
          if (!mbar_wait(do_empty, (it & 1u) ^ 1u, abort_flag, p.status, ST_TIMEOUT_EMPTY)) break;
          mbar_expect_tx(do_full, FB_TILE);
          tma_load_4d(smem + FbSmem::DO_OFF, &tmDO, do_full, 0, head, batch, q0);
          tma_load_4d(smem + FbSmem::DO_OFF + FB_CHUNK, &tmDO, do_full, 64, head, batch, q0);
          ++it;
        }
        if (*abort_flag) {
          const uint64_t t0 = globaltimer_ns();
          while (globaltimer_ns() - t0 < 200000ull) {}
        }
      }
      __syncwarp();
    } else if (warp == FB_MMA_WARP) {
      if (n_it > 0 && elect_one()) {           // one thread runs the whole role, see elect_one()
        constexpr uint32_t id_kk = make_idesc_bf16(FB_T, FB_T, false, false);   // A K-major, B K-major
        constexpr uint32_t id_mm = make_idesc_bf16(FB_T, FB_T, true, true);     // A MN-major, B MN-major
        constexpr uint32_t id_km = make_idesc_bf16(FB_T, FB_T, false, true);    // A K-major (or TMEM), B MN-major
          // Descriptors of an operand for 16-deep step k: K-major rows, or MN-major with 64-wide chunks.  Only the low
        // word depends on the address; `lo` is made opaque once per tile, or the compiler would keep all 40 of them
        // in registers.
        uint32_t lo = (smem_u32(smem) & 0x3FFFFu) >> 4;
        constexpr uint64_t DESC_HI = make_smem_desc(0, 0, 1024);
        auto desc = [&](uint32_t lbo, int off) { return DESC_HI | (lo + ((lbo >> 4) << 16) + static_cast<uint32_t>(off >> 4)); };
        auto kmaj = [&](int off, int k) { return desc(16, off + (k >> 2) * FB_CHUNK + (k & 3) * 32); };
        auto mnmaj = [&](int off, int k) { return desc(FB_CHUNK, off + k * 2048); };
        bool ok = true;
        auto wait = [&](uint64_t* bar, uint32_t parity, int code) {
          ok = mbar_wait(bar, parity, abort_flag, p.status, code);
          if (ok) tc_fence_after();
          return ok;
        };
        auto issue_s = [&](int i) {
          const int q = FbSmem::Q_OFF + (i & 1) * FB_TILE;
#pragma unroll
          for (int k = 0; k < 8; ++k) umma_ss(t_s, kmaj(FbSmem::K_OFF, k), kmaj(q, k), id_kk, k > 0);
          umma_commit(s_full);
        };
        if (wait(kv_full, 0, ST_TIMEOUT_FULL) && wait(&q_full[0], 0, ST_TIMEOUT_FULL)) issue_s(0);
        for (int it = 0; it < n_it && ok; ++it) {
          const uint32_t ph = it & 1u;
          const int q = FbSmem::Q_OFF + (it & 1) * FB_TILE;
          asm volatile("" : "+r"(lo));
          // dPᵀ(it) overwrites the columns that held dQ(it-1)
          if (!wait(do_full, ph, ST_TIMEOUT_FULL) || !wait(dq_empty, ph ^ 1u, ST_TIMEOUT_TMEM_EMPTY)) break;
#pragma unroll
          for (int k = 0; k < 8; ++k) umma_ss(t_dp, kmaj(FbSmem::V_OFF, k), kmaj(FbSmem::DO_OFF, k), id_kk, k > 0);
          umma_commit(dp_full);
          if (!wait(p_full, ph, ST_TIMEOUT_TMEM_FULL)) break;
#pragma unroll
          for (int k = 0; k < 8; ++k)          // 16 queries: 8 columns of Pᵀ, 16 rows of dO
            umma_ts(t_dv, t_s + (k >> 1) * 32 + (k & 1) * 8, mnmaj(FbSmem::DO_OFF, k), id_km, (it > 0 || k > 0));
          umma_commit(do_empty);
          if (it + 1 < n_it) {
            // overwrites Pᵀ(it): the product before it reads it in order
            if (!wait(&q_full[(it + 1) & 1], ((it + 1) >> 1) & 1u, ST_TIMEOUT_FULL)) break;
            issue_s(it + 1);
          }
          if (!wait(ds_full, ph, ST_TIMEOUT_TMEM_FULL)) break;
#pragma unroll
          for (int k = 0; k < 8; ++k) umma_ss(t_dq, mnmaj(FbSmem::DS_OFF, k), mnmaj(FbSmem::K_OFF, k), id_mm, k > 0);
          umma_commit(dq_full);
#pragma unroll
          for (int k = 0; k < 8; ++k) umma_ss(t_dk, kmaj(FbSmem::DS_OFF, k), mnmaj(q, k), id_km, (it > 0 || k > 0));
          umma_commit(&q_empty[it & 1]);
          umma_commit(ds_empty);
        }
        if (ok) umma_commit(all_done);
      }
      __syncwarp();
    }
  } else if (warp < FB_SOFTMAX_WARPS) {
    const uint32_t lane_addr = static_cast<uint32_t>((warp & 3) * 32) << 16;
    const int c = warp >> 2;                       // chunk of 32 query columns
    // this thread's fragment: key rows frag_row + 8 x (0..3), query columns frag_col + 8 n + (0, 1) of the chunk
    const int frag_row = (warp & 3) * 32 + (lane >> 2), frag_col = 2 * (lane & 3);
    // the row of dSᵀ whose address this thread gives to the matrix stores (two 64-wide swizzled chunks per row)
    const uint32_t ds_row = smem_u32(smem) + FbSmem::DS_OFF + (c >> 1) * FB_CHUNK + ((warp & 3) * 32 + lane) * 128;
    const float2 sc2 = make_float2(p.scale_log2, p.scale_log2), scale2 = make_float2(p.scale, p.scale);
    bool ok = true;
    int it = -1;
    QTiles tiles(p, n_q, k0, head0);
    while (ok && tiles.next(p, k0, head1)) {
      ++it;
      const uint32_t ph = it & 1u;
      const int q0 = tiles.qt * FB_T;
      const int q_off = p.geom.q_offset_of(q0, p.q_offset);
      const float* stat = reinterpret_cast<const float*>(smem + FbSmem::STAT_OFF + (it & 1) * FB_STATS * 4) + c * 32 + frag_col;
      const bool tile_mask = (p.causal && k0 + FB_T - 1 > q_off + q0) || (k0 + FB_T > p.skv);
      // the scores were issued behind the arrival of Q and its statistics; this wait makes the latter visible here
      ok = __all_sync(0xffffffffu,
                      mbar_wait(&q_full[it & 1], (it >> 1) & 1u, abort_flag, p.status, ST_TIMEOUT_FULL) &&
                          mbar_wait(s_full, ph, abort_flag, p.status, ST_TIMEOUT_TMEM_FULL));
      if (!ok) break;
      tc_fence_after();
      uint32_t pk[2][8];                           // Pᵀ of the fragment as packed bf16, kept for dSᵀ
      {
        uint32_t sv[2][16];
        tmem_ld_16x256b_x4(t_s + lane_addr + c * 32, sv[0]);
        tmem_ld_16x256b_x4(t_s + lane_addr + (16u << 16) + c * 32, sv[1]);
        tmem_ld_wait();
#pragma unroll
        for (int n = 0; n < 4; ++n) {
          const float2 nl = *reinterpret_cast<const float2*>(stat + 8 * n);   // rows past sq carry −inf: Pᵀ = 0
#pragma unroll
          for (int h = 0; h < 4; ++h) {
            const float2 x = __ffma2_rn(make_float2(__uint_as_float(sv[h >> 1][4 * n + 2 * (h & 1)]),
                                                    __uint_as_float(sv[h >> 1][4 * n + 2 * (h & 1) + 1])), sc2, nl);
            pk[h >> 1][2 * n + (h & 1)] = pack_bf16x2(bwd_exp2(x.x), bwd_exp2(x.y));
          }
        }
      }
      if (tile_mask) {
        // fragment column x sees its key from `first` on
#pragma unroll
        for (int h = 0; h < 4; ++h) {
          const int key = k0 + frag_row + 8 * h;
          const int first = key >= p.skv ? 32 : p.causal ? key - (q_off + q0 + c * 32 + frag_col) : 0;
#pragma unroll
          for (int n = 0; n < 4; ++n) {
            if (8 * n < first) pk[h >> 1][2 * n + (h & 1)] &= 0xffff0000u;
            if (8 * n + 1 < first) pk[h >> 1][2 * n + (h & 1)] &= 0x0000ffffu;
          }
        }
      }
      tmem_st_16x128b_x4(t_s + lane_addr + c * 32, pk[0]);
      tmem_st_16x128b_x4(t_s + lane_addr + (16u << 16) + c * 32, pk[1]);
      tmem_st_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(p_full);
      // ds_empty: the products of the previous tile have read the dS buffer
      ok = __all_sync(0xffffffffu, mbar_wait(ds_empty, ph ^ 1u, abort_flag, p.status, ST_TIMEOUT_EMPTY) &&
                                       mbar_wait(dp_full, ph, abort_flag, p.status, ST_TIMEOUT_TMEM_FULL));
      if (!ok) break;
      tc_fence_after();
      uint32_t dv[2][16];
      tmem_ld_16x256b_x4(t_dp + lane_addr + c * 32, dv[0]);
      tmem_ld_16x256b_x4(t_dp + lane_addr + (16u << 16) + c * 32, dv[1]);
      tmem_ld_wait();
#pragma unroll
      for (int n = 0; n < 4; ++n) {
        const float2 nd = *reinterpret_cast<const float2*>(stat + FB_T + 8 * n);
        uint32_t w[4];
#pragma unroll
        for (int h = 0; h < 4; ++h) {
          const float2 e = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&pk[h >> 1][2 * n + (h & 1)]));
          const float2 d = __fmul2_rn(e, __ffma2_rn(make_float2(__uint_as_float(dv[h >> 1][4 * n + 2 * (h & 1)]),
                                                                __uint_as_float(dv[h >> 1][4 * n + 2 * (h & 1) + 1])), scale2, nd));
          w[h] = pack_bf16x2(d.x, d.y);
        }
        stmatrix_x4(ds_row + ((((c & 1) * 4 + n) ^ (lane & 7)) << 4), w);
      }
      tc_fence_before();
      fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) mbar_arrive(ds_full);
    }
    // dV and dK of this key tile (rows = keys); this warp has columns 32c..32c+31 of both
    const int row = (warp & 3) * 32 + lane;
    if (n_it > 0) {
      if (ok) ok = mbar_wait(all_done, 0, abort_flag, p.status, ST_TIMEOUT_TMEM_FULL);
      __syncwarp();
      tc_fence_after();
    }
    if (p.heads < p.rep) {
      // one query head of several: into the fp32 accumulators
      const int key = k0 + row;
      const bool kvalid = ok && n_it > 0 && key < p.skv;
      const size_t base = ((static_cast<size_t>(kvalid ? key : 0) * p.b + batch) * (p.hq / p.rep) + g) * FB_T;
#pragma unroll 1
      for (int which = 0; which < 2 && n_it > 0; ++which) {
        float* dst = (which == 0 ? p.dv_acc : p.dk_acc) + base + c * 32;
        uint32_t v[32];
        tmem_ld_32x32((which == 0 ? t_dv : t_dk) + lane_addr + c * 32, v);
        tmem_ld_wait();
        if (kvalid) {
#pragma unroll
          for (int j = 0; j < 8; ++j)
            red_add_v4(dst + 4 * j, __uint_as_float(v[4 * j]), __uint_as_float(v[4 * j + 1]), __uint_as_float(v[4 * j + 2]),
                       __uint_as_float(v[4 * j + 3]));
        }
      }
    } else {
      // bf16 through shared memory (the query buffers, read to the end by now), then whole rows; keys that no
      // query sees get zeros
      constexpr int PITCH = FB_T * 2 + 16;
      static_assert(FbSmem::Q_OFF + 2 * FB_T * PITCH <= FbSmem::DS_OFF, "staging of dV and dK");
      uint8_t* stg = smem + FbSmem::Q_OFF;
#pragma unroll 1
      for (int which = 0; which < 2; ++which) {
        uint32_t v[32];
        if (n_it > 0) {
          tmem_ld_32x32((which == 0 ? t_dv : t_dk) + lane_addr + c * 32, v);
          tmem_ld_wait();
        } else {
#pragma unroll
          for (int j = 0; j < 32; ++j) v[j] = 0u;
        }
        const uint32_t dst = smem_u32(stg) + which * FB_T * PITCH + row * PITCH + c * 64;
#pragma unroll
        for (int j = 0; j < 4; ++j)
          st_shared_v4(dst + j * 16, pack_bf16x2(__uint_as_float(v[8 * j]), __uint_as_float(v[8 * j + 1])),
                       pack_bf16x2(__uint_as_float(v[8 * j + 2]), __uint_as_float(v[8 * j + 3])),
                       pack_bf16x2(__uint_as_float(v[8 * j + 4]), __uint_as_float(v[8 * j + 5])),
                       pack_bf16x2(__uint_as_float(v[8 * j + 6]), __uint_as_float(v[8 * j + 7])));
      }
      asm volatile("bar.sync 1, %0;" ::"n"(FB_SOFTMAX_WARPS * 32) : "memory");
      if (ok) {
        const BwdOut& o = p.out;
#pragma unroll 1
        for (int which = 0; which < 2; ++which) {
          const long st_s = which == 0 ? o.dvs_s : o.dks_s;
          __nv_bfloat16* dst = which == 0 ? reinterpret_cast<__nv_bfloat16*>(o.dv) + batch * o.dvs_b + g * o.dvs_g
                                          : reinterpret_cast<__nv_bfloat16*>(o.dk) + batch * o.dks_b + g * o.dks_g;
          // a key tile never crosses a chunk of the row map
          dst += (which == 0 ? o.dv_rows.at(k0) : o.dk_rows.at(k0)) * st_s + lane * 4;
          const uint8_t* src = stg + which * FB_T * PITCH + lane * 8;
#pragma unroll
          for (int x = warp; x < FB_T; x += FB_SOFTMAX_WARPS)
            if (k0 + x < p.skv) *reinterpret_cast<uint2*>(dst + x * st_s) = *reinterpret_cast<const uint2*>(src + x * PITCH);
        }
      }
    }
  } else {
    // dQ tile → fp32 reductions into the global accumulator.  The warp's 32 rows go out 32 columns (4 KB) at a time
    // through two buffers: 128-byte rows with their 16-byte units swizzled by row, as the tensor map expects.
    regs_inc<FB_REGS_DQ>();
    const int quarter = warp & 3;
    const uint32_t t_mine = t_dq + (static_cast<uint32_t>(quarter * 32) << 16);
    uint8_t* stg = smem + FbSmem::STG_OFF + quarter * 8192;
    const uint32_t stg_row = smem_u32(stg) + lane * 128;
    auto put = [&](int buf, const uint32_t (&v)[32]) {
#pragma unroll
      for (int j = 0; j < 8; ++j)
        st_shared_v4(stg_row + buf * 4096 + ((j ^ (lane & 7)) << 4), v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]);
    };
    int it = -1;
    QTiles tiles(p, n_q, k0, head0);
    while (tiles.next(p, k0, head1)) {
      ++it;
      const int qt = tiles.qt, head = tiles.head;
      if (!__all_sync(0xffffffffu, mbar_wait(dq_full, it & 1u, abort_flag, p.status, ST_TIMEOUT_TMEM_FULL))) break;
      tc_fence_after();
      const int row0 = qt * FB_T + quarter * 32;
      auto send = [&](int col) {                      // both buffers: 64 columns from `col` on
        fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0 && row0 < p.sq) {               // the tensor map clips rows past sq
          tma_reduce_add_4d(&tmDQ, stg, col, head, batch, row0);
          tma_reduce_add_4d(&tmDQ, stg + 4096, col + 32, head, batch, row0);
          tma_store_commit();
        }
      };
      auto buffers_free = [&] {                       // the reductions before this one have read both buffers
        if (lane == 0) tma_store_wait_read<0>();
        __syncwarp();
      };
      uint32_t v0[32], v1[32], v2[32];
      tmem_ld_32x32(t_mine, v0);
      tmem_ld_32x32(t_mine + 32, v1);
      tmem_ld_32x32(t_mine + 64, v2);
      tmem_ld_wait();
      buffers_free();
      // dPᵀ of the next tile waits for these columns: read all of them before anything is sent
      put(0, v0);
      tmem_ld_32x32(t_mine + 96, v0);
      tmem_ld_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(dq_empty);
      put(1, v1);
      send(0);
      buffers_free();
      put(0, v2);
      put(1, v0);
      send(64);
    }
    if (lane == 0) tma_store_wait<0>();               // nothing in flight out of shared memory at exit
    __syncwarp();
  }

  tc_fence_before();
  __syncthreads();
  if (warp == FB_MMA_WARP) {
    tc_fence_after();
    tmem_dealloc(tmem_base, 512);
  }
}

// Row statistics for the kernel above, one 1 KB block per query tile of one (batch, head): 128 x −lse·log2(e), then
// 128 x −δ·scale with δ = Σ_d dO·O (both [s,b,h,d] contiguous).  Rows past S get −inf and 0.  Half a warp per row, which also
// zeroes its row of the dQ accumulator; `zero` (n_zero vectors) are the accumulators of dK and dV, if there are any.
// dO is 16-byte aligned (TMA reads it too); O need not be (`wide` false: 8 bytes).
__global__ void __launch_bounds__(256)
attn_stats_kernel(const __nv_bfloat16* __restrict__ dO, const __nv_bfloat16* __restrict__ O,
                  const float* __restrict__ lse, float* __restrict__ stats, float4* __restrict__ dq_acc,
                  float4* __restrict__ zero, long n_zero, unsigned S, unsigned S_pad, unsigned B, unsigned H, float scale,
                  bool wide) {
  pdl_begin();
  const float4 z = make_float4(0.f, 0.f, 0.f, 0.f);
  for (long i = static_cast<long>(blockIdx.x) * blockDim.x + threadIdx.x; i < n_zero;
       i += static_cast<long>(gridDim.x) * blockDim.x)
    zero[i] = z;
  const unsigned rows = static_cast<unsigned>(S_pad) * B * H;
  const int l = threadIdx.x & 15;
  const unsigned step = (gridDim.x * blockDim.x) >> 4;
#pragma unroll 2
  for (unsigned w0 = (blockIdx.x * blockDim.x + (threadIdx.x & ~31)) >> 4; w0 < rows; w0 += step) {
    const unsigned w = w0 + ((threadIdx.x >> 4) & 1);
    const unsigned sb = w / H, h = w - sb * H, ss = sb / B, bb = sb - ss * B;
    float s = 0.f;
    if (ss < S && w < rows) {
      float4* acc = dq_acc + static_cast<size_t>(w) * (FB_T / 4) + l;
      acc[0] = z;
      acc[16] = z;
      const uint4 a = reinterpret_cast<const uint4*>(dO + static_cast<size_t>(w) * FB_T)[l];
      const __nv_bfloat16* o = O + static_cast<size_t>(w) * FB_T + l * 8;
      uint4 b;
      if (wide) {
        b = *reinterpret_cast<const uint4*>(o);
      } else {
        const uint2 b0 = reinterpret_cast<const uint2*>(o)[0], b1 = reinterpret_cast<const uint2*>(o)[1];
        b = make_uint4(b0.x, b0.y, b1.x, b1.y);
      }
      const __nv_bfloat162* a2 = reinterpret_cast<const __nv_bfloat162*>(&a);
      const __nv_bfloat162* b2 = reinterpret_cast<const __nv_bfloat162*>(&b);
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float2 x = __bfloat1622float2(a2[i]), y = __bfloat1622float2(b2[i]);
        s += x.x * y.x + x.y * y.y;
      }
    }
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (l == 0 && w < rows) {
      const long bh = static_cast<long>(bb) * H + h;
      float* t = stats + (bh * (S_pad / FB_T) + ss / FB_T) * FB_STATS + ss % FB_T;
      t[0] = ss < S ? lse[bh * S + ss] * -1.4426950408889634f : -INFINITY;
      t[FB_T] = -s * scale;
    }
  }
}

// fp32 accumulator [rows(s,b), heads, d] → bf16 strided view (strides in elements per s, b, group, head
// of the group); `rows_of` moves chunks of s (dK/dV straight into the layout a reduce-scatter expects).
struct Convert {
  const float* acc;
  __nv_bfloat16* out;
  unsigned rows, G, R;
  long st_s, st_b, st_g, st_r;
  bool wide;                  // the view is aligned to 16 bytes
  RowMap rows_of;
};
// All accumulators of a call in one launch.  Half a warp per head vector, 8 elements a thread: 16-byte stores, or two of
// 8 bytes where the view is not aligned to 16.  Bound by memory: 201 MB in and 101 MB out take 51 us (72 with 4 elements
// a thread and 64-bit divisions).
__global__ void __launch_bounds__(256)
attn_convert_kernel(const __grid_constant__ Convert dq, const __grid_constant__ Convert dk, const __grid_constant__ Convert dv,
                    unsigned B) {
  pdl_begin();
  const int l = threadIdx.x & 15;
  const unsigned step = (gridDim.x * blockDim.x) >> 4, total = dq.rows + dk.rows + dv.rows;
  auto convert = [&](const Convert& c, unsigned w) {
    const float4* src = reinterpret_cast<const float4*>(c.acc + static_cast<size_t>(w) * FB_T) + l * 2;
    const float4 a = __ldcs(src), b = __ldcs(src + 1);
    const unsigned t = w / c.R, rr = w - t * c.R, u = t / c.G, gg = t - u * c.G, ss = u / B, bb = u - ss * B;
    __nv_bfloat16* o = c.out + c.rows_of.at(ss) * c.st_s + bb * c.st_b + gg * c.st_g + rr * c.st_r + l * 8;
    uint4 v;
    v.x = pack_bf16x2(a.x, a.y);
    v.y = pack_bf16x2(a.z, a.w);
    v.z = pack_bf16x2(b.x, b.y);
    v.w = pack_bf16x2(b.z, b.w);
    if (c.wide) {
      *reinterpret_cast<uint4*>(o) = v;
    } else {
      reinterpret_cast<uint2*>(o)[0] = make_uint2(v.x, v.y);
      reinterpret_cast<uint2*>(o)[1] = make_uint2(v.z, v.w);
    }
  };
  for (unsigned w = (blockIdx.x * blockDim.x + threadIdx.x) >> 4; w < total; w += step) {
    if (w < dq.rows) convert(dq, w);
    else if (w < dq.rows + dk.rows) convert(dk, w - dq.rows);
    else convert(dv, w - dq.rows - dk.rows);
  }
}

static int make_qkv_map(CUtensorMap* m, const void* ptr, int d, int inner_heads, int g, int b, int s, long st_r,
                        long st_g, long st_b, long st_s, int rank5) {
  if (rank5) {
    uint64_t dims[5] = {(uint64_t)d, (uint64_t)inner_heads, (uint64_t)g, (uint64_t)b, (uint64_t)s};
    uint64_t str[4] = {(uint64_t)st_r * 2, (uint64_t)st_g * 2, (uint64_t)st_b * 2, (uint64_t)st_s * 2};
    uint32_t box[5] = {64, 1, 1, 1, FB_T};
    for (int i = 0; i < 4; ++i) if (str[i] == 0 || (str[i] & 15)) str[i] = (uint64_t)d * 2;
    return make_tmap(m, ptr, 2, 5, dims, str, box, 3);
  }
  uint64_t dims[4] = {(uint64_t)d, (uint64_t)g, (uint64_t)b, (uint64_t)s};
  uint64_t str[3] = {(uint64_t)st_g * 2, (uint64_t)st_b * 2, (uint64_t)st_s * 2};
  uint32_t box[4] = {64, 1, 1, FB_T};
  for (int i = 0; i < 3; ++i) if (str[i] == 0 || (str[i] & 15)) str[i] = (uint64_t)d * 2;
  return make_tmap(m, ptr, 2, 4, dims, str, box, 3);
}

}  // namespace kb

using namespace kb;

namespace kb {

// Does a CTA walk all query heads of its KV group?  Rounds of CTAs over the SMs, plus half a round for the uneven end,
// times the length of a CTA in query tiles, of which three pay for its start and end.
static bool merge_heads(int sq, int skv, int b, int g, int rep) {
  if (rep == 1) return true;
  const double n_q = (sq + FB_T - 1) / FB_T, ctas = (double)((skv + FB_T - 1) / FB_T) * b * g, sms = device_sm_count();
  return (ctas / sms + 0.5) * (n_q * rep + 3) < (ctas * rep / sms + 0.5) * (n_q + 3);
}
static long stats_floats(int sq, int b, int hq) { return (long)b * hq * ((sq + FB_T - 1) / FB_T) * FB_STATS; }

}  // namespace kb

// Scratch: `work` (16-byte aligned) must hold the fp32 accumulators, zeroed by the call, and the row statistics.
extern "C" long kb_flash_attn_bwd_scratch_floats(int sq, int skv, int b, int g, int rep, int d) {
  return (long)sq * b * g * rep * d + stats_floats(sq, b, g * rep) +
         (merge_heads(sq, skv, b, g, rep) ? 0 : 2L * skv * b * g * d);
}
namespace kb {

static int launch_bwd(const CUtensorMap& tmQ, const KvMaps& kv, const ChunkGeom& geom, const void* o, const void* dO,
                      const float* lse, const BwdOut& out, float* work, int sq, int skv, int b, int g, int rep, int d,
                      float scale, int causal, int q_offset, int last_key, int* status, cudaStream_t stream) {
  const int hq = g * rep;
  const long n_dq = (long)sq * b * hq * d, n_dkv = (long)skv * b * g * d;
  const bool merged = merge_heads(sq, skv, b, g, rep);
  float* dq_acc = work;
  float* stats = dq_acc + n_dq;
  float* dk_acc = merged ? nullptr : stats + stats_floats(sq, b, hq);
  float* dv_acc = merged ? nullptr : dk_acc + n_dkv;
  cudaError_t e;
  // refused before anything is launched: the statistics kernel reads dO 16 bytes at a time
  CUtensorMap tmDO;
  int rc = make_qkv_map(&tmDO, dO, d, 1, hq, b, sq, 0, d, (long)hq * d, (long)b * hq * d, 0);
  if (rc) return rc;
  if (reinterpret_cast<uintptr_t>(o) & 7) return ST_BAD_ARG;
  {
    const int s_pad = (sq + FB_T - 1) / FB_T * FB_T;
    const long rows = (long)s_pad * b * hq;
    long blocks = (rows * 16 + 255) / 256;
    if (blocks > 148 * 16) blocks = 148 * 16;
    KB_LAUNCH_PDL(attn_stats_kernel, (int)blocks, 256, 0, stream, (const __nv_bfloat16*)dO, (const __nv_bfloat16*)o, lse, stats,
              reinterpret_cast<float4*>(dq_acc), reinterpret_cast<float4*>(dk_acc), merged ? 0L : 2 * n_dkv / 4, sq, s_pad, b, hq, scale,
              (reinterpret_cast<uintptr_t>(o) & 15) == 0);
  }
  BwdParams p;
  p.stats = stats; p.dk_acc = dk_acc; p.dv_acc = dv_acc; p.heads = merged ? rep : 1; p.out = out;
  p.sq = sq; p.skv = skv; p.b = b; p.hq = hq; p.rep = rep; p.q_offset = q_offset; p.causal = causal;
  p.scale = scale; p.scale_log2 = scale * 1.4426950408889634f; p.status = status;
  p.geom = geom;
  static bool configured = false;
  if (!configured) {
    e = cudaFuncSetAttribute(flash_attn_bwd_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, FbSmem::TOTAL);
    if (e != cudaSuccess) return 1000 + (int)e;
    cudaFuncAttributes attr;
    e = cudaFuncGetAttributes(&attr, flash_attn_bwd_kernel);
    if (e != cudaSuccess) return 1000 + (int)e;
    if (attr.numRegs < FB_REGS) return ST_BAD_ARG;   // the register split would wait forever
    configured = true;
  }
  CUtensorMap tmDQ;
  {
    // fp32 accumulator [sq, b, hq, d]: boxes of 32 rows x 32 columns (128 bytes, swizzled) of one (b, head)
    uint64_t dims[4] = {(uint64_t)d, (uint64_t)hq, (uint64_t)b, (uint64_t)sq};
    uint64_t str[3] = {(uint64_t)d * 4, (uint64_t)hq * d * 4, (uint64_t)b * hq * d * 4};
    uint32_t box[4] = {32, 1, 1, 32};
    rc = make_tmap(&tmDQ, dq_acc, 4, 4, dims, str, box, 3);
    if (rc) return rc;
  }
  int n_kv = (skv + FB_T - 1) / FB_T;
  if (causal && !merged) {
    const int lim = (last_key + FB_T - 1) / FB_T;      // keys >= last_key are seen by no query
    if (lim < n_kv) n_kv = lim > 0 ? lim : 0;
  }
  if (n_kv > 0) {
    const dim3 grid((unsigned)(hq / p.heads * b) * n_kv);
    KB_LAUNCH_PDL(flash_attn_bwd_kernel, grid, FB_THREADS, FbSmem::TOTAL, stream, tmQ, kv, tmDO, tmDQ, p);
  }
  {
    auto segment = [&](const float* acc, void* dst, long rows, int r, long st_s, long st_b, long st_g, long st_r,
                       const RowMap& map) {
      const bool wide = ((reinterpret_cast<uintptr_t>(dst) | ((st_s | st_b | st_g | st_r) * 2)) & 15) == 0;
      return Convert{acc, (__nv_bfloat16*)dst, (unsigned)rows, (unsigned)g, (unsigned)r, st_s, st_b, st_g, st_r, wide, map};
    };
    const long kv_rows = merged ? 0 : (long)skv * b * g;
    RowMap plain;
    plain.chunk_rows = 0;
    const Convert cq = segment(dq_acc, out.dq, (long)sq * b * hq, rep, out.dqs_s, out.dqs_b, out.dqs_g, out.dqs_r, plain);
    const Convert ck = segment(dk_acc, out.dk, kv_rows, 1, out.dks_s, out.dks_b, out.dks_g, 0, out.dk_rows);
    const Convert cv = segment(dv_acc, out.dv, kv_rows, 1, out.dvs_s, out.dvs_b, out.dvs_g, 0, out.dv_rows);
    const long blocks = (((long)sq * b * hq + 2 * kv_rows) * 16 + 255) / 256;
    KB_LAUNCH_PDL(attn_convert_kernel, (int)blocks, 256, 0, stream, cq, ck, cv, (unsigned)b);
  }
  e = cudaGetLastError();
  return e == cudaSuccess ? 0 : 2000 + (int)e;
}

}  // namespace kb

// q: view [sq,b,g,rep,d]; k,v: views [skv,b,g,d]; o, dO: [sq,b,hq,d] contiguous; lse [b,hq,sq].
// dq/dk/dv: destination views with the same geometry as q/k/v (strides in elements).
extern "C" int kb_flash_attn_bwd(const void* q, long qs_s, long qs_b, long qs_g, long qs_r, const void* k, long ks_s,
                                 long ks_b, long ks_g, const void* v, long vs_s, long vs_b, long vs_g, const void* o,
                                 const void* dO, const float* lse, void* dq, long dqs_s, long dqs_b, long dqs_g,
                                 long dqs_r, void* dk, long dks_s, long dks_b, long dks_g, void* dv, long dvs_s,
                                 long dvs_b, long dvs_g, float* work, int sq, int skv, int b, int g, int rep, int d,
                                 float scale, int causal, int q_offset, int* status, cudaStream_t stream) {
  if (d != FB_T || sq <= 0 || skv <= 0) return ST_BAD_ARG;
  CUtensorMap tmQ;
  KvMaps kv;
  memset(&kv, 0, sizeof(kv));
  int rc = make_qkv_map(&tmQ, q, d, rep, g, b, sq, qs_r, qs_g, qs_b, qs_s, 1);
  if (rc) return rc;
  rc = make_qkv_map(&kv.k[0], k, d, 1, g, b, skv, 0, ks_g, ks_b, ks_s, 0);
  if (rc) return rc;
  rc = make_qkv_map(&kv.v[0], v, d, 1, g, b, skv, 0, vs_g, vs_b, vs_s, 0);
  if (rc) return rc;
  ChunkGeom geom;
  memset(&geom, 0, sizeof(geom));
  BwdOut out;
  memset(&out, 0, sizeof(out));
  out.dq = dq; out.dqs_s = dqs_s; out.dqs_b = dqs_b; out.dqs_g = dqs_g; out.dqs_r = dqs_r;
  out.dk = dk; out.dks_s = dks_s; out.dks_b = dks_b; out.dks_g = dks_g;
  out.dv = dv; out.dvs_s = dvs_s; out.dvs_b = dvs_b; out.dvs_g = dvs_g;
  return launch_bwd(tmQ, kv, geom, o, dO, lse, out, work, sq, skv, b, g, rep, d, scale, causal, q_offset,
                    q_offset + sq, status, stream);
}

// Chunked variant (see kb_flash_attn_fwd_chunked for the key/query chunk description).  dK and dV of the
// whole logical key range go to ONE destination `dkv` ([rows, b, g, d] with the strides given): logical
// chunk c of dK starts at row dk_row_base[c], of dV at dv_row_base[c] — e.g. the rank-ordered input
// buffer of a reduce-scatter, so that nothing is copied between this kernel and the collective.
extern "C" int kb_flash_attn_bwd_chunked(const void* q, long qs_s, long qs_b, long qs_g, long qs_r,
                                         const void* const* k_ptrs, const void* const* v_ptrs, int n_src, int src_rows,
                                         long ks_s, long ks_b, long ks_g, long vs_s, long vs_b, long vs_g,
                                         const int* kv_src, const int* kv_row_base, int n_chunks, int chunk_rows,
                                         int q_chunk_rows, const int* q_pos, const void* o, const void* dO,
                                         const float* lse, void* dq, long dqs_s, long dqs_b, long dqs_g, long dqs_r,
                                         void* dkv, long dkvs_s, long dkvs_b, long dkvs_g, const int* dk_row_base,
                                         const int* dv_row_base, float* work, int sq, int b, int g, int rep, int d,
                                         float scale, int causal, int* status, cudaStream_t stream) {
  ChunkGeom geom;
  int rc = fill_chunk_geom(&geom, n_src, kv_src, kv_row_base, n_chunks, chunk_rows, src_rows, q_chunk_rows, q_pos, sq);
  if (rc || d != FB_T) return ST_BAD_ARG;
  const int skv = n_chunks * chunk_rows;
  CUtensorMap tmQ;
  KvMaps kv;
  memset(&kv, 0, sizeof(kv));
  rc = make_qkv_map(&tmQ, q, d, rep, g, b, sq, qs_r, qs_g, qs_b, qs_s, 1);
  if (rc) return rc;
  for (int i = 0; i < n_src; ++i) {
    rc = make_qkv_map(&kv.k[i], k_ptrs[i], d, 1, g, b, src_rows, 0, ks_g, ks_b, ks_s, 0);
    if (rc) return rc;
    rc = make_qkv_map(&kv.v[i], v_ptrs[i], d, 1, g, b, src_rows, 0, vs_g, vs_b, vs_s, 0);
    if (rc) return rc;
  }
  BwdOut out;
  memset(&out, 0, sizeof(out));
  out.dq = dq; out.dqs_s = dqs_s; out.dqs_b = dqs_b; out.dqs_g = dqs_g; out.dqs_r = dqs_r;
  out.dk = dkv; out.dks_s = dkvs_s; out.dks_b = dkvs_b; out.dks_g = dkvs_g;
  out.dv = dkv; out.dvs_s = dkvs_s; out.dvs_b = dkvs_b; out.dvs_g = dkvs_g;
  out.dk_rows.chunk_rows = out.dv_rows.chunk_rows = chunk_rows;
  int last_key = 0;
  for (int i = 0; i < sq / q_chunk_rows; ++i) last_key = q_pos[i] + q_chunk_rows > last_key ? q_pos[i] + q_chunk_rows : last_key;
  for (int c = 0; c < n_chunks; ++c) {
    out.dk_rows.base[c] = dk_row_base[c];
    out.dv_rows.base[c] = dv_row_base[c];
  }
  return launch_bwd(tmQ, kv, geom, o, dO, lse, out, work, sq, skv, b, g, rep, d, scale, causal, 0, last_key, status,
                    stream);
}
