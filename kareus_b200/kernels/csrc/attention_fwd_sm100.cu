// Causal GQA flash-attention forward for sm_100a, head dim 128, bf16 in / bf16 out, fp32 softmax.
//
// One CTA owns two tiles of 128 query rows of one (batch, head) and walks the key tiles they see; one
// K and V tile in shared memory serves both.  Three warpgroups:
//   warps 0..3  softmax of the first query tile, warps 4..7 of the second: one thread per query row.  All 128
//               scores of the row come from TMEM into registers, the row maximum needs no exchange, and
//               P (bf16) goes back into the TMEM columns the scores came from
//   warp 8      TMA producer: both Q tiles once, then K and V tiles through a ring of five 32 KB stages
//   warp 9      MMA issuer (warps 10 and 11 fill its warpgroup): S = Q·Kᵀ (both operands from shared memory) and O += P·V (P from TMEM)
// The two query tiles alternate: while one is in its softmax the tensor cores work on the other.
// Where single query tiles already fit the chip in one wave, a CTA has one (its share is half as long) and the two softmax
// warpgroups take its even and odd key tiles, each with its own scores, O, maximum and sum; they meet in the epilogue
// (616 queries against 9448 keys, 2 x 8 heads: 121 us with one warpgroup, 78 with both; 4096 tokens, one head: 53 and 34).
// TMEM: S|P and O of both tiles, 4 x 128 columns.  S of the next key tile is issued behind the P·V that
// read P, so its arrival also says that O may be touched; O is rescaled only when the running maximum
// moves by more than 2^8 ("lazy rescale"), which happens on the first tiles only.
//
// Why this split: with P in shared memory and one query tile per CTA a key tile costs the shared memory
// pipe 64 KB of loads in, 32 KB of P in and 128 KB of operands out for 1024 tensor clocks; here it is
// 32 + 0 + 96 KB.  The pace is then set by the exponentials (16 a clock and SM: 1024 clocks per tile and
// head, as many as the two products need) and by how well two warps per scheduler cover each other.  One B200, 4 x 4096
// tokens, 24 / 8 heads: 590 → 373 us (0.70 → 1.10 PFLOP/s); 4096 queries against 16 k keys, 6 heads: 300 → 222 us.
//
// Chunked keys (context parallelism without a gathered copy): the logical key sequence may be cut
// into equal chunks that live in different buffers — each context-parallel rank's K/V shard inside
// its own heap, reached through its peer mapping.  The producer picks the tensor map and the row
// inside it from a small chunk table (`ChunkGeom`), everything else works on logical key positions,
// so one launch covers what a ring of per-chunk launches plus log-sum-exp merges would compute
// (3rdparty/TransformerEngine/.../context_parallel.py:94-162,676-712).  Query rows may likewise be
// two chunks with their own absolute positions (dual-chunk causal load balance).  Remote tiles are
// fetched with plain (non-multicast) TMA loads.
//
// Q, K and V are read through TMA from strided views of the packed QKV projection
// ([s, b, groups, (rep+2)·d]), so no transpose or copy precedes the kernel (the reference
// transposes sbhd→bshd and calls the FlashAttention-2 wheel:
// kareus/transformer_engine/pytorch/attention/dot_product_attention/backends.py:179-186,328-333).
#include "sm100.cuh"
#include "launch.h"
#include "pdl.cuh"
#include "host_utils.h"
#include "native_calls.h"
#include <string.h>

namespace kb {

constexpr int FA_BM = 128;      // query rows per CTA
constexpr int FA_BN = 128;      // keys per tile
constexpr int FA_D = 128;       // head dim
constexpr int FA_THREADS = 12 * 32;   // three warpgroups: the register split below is by warpgroup
constexpr int FA_REGS_SOFTMAX = 208, FA_REGS_AUX = 80;   // a row of scores lives in registers
constexpr int FA_REGS_TOTAL = 256 * FA_REGS_SOFTMAX + 128 * FA_REGS_AUX;   // must not exceed registers at launch x threads
constexpr int FA_STAGES = 5;    // K and V tiles alternate in one ring
constexpr int FA_STAGES_SINGLE = 6;   // with one query tile: the place of the second is one more stage
constexpr int FA_TILE_BYTES = FA_BN * FA_D * 2;   // 32 KB: two 64-wide swizzled chunks of 16 KB
constexpr int FA_CHUNK = 16384;

__device__ __forceinline__ float fast_exp2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

__device__ __forceinline__ float fmax3(float a, float b, float c) {
  float d;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
  return d;
}

}  // namespace kb
#include "attention_chunks.h"
namespace kb {

struct FwdParams {
  __nv_bfloat16* out;   // [sq, b, hq, d] contiguous
  float* lse;           // [b, hq, sq]
  int sq, skv, b, hq, rep;
  int q_offset;         // absolute position of query row 0 relative to key 0
  float scale_log2;     // softmax scale * log2(e)
  int causal;
  int* status;
  ChunkGeom geom;       // chunk tables (all zero: one K/V buffer, one query chunk at q_offset)
};

struct FaSmem {
  static constexpr int Q_OFF = 0;                               // two query tiles; O leaves through them as well
  static constexpr int KV_OFF = 2 * FA_TILE_BYTES;
  static constexpr int BAR_OFF = KV_OFF + FA_STAGES * FA_TILE_BYTES;
  static constexpr int TOTAL = BAR_OFF + 256 + 1024;
  static_assert(TOTAL <= 227 * 1024, "shared memory per CTA");
};

// `single`: a CTA has one query tile and warpgroup t takes its key tiles t, t + 2, ...; else warpgroup t has query tile t.
template <bool single>
__global__ void __launch_bounds__(FA_THREADS, 1)
flash_attn_fwd_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ KvMaps kv,
                      const __grid_constant__ CUtensorMap tmO, const FwdParams p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + FaSmem::BAR_OFF);
  uint64_t* q_full = bars + 0;     // [2] per query tile
  uint64_t* full = bars + 2;       // [stages] K(j) is in stage 2j, V(j) in stage 2j + 1 (modulo the ring)
  uint64_t* empty = bars + 8;      // [stages]
  uint64_t* s_full = bars + 14;    // [2] scores are in TMEM (and the tile's previous P·V has retired)
  uint64_t* p_most = bars + 16;    // [2] P of the first 96 keys is in TMEM (one arrival per warp)
  uint64_t* p_rest = bars + 18;    // [2] P of the last 32 keys
  uint64_t* o_full = bars + 20;    // [2] the tile's last P·V has retired
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 22);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;

  // late query tiles see the most keys: they go first, over all heads and batches, so that the short ones fill the end
  const int n_qtiles = (p.sq + FA_BM - 1) / FA_BM;
  const int bh = static_cast<int>(blockIdx.x) % (p.hq * p.b), from_last = static_cast<int>(blockIdx.x) / (p.hq * p.b);
  constexpr int tiles_per_cta = single ? 1 : 2;
  const int qt0 = ((n_qtiles - 1) / tiles_per_cta - from_last) * tiles_per_cta;
  const int batch = bh / p.hq, head = bh - batch * p.hq;
  const int g = head / p.rep, r = head % p.rep;
  constexpr int stages = single ? FA_STAGES_SINGLE : FA_STAGES;
  constexpr int kv_off = single ? FaSmem::KV_OFF - FA_TILE_BYTES : FaSmem::KV_OFF;
  // warpgroup t: first query row, are there such rows, key tiles that it walks
  auto tile_q0 = [&](int t) { return (single ? qt0 : qt0 + t) * FA_BM; };
  auto tile_valid = [&](int t) { return single || qt0 + t < n_qtiles; };
  auto tile_nkv = [&](int t) {
    if (!tile_valid(t)) return 0;
    const int q0 = tile_q0(t);
    int kv_end = p.skv;    // keys visible to the tile: [0, kv_end)
    if (p.causal) kv_end = min(p.skv, p.geom.q_offset_of(q0, p.q_offset) + min(q0 + FA_BM, p.sq));
    const int n = kv_end > 0 ? (kv_end + FA_BN - 1) / FA_BN : 0;
    return single ? (n + 1 - t) >> 1 : n;
  };

  if (threadIdx.x == 0) {
    for (int i = 0; i < FA_STAGES_SINGLE; ++i) {
      mbar_init(&full[i], 1);
      mbar_init(&empty[i], 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(&q_full[i], 1);
      mbar_init(&s_full[i], 1);
      mbar_init(&p_most[i], 4);
      mbar_init(&p_rest[i], 4);
      mbar_init(&o_full[i], 1);
    }
    *abort_flag = 0;
    mbar_fence_init();
  }
  if (warp == 9) tmem_alloc(tmem_slot, 512);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  pdl_begin();
  const uint32_t tmem_base = *tmem_slot;     // S|P of tile t at 128 t, O of tile t at 256 + 128 t

  if (warp >= 8) {
    regs_dec<FA_REGS_AUX>();
    if (warp == 8) {
      // ------------------------------------------------------------------ producer
      const int n0 = tile_nkv(0), n1 = tile_nkv(1), n = single ? n0 + n1 : max(n0, n1);
      if (n > 0 && elect_one()) {
        prefetch_tmap(&tmQ);
        prefetch_tmap(&kv.k[0]);
        prefetch_tmap(&kv.v[0]);
        bool okp = true;
        int st = 0;
        uint32_t ph = 1;
        auto load = [&](const CUtensorMap* map, int srow) {
          if (!mbar_wait(&empty[st], ph, abort_flag, p.status, ST_TIMEOUT_EMPTY)) { okp = false; return; }
          uint8_t* d = smem + kv_off + st * FA_TILE_BYTES;
          mbar_expect_tx(&full[st], FA_TILE_BYTES);
          tma_load_4d(d, map, &full[st], 0, g, batch, srow);
          tma_load_4d(d + FA_CHUNK, map, &full[st], 64, g, batch, srow);
          if (++st == stages) { st = 0; ph ^= 1u; }
        };
        auto load_q = [&](int t) {
          uint8_t* d = smem + FaSmem::Q_OFF + t * FA_TILE_BYTES;
          mbar_expect_tx(&q_full[t], FA_TILE_BYTES);
          tma_load_5d(d, &tmQ, &q_full[t], 0, r, g, batch, tile_q0(t));
          tma_load_5d(d + FA_CHUNK, &tmQ, &q_full[t], 64, r, g, batch, tile_q0(t));
        };
        if (n0 > 0) load_q(0);
        for (int j = 0; j < n && okp; ++j) {
          int src, srow;
          p.geom.locate(j * FA_BN, src, srow);
          load(&kv.k[src], srow);
          if (j == 0 && n1 > 0 && !single) load_q(1);
          if (okp) load(&kv.v[src], srow);
        }
        if (*abort_flag) {
          const uint64_t t0 = globaltimer_ns();
          while (globaltimer_ns() - t0 < 200000ull) {}
        }
      }
      __syncwarp();
    } else if (warp == 9) {
      // ------------------------------------------------------------------ MMA issuer
      const int n0 = tile_nkv(0), n1 = tile_nkv(1), n = single ? n0 + n1 : max(n0, n1);
      if (n > 0 && elect_one()) {             // one thread runs the whole role, see elect_one()
        constexpr uint32_t idesc_s = make_idesc_bf16(FA_BM, FA_BN, false, false);  // Q K-major, K K-major
        constexpr uint32_t idesc_o = make_idesc_bf16(FA_BM, FA_D, false, true);    // P (TMEM), V MN-major
        const uint32_t smem0 = smem_u32(smem);
        const uint64_t qd0 = make_smem_desc(smem0 + FaSmem::Q_OFF, 16, 1024);
        const uint64_t kd0 = make_smem_desc(smem0 + kv_off, 16, 1024);
        const uint64_t vd0 = make_smem_desc(smem0 + kv_off, FA_CHUNK, 1024);
        bool ok = true;
        auto wait = [&](uint64_t* bar, uint32_t parity, int code) {
          if (ok) ok = mbar_wait(bar, parity, abort_flag, p.status, code);
          return ok;
        };
        // scores of warpgroup t from query tile `qt` and the K in stage ks
        auto issue_s = [&](int t, int qt, int ks) {
          const uint64_t qd = qd0 + static_cast<uint64_t>(qt * (FA_TILE_BYTES >> 4));
          const uint64_t kd = kd0 + static_cast<uint64_t>(ks * (FA_TILE_BYTES >> 4));
          const uint32_t d = tmem_base + t * 128;
#pragma unroll
          for (int k = 0; k < FA_D / 16; ++k) {
            const uint64_t off = ((k >> 2) * FA_CHUNK + (k & 3) * 32) >> 4;
            umma_ss(d, qd + off, kd + off, idesc_s, k > 0 ? 1u : 0u);
          }
          umma_commit(&s_full[t]);
        };
        // O of warpgroup t += P · (V in stage vs), for its i-th key tile
        auto issue_pv = [&](int t, int vs, int i) {
          const uint64_t vd = vd0 + static_cast<uint64_t>(vs * (FA_TILE_BYTES >> 4));
          const uint32_t d = tmem_base + 256 + t * 128, a = tmem_base + t * 128;
          if (!wait(&p_most[t], i & 1u, ST_TIMEOUT_TMEM_FULL)) return;
          tc_fence_after();
#pragma unroll
          for (int k = 0; k < 6; ++k)            // 16 keys: 8 columns of P, 16 rows of V
            umma_ts(d, a + k * 8, vd + k * (2048 >> 4), idesc_o, (i > 0 || k > 0) ? 1u : 0u);
          if (!wait(&p_rest[t], i & 1u, ST_TIMEOUT_TMEM_FULL)) return;
          tc_fence_after();
#pragma unroll
          for (int k = 6; k < 8; ++k) umma_ts(d, a + k * 8, vd + k * (2048 >> 4), idesc_o, 1u);
        };
        if constexpr (single) {
          // scores of key tile j; they overwrite P of tile j - 2: the products before them read it in order
          auto scores = [&](int j) {
            const int x = 2 * j, st = x % FA_STAGES_SINGLE;
            if (!wait(&full[st], (x / FA_STAGES_SINGLE) & 1u, ST_TIMEOUT_FULL)) return;
            tc_fence_after();
            issue_s(j & 1, 0, st);
            umma_commit(&empty[st]);
          };
          if (wait(&q_full[0], 0, ST_TIMEOUT_FULL)) {
            scores(0);
            if (n > 1) scores(1);
          }
          for (int j = 0; j < n && ok; ++j) {
            const int x = 2 * j + 1, st = x % FA_STAGES_SINGLE;
            if (!wait(&full[st], (x / FA_STAGES_SINGLE) & 1u, ST_TIMEOUT_FULL)) break;
            issue_pv(j & 1, st, j >> 1);
            if (!ok) break;
            umma_commit(&empty[st]);
            if (j + 2 < n) scores(j + 2);
            else umma_commit(&o_full[j & 1]);
          }
        } else {
          int ks = 0;                                // stage of K(j) / K(j+1), its phase
          uint32_t kph = 0;
          if (wait(&full[0], 0, ST_TIMEOUT_FULL)) {
#pragma unroll
            for (int t = 0; t < 2; ++t)
              if ((t ? n1 : n0) > 0 && wait(&q_full[t], 0, ST_TIMEOUT_FULL)) {
                tc_fence_after();
                issue_s(t, t, 0);
              }
            if (ok) umma_commit(&empty[0]);
          }
          for (int j = 0; j < n && ok; ++j) {
            int vs = ks + 1;
            uint32_t vph = kph;
            if (vs == FA_STAGES) { vs = 0; vph ^= 1u; }
            ks = vs + 1;
            kph = vph;
            if (ks == FA_STAGES) { ks = 0; kph ^= 1u; }
            if (!wait(&full[vs], vph, ST_TIMEOUT_FULL)) break;
#pragma unroll
            for (int t = 0; t < 2; ++t) {
              const int nt = t ? n1 : n0;
              if (j >= nt || !ok) continue;
              issue_pv(t, vs, j);
              if (!ok) continue;
              if (j + 1 < nt) {
                if (!wait(&full[ks], kph, ST_TIMEOUT_FULL)) continue;
                tc_fence_after();
                issue_s(t, t, ks);                   // overwrites P: the products before it read it in order
              } else {
                umma_commit(&o_full[t]);
              }
            }
            if (!ok) break;
            umma_commit(&empty[vs]);
            if (j + 1 < n) umma_commit(&empty[ks]);
          }
        }
      }
      __syncwarp();
    }
  } else {
    regs_inc<FA_REGS_SOFTMAX>();
    // ------------------------------------------------------------------ softmax + epilogue
    const int t = warp >> 2;                       // query tile, or share of the key tiles of the one
    const int row = (warp & 3) * 32 + lane;        // row inside the tile = TMEM lane
    const int n_kv = tile_nkv(t);
    const int q0 = tile_q0(t);
    const int qrow = q0 + row;
    const int q_off = tile_valid(t) ? p.geom.q_offset_of(q0, p.q_offset) : 0;
    const uint32_t lane_addr = static_cast<uint32_t>((warp & 3) * 32) << 16;
    const uint32_t t_s = tmem_base + t * 128 + lane_addr, t_o = tmem_base + 256 + t * 128 + lane_addr;
    const uint32_t all = 0xffffffffu;
    float m_ref = -INFINITY;   // reference maximum (scaled, log2 domain) used for the exponentials
    float l_sum = 0.f;
    const int key_first = single ? t * FA_BN : 0, key_step = single ? 2 * FA_BN : FA_BN;
    bool ok = true;            // warp-uniform
    for (int j = 0; j < n_kv; ++j) {
      ok = mbar_wait_warp(&s_full[t], j & 1u, abort_flag, p.status, ST_TIMEOUT_TMEM_FULL);
      if (!ok) break;
      tc_fence_after();
      uint32_t v[4][32];
#pragma unroll
      for (int c = 0; c < 4; ++c) tmem_ld_32x32(t_s + c * 32, v[c]);
      tmem_ld_wait();
      const int key0 = key_first + j * key_step;
      // warp-uniform: does any row of this tile need masking?
      if ((p.causal && key0 + FA_BN - 1 > q_off + q0) || (key0 + FA_BN > p.skv)) {
        // keys at or above `lim` (relative to this tile) are hidden from this row
        const int lim = min(p.causal ? q_off + qrow + 1 : p.skv, p.skv) - key0;
#pragma unroll
        for (int c = 0; c < 4; ++c)
#pragma unroll
          for (int i = 0; i < 32; ++i)
            if (c * 32 + i >= lim) v[c][i] = 0xff800000u;   // -inf
      }
      float mx4[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
      for (int c = 0; c < 4; ++c)
#pragma unroll
        for (int i = 0; i < 32; i += 8)
#pragma unroll
          for (int h = 0; h < 4; ++h)
            mx4[h] = fmax3(mx4[h], __uint_as_float(v[c][i + 2 * h]), __uint_as_float(v[c][i + 2 * h + 1]));
      const float mx = fmaxf(fmaxf(mx4[0], mx4[1]), fmaxf(mx4[2], mx4[3])) * p.scale_log2;
      float rescale = 1.f;
      if (mx > m_ref + 8.f) {       // also true on the first tile (m_ref = -inf)
        rescale = m_ref == -INFINITY ? 1.f : fast_exp2(m_ref - mx);
        m_ref = mx;
      }
      // s_full also covers the tile's previous P·V, so O is at rest here; made warp-uniform for the .aligned accesses
      if (__any_sync(all, rescale != 1.f)) {
#pragma unroll 1
        for (int c = 0; c < 4; ++c) {
          uint32_t o[32];
          tmem_ld_32x32(t_o + c * 32, o);
          tmem_ld_wait();
#pragma unroll
          for (int i = 0; i < 32; ++i) o[i] = __float_as_uint(__uint_as_float(o[i]) * rescale);
          tmem_st_32x32(t_o + c * 32, o);
        }
        tmem_st_wait();
      }
      const float mref = (m_ref == -INFINITY) ? 0.f : m_ref;
      const float2 sc2 = make_float2(p.scale_log2, p.scale_log2);
      const float2 nm2 = make_float2(-mref, -mref);
      float2 ps2[2] = {make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
      // P = exp2(S·scale − m) of 32 keys: partial row sum, bf16 pairs into 16 columns of TMEM
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        uint32_t w[16];
#pragma unroll
        for (int i = 0; i < 16; ++i) {
          float2 x = __ffma2_rn(make_float2(__uint_as_float(v[c][2 * i]), __uint_as_float(v[c][2 * i + 1])), sc2, nm2);
          x.x = fast_exp2(x.x);
          x.y = fast_exp2(x.y);
          ps2[i & 1] = __fadd2_rn(ps2[i & 1], x);
          w[i] = pack_bf16x2(x.x, x.y);
        }
        tmem_st_32x32_x16(t_s + c * 16, w);
        if (c >= 2) {
          tmem_st_wait();
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(c == 2 ? &p_most[t] : &p_rest[t]);
        }
      }
      l_sum = l_sum * rescale + ((ps2[0].x + ps2[0].y) + (ps2[1].x + ps2[1].y));
    }
    // ---- epilogue: O / l through the query tile's Q buffer (the warp's 32 rows) and a TMA store; LSE
    float* lse = p.lse + (static_cast<size_t>(batch) * p.hq + head) * p.sq;
    // two 64-wide halves of 32 rows x 128 bytes, 16-byte units swizzled by row as the tensor map expects
    uint8_t* stg = smem + FaSmem::Q_OFF + (single ? 0 : t) * FA_TILE_BYTES + (warp & 3) * 8192;
    const int row0 = q0 + (warp & 3) * 32;
    auto stage32 = [&](int c, const uint32_t (&o)[32], float f) {     // columns 32c.. of this thread's row, times f
      const uint32_t stg_row = smem_u32(stg) + lane * 128;
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        uint32_t w[4];
#pragma unroll
        for (int h = 0; h < 4; ++h)
          w[h] = pack_bf16x2(__uint_as_float(o[8 * u + 2 * h]) * f, __uint_as_float(o[8 * u + 2 * h + 1]) * f);
        const int unit = (c & 1) * 4 + u;
        st_shared_v4(stg_row + (c >> 1) * 4096 + ((unit ^ (lane & 7)) << 4), w[0], w[1], w[2], w[3]);
      }
    };
    auto put_lse = [&](float m, float l) {
      if (qrow < p.sq) lse[qrow] = (l > 0.f) ? (m + log2f(l)) * 0.6931471805599453f : -INFINITY;
    };
    if (tile_valid(t) && (single ? tile_nkv(0) : n_kv) == 0) {
      // no visible key at all (only possible with a negative q_offset): zero output
      if (qrow < p.sq && !(single && t)) {
        uint4* orow = reinterpret_cast<uint4*>(p.out + ((static_cast<size_t>(qrow) * p.b + batch) * p.hq + head) * FA_D);
        for (int i = 0; i < FA_D / 8; ++i) orow[i] = make_uint4(0, 0, 0, 0);
        lse[qrow] = -INFINITY;
      }
    } else if constexpr (single) {
      // Both warpgroups put their maximum and sum where the key tiles were (all products have retired) and each writes
      // half of the columns of O = (O_0 2^(m_0 - m) + O_1 2^(m_1 - m)) / l.  A warp whose waits failed comes to the
      // barrier as well; the abort flag, set by then, keeps all of them from storing.
      for (int h = 0; h < 2; ++h)
        if (ok && tile_nkv(h) > 0) ok = mbar_wait_warp(&o_full[h], 0, abort_flag, p.status, ST_TIMEOUT_TMEM_FULL);
      tc_fence_after();
      float2* stat = reinterpret_cast<float2*>(smem + kv_off);           // [2][128]
      stat[t * FA_BM + row] = make_float2(m_ref, l_sum);
      asm volatile("bar.sync 1, 256;" ::: "memory");
      ok = __all_sync(all, ok && *abort_flag == 0);
      if (ok) {
        const float2 s0 = stat[row], s1 = stat[FA_BM + row];
        const float m = fmaxf(s0.x, s1.x);
        // a share without visible keys has l = 0 and an O that was never written; a NaN sum stays visible
        const bool use0 = s0.y != 0.f, use1 = s1.y != 0.f;
        const float f0 = s0.x == m ? 1.f : fast_exp2(s0.x - m), f1 = s1.x == m ? 1.f : fast_exp2(s1.x - m);
        const float l = (use0 ? s0.y * f0 : 0.f) + (use1 ? s1.y * f1 : 0.f);
        const float inv = l > 0.f ? 1.f / l : 0.f;
#pragma unroll 1
        for (int c2 = 0; c2 < 2; ++c2) {
          const int c = 2 * t + c2;
          uint32_t o0[32], o1[32];
          tmem_ld_32x32(tmem_base + 256 + lane_addr + c * 32, o0);
          tmem_ld_32x32(tmem_base + 384 + lane_addr + c * 32, o1);
          tmem_ld_wait();
#pragma unroll
          for (int i = 0; i < 32; ++i)
            o0[i] = __float_as_uint((use0 ? __uint_as_float(o0[i]) * f0 : 0.f) + (use1 ? __uint_as_float(o1[i]) * f1 : 0.f));
          stage32(c, o0, inv);
        }
        fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0 && row0 < p.sq) {                // the tensor map clips rows past sq
          tma_store_4d(&tmO, stg + t * 4096, 64 * t, head, batch, row0);
          tma_store_commit();
        }
        if (t == 0) put_lse(m, l);
        if (lane == 0) tma_store_wait<0>();            // nothing in flight out of shared memory at exit
      }
    } else if (n_kv > 0) {
      if (ok) ok = mbar_wait_warp(&o_full[t], 0, abort_flag, p.status, ST_TIMEOUT_TMEM_FULL);
      if (ok) {
        tc_fence_after();
        const float inv = l_sum > 0.f ? 1.f / l_sum : 0.f;
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          uint32_t o[32];
          tmem_ld_32x32(t_o + c * 32, o);
          tmem_ld_wait();
          stage32(c, o, inv);
        }
        fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0 && row0 < p.sq) {                // the tensor map clips rows past sq
          tma_store_4d(&tmO, stg, 0, head, batch, row0);
          tma_store_4d(&tmO, stg + 4096, 64, head, batch, row0);
          tma_store_commit();
        }
        put_lse(m_ref, l_sum);
        if (lane == 0) tma_store_wait<0>();            // nothing in flight out of shared memory at exit
      }
    }
    __syncwarp();
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 9) {
    tc_fence_after();
    tmem_dealloc(tmem_base, 512);
  }
}

}  // namespace kb

namespace kb {

static int make_q_map(CUtensorMap* m, const void* q, int d, int rep, int g, int b, int sq, long qs_s, long qs_b,
                      long qs_g, long qs_r) {
  uint64_t dims[5] = {(uint64_t)d, (uint64_t)rep, (uint64_t)g, (uint64_t)b, (uint64_t)sq};
  uint64_t str[4] = {(uint64_t)qs_r * 2, (uint64_t)qs_g * 2, (uint64_t)qs_b * 2, (uint64_t)qs_s * 2};
  uint32_t box[5] = {64, 1, 1, 1, FA_BM};
  // a size-1 dimension may carry any stride; TMA still wants it to be a multiple of 16 bytes
  for (int i = 0; i < 4; ++i) if (str[i] == 0 || (str[i] & 15)) str[i] = (uint64_t)d * 2;
  return make_tmap(m, q, 2, 5, dims, str, box, 3);
}

static int make_kv_map(CUtensorMap* m, const void* ptr, int d, int g, int b, int rows, long s_s, long s_b, long s_g) {
  uint64_t dims[4] = {(uint64_t)d, (uint64_t)g, (uint64_t)b, (uint64_t)rows};
  uint32_t box[4] = {64, 1, 1, FA_BN};
  uint64_t str[3] = {(uint64_t)s_g * 2, (uint64_t)s_b * 2, (uint64_t)s_s * 2};
  for (int i = 0; i < 3; ++i) if (str[i] == 0 || (str[i] & 15)) str[i] = (uint64_t)d * 2;
  return make_tmap(m, ptr, 2, 4, dims, str, box, 3);
}

template <bool single>
static int launch_variant(const CUtensorMap& tmQ, const KvMaps& kv, const CUtensorMap& tmO, const FwdParams& p, int ctas,
                          cudaStream_t stream) {
  auto kern = flash_attn_fwd_kernel<single>;
  static bool configured = false;
  if (!configured) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, FaSmem::TOTAL);
    if (e != cudaSuccess) return 1000 + (int)e;
    cudaFuncAttributes attr;
    e = cudaFuncGetAttributes(&attr, kern);
    if (e != cudaSuccess) return 1000 + (int)e;
    if (attr.numRegs * FA_THREADS < FA_REGS_TOTAL) return ST_BAD_ARG;   // the register split would wait forever
    configured = true;
  }
  KB_LAUNCH_PDL(kern, (unsigned)ctas, FA_THREADS, FaSmem::TOTAL, stream, tmQ, kv, tmO, p);
  const cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? 0 : 2000 + (int)e;
}

static int launch_fwd(const CUtensorMap& tmQ, const KvMaps& kv, const ChunkGeom& geom, void* out, float* lse, int sq,
                      int skv, int b, int g, int rep, float scale, int causal, int q_offset, int* status,
                      cudaStream_t stream) {
  FwdParams p;
  p.out = reinterpret_cast<__nv_bfloat16*>(out);
  p.lse = lse;
  p.sq = sq; p.skv = skv; p.b = b; p.hq = g * rep; p.rep = rep;
  p.q_offset = q_offset;
  p.scale_log2 = scale * 1.4426950408889634f;
  p.causal = causal;
  p.status = status;
  p.geom = geom;
  CUtensorMap tmO;
  {
    // [sq, b, hq, d]: boxes of 32 rows x 64 columns of one (batch, head)
    const uint64_t hq = (uint64_t)g * rep;
    uint64_t dims[4] = {FA_D, hq, (uint64_t)b, (uint64_t)sq};
    uint64_t str[3] = {FA_D * 2, hq * FA_D * 2, (uint64_t)b * hq * FA_D * 2};
    uint32_t box[4] = {64, 1, 1, 32};
    const int rc = make_tmap(&tmO, out, 2, 4, dims, str, box, 3);
    if (rc) return rc;
  }
  // Pairs of query tiles halve the K/V traffic; where single tiles already fit the chip in one wave, they halve the
  // work of the longest CTA instead.  One key tile cannot be shared, and the meeting of the warpgroups costs 0.5 us.
  const int n_q = (sq + FA_BM - 1) / FA_BM, bh = g * rep * b;
  if (skv > FA_BN && (long)n_q * bh <= device_sm_count()) return launch_variant<true>(tmQ, kv, tmO, p, bh * n_q, stream);
  return launch_variant<false>(tmQ, kv, tmO, p, bh * ((n_q + 1) / 2), stream);
}

}  // namespace kb

// q: view [sq, b, g, rep, d] (strides in elements, d contiguous); k, v: views [skv, b, g, d];
// out: [sq, b, g*rep, d] contiguous; lse: [b, g*rep, sq] fp32.
extern "C" int kb_flash_attn_fwd(const void* q, long qs_s, long qs_b, long qs_g, long qs_r, const void* k, long ks_s,
                                 long ks_b, long ks_g, const void* v, long vs_s, long vs_b, long vs_g, void* out,
                                 float* lse, int sq, int skv, int b, int g, int rep, int d, float scale, int causal,
                                 int q_offset, int* status, cudaStream_t stream) {
  using namespace kb;
  if (d != FA_D || sq <= 0 || skv <= 0) return ST_BAD_ARG;
  CUtensorMap tmQ;
  KvMaps kv;
  memset(&kv, 0, sizeof(kv));
  int rc = make_q_map(&tmQ, q, d, rep, g, b, sq, qs_s, qs_b, qs_g, qs_r);
  if (rc) return rc;
  rc = make_kv_map(&kv.k[0], k, d, g, b, skv, ks_s, ks_b, ks_g);
  if (rc) return rc;
  rc = make_kv_map(&kv.v[0], v, d, g, b, skv, vs_s, vs_b, vs_g);
  if (rc) return rc;
  ChunkGeom geom;
  memset(&geom, 0, sizeof(geom));
  return launch_fwd(tmQ, kv, geom, out, lse, sq, skv, b, g, rep, scale, causal, q_offset, status, stream);
}

// Chunked variant.  The logical key sequence is `n_chunks` chunks of `chunk_rows` keys (a multiple of
// 128); chunk c lives in source buffer kv_src[c] (0..n_src-1) starting at row kv_row_base[c].  Every
// source is a [src_rows, b, g, d] view with the strides given (the same for all sources); k_ptrs and
// v_ptrs hold their base addresses, which may be peer mappings of other GPUs' memory.  The local
// queries are `sq / q_chunk_rows` chunks whose first rows sit at absolute positions q_pos[i].
extern "C" int kb_flash_attn_fwd_chunked(const void* q, long qs_s, long qs_b, long qs_g, long qs_r,
                                         const void* const* k_ptrs, const void* const* v_ptrs, int n_src, int src_rows,
                                         long ks_s, long ks_b, long ks_g, long vs_s, long vs_b, long vs_g,
                                         const int* kv_src, const int* kv_row_base, int n_chunks, int chunk_rows,
                                         int q_chunk_rows, const int* q_pos, void* out, float* lse, int sq, int b, int g,
                                         int rep, int d, float scale, int causal, int* status, cudaStream_t stream) {
  using namespace kb;
  ChunkGeom geom;
  int rc = fill_chunk_geom(&geom, n_src, kv_src, kv_row_base, n_chunks, chunk_rows, src_rows, q_chunk_rows, q_pos, sq);
  if (rc || d != FA_D) return ST_BAD_ARG;
  CUtensorMap tmQ;
  KvMaps kv;
  memset(&kv, 0, sizeof(kv));
  rc = make_q_map(&tmQ, q, d, rep, g, b, sq, qs_s, qs_b, qs_g, qs_r);
  if (rc) return rc;
  for (int i = 0; i < n_src; ++i) {
    rc = make_kv_map(&kv.k[i], k_ptrs[i], d, g, b, src_rows, ks_s, ks_b, ks_g);
    if (rc) return rc;
    rc = make_kv_map(&kv.v[i], v_ptrs[i], d, g, b, src_rows, vs_s, vs_b, vs_g);
    if (rc) return rc;
  }
  return launch_fwd(tmQ, kv, geom, out, lse, sq, n_chunks * chunk_rows, b, g, rep, scale, causal, 0, status, stream);
}
