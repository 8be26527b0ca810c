// Absorbed latent attention for the rows of prompt chunks on the 5th-generation tensor cores. Cache rows of 512 + 64 columns:
// a token's score is a dot product over all 576, its value is the first 512. Same results as mla_decode.cu, whose CTA serves one
// token's 16 heads on mma.sync and streams the whole context for it.
//
// Here a CTA takes 128 query rows = 128 / H neighbouring tokens of one sequence with all H heads, and ONE HALF of the value
// columns: O[128, 256] is 256 of the 512 TMEM columns, which leaves room for two score tiles and for part of the query. The two
// CTAs of a row block both compute the scores: 832 multiply-adds per (row, key) instead of 544, in exchange for no traffic
// between them. What bounds it is shared memory: an operand pair of 128 x 16 and 64 x 16 takes 48 cycles to read and 32 to
// multiply, so four of the nine 64-column pieces of the query live in TMEM, and P is read from TMEM as well.
//
//   TMEM columns   [0, 256) O   [256, 320) S_0 / P_0   [320, 384) S_1 / P_1   [384, 512) query columns 0 .. 255, bf16
//   shared memory  query pieces 4 .. 8 (80 KB), two key tiles of 64 tokens (nine 64 x 64 pieces of 8 KB each)
//
// 320 threads: warp 0 loads, warp 1 owns TMEM and issues the MMAs, warps 2-9 do the softmax with two threads per row. P_j is
// written over S_j. O stays in TMEM for the whole row block; it is rescaled where a row's maximum has grown, behind the weights, so that
// the largest weight is always 1, which bf16 holds exactly (with weights that may grow to 2^8 first: a tenth faster when the case below
// took 247 us, and an error of 0.0021 against 64 bits instead of 0.0019). A key tile has two parts with
// barriers of their own: the half of its columns that this CTA also uses as values is busy until P V, the rest only until the
// scores are done, so that most of the next tile but one is on its way early. P_j V_j is issued between the two parts of S_{j+1}, or behind
// both: that S_{j+1} is there only says that P_{j-1} V_{j-1} is done. Products alternate between two barriers, since a warp that has not
// rescaled may ask for the last one while the one before is still to come, and a single barrier's parity would not tell them apart.
//
// Measured, three chunks of 750 - 1500 tokens, 16 heads: 233 us a call (506 TFLOP/s counted without the second scores), against 898; 212 where a graph
// replays the launch.
//
// Every wait is bounded as in attention_tc.cu: a role that gives up records TIMEOUT and raises a flag for the others.
#include <cstdint>
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include "b2/api.h"
#include "b2/config.h"
#include "b2/launch.h"
#include "b2/ptx.cuh"
#include "b2/status.h"
#include "b2/tma.h"

namespace b2 {
namespace {

constexpr int kRows = 128, kKeys = 64, kThreads = 320;
constexpr int kPieces = 9, kValuePieces = 4;                     // 64-column pieces of a row; of this CTA's half of the values
constexpr int kPieceBytes = kKeys * 128;                         // 64 tokens x 64 columns
constexpr int kQPieceBytes = kRows * 128;
constexpr int kKeyBytes = kPieces * kPieceBytes;
constexpr int kOwnBytes = kValuePieces * kPieceBytes, kRestBytes = kKeyBytes - kOwnBytes;
constexpr int kQTmem = 4;                                        // query pieces in TMEM
constexpr int kOffK = (kPieces - kQTmem) * kQPieceBytes;         // 80 KB of query, then the keys
constexpr int kOffMax = kOffK + 2 * kKeyBytes;                   // float [2][2][128]
constexpr int kOffBar = kOffMax + 4 * kRows * 4;
constexpr int kNumBars = 17;
constexpr int kOffFlags = kOffBar + kNumBars * 8;
constexpr int kSmem = kOffFlags + 16;
static_assert(kSmem <= kMaxSmemPerCta, "shared memory");
constexpr uint32_t kColS = 256, kColQ = 384;

struct MlaTcParams {
  const __nv_bfloat16* q_lat;
  __nv_bfloat16* out;             // [T, H, 512]
  int64_t q_stride;
  const int *cu_q, *ctx_lens, *block_tables;
  int max_blocks, heads, tokens, page_size;      // tokens: of a row block, 128 / heads
  int64_t num_pages;
  float scale_log2;
};

// MN-major operand (values: rows are tokens): `lbo` between 64-column pieces, 1 KB between groups of 8 tokens, 128-byte swizzle
__device__ __forceinline__ uint64_t value_desc(uint32_t addr) {
  uint64_t d = 0;
  d |= static_cast<uint64_t>((addr & 0x3FFFF) >> 4);
  d |= static_cast<uint64_t>(kPieceBytes >> 4) << 16;
  d |= static_cast<uint64_t>(1024 >> 4) << 32;
  d |= static_cast<uint64_t>(1) << 46;
  d |= static_cast<uint64_t>(2) << 61;
  return d;
}

__global__ void __launch_bounds__(kThreads, 1)
mla_prefill_tc_kernel(const __grid_constant__ CUtensorMap tmap_q, const __grid_constant__ CUtensorMap tmap_r, const __grid_constant__ CUtensorMap tmap_kv,
                      MlaTcParams prm, Status* status) {
  ptx::grid_dep_sync();
  const int half = blockIdx.x & 1, seq = blockIdx.y;
  const int q_begin = prm.cu_q[seq], q_len = prm.cu_q[seq + 1] - q_begin;
  const int blocks = (q_len + prm.tokens - 1) / prm.tokens, turn = blockIdx.x >> 1;
  if (turn >= blocks) return;                              // uniform per CTA: before any barrier or allocation
  const int qb = blocks - 1 - turn;                        // longest contexts first
  const int ctx = prm.ctx_lens[seq];
  const int pos0 = ctx - q_len + qb * prm.tokens;          // position of the block's first token
  const int tok0 = q_begin + qb * prm.tokens, n_tok = min(prm.tokens, q_len - qb * prm.tokens);
  const int n_tiles = (min(ctx, pos0 + n_tok) + kKeys - 1) / kKeys;

  extern __shared__ __align__(1024) uint8_t smem[];
  const uint32_t base = ptx::smem_u32(smem);
  auto bar = [&](int i) { return base + kOffBar + 8u * i; };
  const uint32_t q_full = bar(0), q_tmem = bar(1), drain_bar = bar(16);
  auto pv_done = [&](int a) { return bar(2 + a); };
  auto own_full = [&](int s) { return bar(4 + s); };
  auto rest_full = [&](int s) { return bar(6 + s); };
  auto own_empty = [&](int s) { return bar(8 + s); };
  auto rest_empty = [&](int s) { return bar(10 + s); };
  auto s_full = [&](int a) { return bar(12 + a); };
  auto p_full = [&](int a) { return bar(14 + a); };
  float* row_max = reinterpret_cast<float*>(smem + kOffMax);
  uint32_t* tmem_holder = reinterpret_cast<uint32_t*>(smem + kOffFlags);
  volatile uint32_t* fail = reinterpret_cast<volatile uint32_t*>(smem + kOffFlags + 4);

  const int warp = ptx::warp_id(), lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    ptx::prefetch_tensormap(&tmap_q);
    ptx::prefetch_tensormap(&tmap_r);
    ptx::prefetch_tensormap(&tmap_kv);
    ptx::mbar_init(q_full, 1);
    ptx::mbar_init(q_tmem, 8);
    ptx::mbar_init(drain_bar, 1);
    for (int s = 0; s < 2; ++s) {
      ptx::mbar_init(own_full(s), 1);
      ptx::mbar_init(rest_full(s), 1);
      ptx::mbar_init(own_empty(s), 1);
      ptx::mbar_init(rest_empty(s), 1);
      ptx::mbar_init(s_full(s), 1);
      ptx::mbar_init(p_full(s), 8);
      ptx::mbar_init(pv_done(s), 1);
    }
    ptx::fence_mbar_init();
    *fail = (base & 1023u) != 0;      // the swizzle needs the alignment
  }
  if (warp == 1) {
    ptx::tmem_alloc(ptx::smem_u32(tmem_holder), 512);
    ptx::tmem_relinquish();
  }
  ptx::tc_fence_before();
  __syncthreads();
  ptx::tc_fence_after();
  const uint32_t tmem = *tmem_holder;
  auto give_up = [&](int a, int b) {
    status_record(status, kTimeout, kSiteAttn, a, b);
    *fail = 1;
  };
  // column piece at place i of a key tile: this CTA's values first, then the other half's columns and the rotated part
  auto piece = [&](int i) { return i < kValuePieces ? half * kValuePieces + i : i < 8 ? (half ^ 1) * kValuePieces + i - kValuePieces : 8; };
  const bool aligned = *fail == 0;
  if (!aligned && threadIdx.x == 0) status_record(status, kBadArgument, kSiteAttn, 20, 0);

  if (!aligned) {
  } else if (warp == 0) {
    // ------------------------------------------------------------------ loads
    if (ptx::elect_one()) {
      ptx::mbar_arrive_expect_tx(q_full, (kPieces - kQTmem) * prm.tokens * prm.heads * 128);
      for (int c = kQTmem; c < kPieces; ++c) {
        if (c < 8) ptx::tma_load_3d(base + (c - kQTmem) * kQPieceBytes, &tmap_q, q_full, c * 64, 0, tok0, ptx::kEvictFirst);
        else ptx::tma_load_3d(base + (c - kQTmem) * kQPieceBytes, &tmap_r, q_full, 0, 0, tok0, ptx::kEvictFirst);
      }
      bool ok = true;
      int own_n = 0, rest_n = 0;
      for (int j = 0; j < n_tiles && ok; ++j) {
        const int s = j & 1, pos = j * kKeys;
        const uint32_t ph = static_cast<uint32_t>((j >> 1) & 1), at = base + kOffK + s * kKeyBytes;
        int page = prm.block_tables[static_cast<int64_t>(seq) * prm.max_blocks + pos / prm.page_size];
        if (page < 0 || page >= prm.num_pages) {
          status_record(status, kOutOfBounds, kSiteKvIndex, seq, page);
          page = 0;
        }
        const int row = page * prm.page_size + pos % prm.page_size;
        if (!ptx::mbar_wait(rest_empty(s), ph ^ 1u)) { give_up(1, j); ok = false; break; }
        ptx::mbar_arrive_expect_tx(rest_full(s), kRestBytes);
        for (int i = kValuePieces; i < kPieces; ++i) ptx::tma_load_2d(at + i * kPieceBytes, &tmap_kv, rest_full(s), piece(i) * 64, row, ptx::kEvictNormal);
        ++rest_n;
        if (!ptx::mbar_wait(own_empty(s), ph ^ 1u)) { give_up(2, j); ok = false; break; }
        ptx::mbar_arrive_expect_tx(own_full(s), kOwnBytes);
        for (int i = 0; i < kValuePieces; ++i) ptx::tma_load_2d(at + i * kPieceBytes, &tmap_kv, own_full(s), piece(i) * 64, row, ptx::kEvictNormal);
        ++own_n;
      }
      if (!ok) {
        // let the copies this thread started land before the CTA gives up its shared memory
        ptx::mbar_wait(q_full, 0, 200000000ull);
        for (int j = max(0, rest_n - 2); j < rest_n; ++j) ptx::mbar_wait(rest_full(j & 1), (j >> 1) & 1, 200000000ull);
        for (int j = max(0, own_n - 2); j < own_n; ++j) ptx::mbar_wait(own_full(j & 1), (j >> 1) & 1, 200000000ull);
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    // ------------------------------------------------------------------ MMAs
    if (ptx::elect_one()) {
      constexpr uint32_t idesc_s = ptx::make_idesc(1, 1, kRows, kKeys);
      constexpr uint32_t idesc_o = ptx::make_idesc(1, 1, kRows, 256) | (1u << 16);      // values are MN-major
      bool ok = true;
      // pieces [n0, n1) of S_j in the order in which they arrive: the rest (0 .. 4), then the own half (5 .. 8)
      auto issue_s = [&](int j, int n0, int n1) {
        const uint32_t d = tmem + kColS + (j & 1) * kKeys, at = base + kOffK + (j & 1) * kKeyBytes;
        for (int n = n0; n < n1; ++n) {
          const int i = n < kPieces - kValuePieces ? n + kValuePieces : n - (kPieces - kValuePieces), c = piece(i);
          const uint64_t db = ptx::make_smem_desc_sw128(at + i * kPieceBytes);
          if (c < kQTmem) {
#pragma unroll
            for (int k = 0; k < 4; ++k) ptx::mma_tmem_a(d, tmem + kColQ + c * 32 + k * 8, db + 2u * k, idesc_s, (n | k) ? 1u : 0u);
          } else {
            const uint64_t da = ptx::make_smem_desc_sw128(base + (c - kQTmem) * kQPieceBytes);
#pragma unroll
            for (int k = 0; k < 4; ++k) ptx::tc_mma_f16(d, da + 2u * k, db + 2u * k, idesc_s, (n | k) ? 1u : 0u);
          }
        }
      };
      auto first_part = [&](int j) -> bool {
        if (!ptx::mbar_wait(rest_full(j & 1), (j >> 1) & 1)) { give_up(3, j); return false; }
        ptx::tc_fence_after();
        issue_s(j, 0, kPieces - kValuePieces);
        ptx::tc_commit(rest_empty(j & 1));
        return true;
      };
      auto second_part = [&](int j) -> bool {
        if (!ptx::mbar_wait(own_full(j & 1), (j >> 1) & 1)) { give_up(4, j); return false; }
        ptx::tc_fence_after();
        issue_s(j, kPieces - kValuePieces, kPieces);
        ptx::tc_commit(s_full(j & 1));
        return true;
      };
      if (!ptx::mbar_wait(q_full, 0) || !ptx::mbar_wait(q_tmem, 0)) { give_up(5, 0); ok = false; }
      ptx::tc_fence_after();
      if (ok && n_tiles > 0) ok = first_part(0) && second_part(0);
      for (int j = 0; j < n_tiles && ok; ++j) {
        // S_{j+1} goes where P_{j-1} was: P_{j-1} V_{j-1} precedes it in the order of issue. Its second part follows as soon as the own half
        // of the tile is there, if that is before P_j is, so that the next softmax finds its scores; else P_j V_j goes first.
        if (j + 1 < n_tiles && !first_part(j + 1)) { ok = false; break; }
        const int s = j & 1;
        bool second = j + 1 >= n_tiles;
        for (int i = 0; i < 4096 && !ptx::mbar_test(p_full(s), (j >> 1) & 1); ++i)      // then the bounded wait below
          if (!second && ptx::mbar_test(own_full((j + 1) & 1), ((j + 1) >> 1) & 1)) {
            second = true;
            if (!(ok = second_part(j + 1))) break;
          }
        if (!ok) break;
        if (!ptx::mbar_wait(p_full(s), (j >> 1) & 1)) { give_up(6, j); ok = false; break; }
        ptx::tc_fence_after();
        const uint32_t at = base + kOffK + s * kKeyBytes;
#pragma unroll
        for (int k = 0; k < kKeys / 16; ++k)
          ptx::mma_tmem_a(tmem, tmem + kColS + s * kKeys + k * 8, value_desc(at + k * 2048), idesc_o, (j | k) ? 1u : 0u);
        ptx::tc_commit(own_empty(s));
        ptx::tc_commit(pv_done(s));
        if (!second && !second_part(j + 1)) { ok = false; break; }
      }
      if (!ok) {
        ptx::tc_commit(drain_bar);
        ptx::mbar_wait(drain_bar, 0, 200000000ull);
      }
    }
    __syncwarp();
  } else {
    // ------------------------------------------------------------------ softmax: thread (r, g) has 32 of a row's 64 keys
    const int g = (warp - 2) >> 2, quarter = warp & 3, r = quarter * 32 + lane;
    const uint32_t lanes = static_cast<uint32_t>(quarter * 32) << 16;
    const int tok = r / prm.heads, head = r - tok * prm.heads;
    const int qpos = pos0 + tok;
    {
      // the query's first four pieces: 128 columns of the row by each of its two threads
      const bool live = tok < n_tok;
      const uint4* src = reinterpret_cast<const uint4*>(prm.q_lat + static_cast<int64_t>(tok0 + (live ? tok : 0)) * prm.q_stride + head * 512 + g * 128);
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        uint32_t v[32];
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const uint4 q = live ? src[c * 8 + i] : make_uint4(0, 0, 0, 0);
          v[i * 4] = q.x; v[i * 4 + 1] = q.y; v[i * 4 + 2] = q.z; v[i * 4 + 3] = q.w;
        }
        ptx::tmem_st_32x32(tmem + kColQ + g * 64 + c * 32 + lanes, v);
      }
      ptx::tc_wait_st();
      ptx::tc_fence_before();
      __syncwarp();
      if (lane == 0) ptx::mbar_arrive(q_tmem);
    }
    float m_used = -INFINITY, l_part = 0.0f;
    bool ok = true;
    // as in attention_tc.cu: a warp that gives up keeps walking (the barriers below count on it) but touches nothing
    auto wait_all = [&](uint32_t b, uint32_t parity, int code, int j) -> bool {
      if (!ok || *fail != 0) return false;
      if (__all_sync(0xffffffffu, ptx::mbar_wait(b, parity))) return true;
      if (lane == 0) give_up(code, j);
      return false;
    };
    for (int j = 0; j < n_tiles; ++j) {
      const int a = j & 1, kv0 = j * kKeys + g * 32;
      const uint32_t s_at = tmem + kColS + a * kKeys + lanes;
      float s[32];
      ok = wait_all(s_full(a), (j >> 1) & 1, 7, j);
      if (ok) {
        ptx::tc_fence_after();
        uint32_t v[32];
        ptx::tmem_ld_32x32(s_at + g * 32, v);
        ptx::tc_wait_ld();
#pragma unroll
        for (int i = 0; i < 32; ++i) s[i] = __uint_as_float(v[i]);
      } else {
#pragma unroll
        for (int i = 0; i < 32; ++i) s[i] = 0.0f;
      }
      if (kv0 + 31 > pos0) {
#pragma unroll
        for (int i = 0; i < 32; ++i)
          if (kv0 + i > qpos) s[i] = -INFINITY;
      }
      float mx[4] = {s[0], s[1], s[2], s[3]};
#pragma unroll
      for (int i = 4; i < 32; ++i) mx[i & 3] = fmaxf(mx[i & 3], s[i]);
      const float m_own = fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3]));
      row_max[(a * 2 + g) * kRows + r] = m_own;
      ptx::tc_fence_before();
      ptx::named_barrier_sync(4 + quarter, 64);      // the two warps of these rows: maxima written, both halves of S_j read
      ptx::tc_fence_after();
      const float m_new = fmaxf(m_used, fmaxf(m_own, row_max[(a * 2 + (g ^ 1)) * kRows + r]));
      const bool rescale = __any_sync(0xffffffffu, m_new > m_used);      // both warps see the same numbers and decide alike
      float alpha = 1.0f;
      if (rescale) {
        alpha = m_used == -INFINITY ? 0.0f : ptx::ex2((m_used - m_new) * prm.scale_log2);
        l_part *= alpha;
        m_used = m_new;
      }
      const float neg_m = m_used == -INFINITY ? 0.0f : -m_used * prm.scale_log2;
      float sum[2] = {0.0f, 0.0f};
      uint32_t p[16];
#pragma unroll
      for (int i = 0; i < 16; ++i) {
        const float p0 = ptx::ex2(fmaf(s[2 * i], prm.scale_log2, neg_m)), p1 = ptx::ex2(fmaf(s[2 * i + 1], prm.scale_log2, neg_m));
        p[i] = ptx::pack_bf16x2(p0, p1);
        sum[0] += ptx::bf16_lo(p[i]);      // of what the product multiplies with: the rounding of a row's large weights cancels
        sum[1] += ptx::bf16_hi(p[i]);
      }
      l_part += sum[0] + sum[1];
      if (ok) {
        ptx::tmem_st_32x16(s_at + g * 16, p);
        if ((j + 1) * kKeys > ctx) {
          // rows past the context hold whatever their page held before: a zero weight times that must stay zero
          uint8_t* v0 = smem + kOffK + a * kKeyBytes;
          const int from = ctx - j * kKeys, n = (kKeys - from) * 8 * kValuePieces;
          for (int i = threadIdx.x - 64; i < n; i += 256) {
            const int row = from + i / (8 * kValuePieces), c = i % (8 * kValuePieces);
            *reinterpret_cast<uint4*>(v0 + (c >> 3) * kPieceBytes + row * 128 + (c & 7) * 16) = make_uint4(0, 0, 0, 0);
          }
          ptx::fence_proxy_async_smem();
        }
        if (rescale && j > 0 && (ok = wait_all(pv_done((j - 1) & 1), ((j - 1) >> 1) & 1, 8, j))) {      // behind the weights: P V of the tile before has had their time to finish
          ptx::tc_fence_after();
#pragma unroll 1
          for (int c = 0; c < 2; ++c) {
            uint32_t v[2][32];
            const uint32_t o_at = tmem + g * 128 + c * 64 + lanes;
#pragma unroll
            for (int k = 0; k < 2; ++k) ptx::tmem_ld_32x32(o_at + k * 32, v[k]);
            ptx::tc_wait_ld();
#pragma unroll
            for (int k = 0; k < 2; ++k) {
#pragma unroll
              for (int i = 0; i < 32; ++i) v[k][i] = __float_as_uint(__uint_as_float(v[k][i]) * alpha);
              ptx::tmem_st_32x32(o_at + k * 32, v[k]);
            }
          }
        }
        if (ok) {
          ptx::tc_wait_st();
          ptx::tc_fence_before();
          __syncwarp();
          if (lane == 0) ptx::mbar_arrive(p_full(a));
        }
      }
    }
    if (n_tiles > 0) ok = wait_all(pv_done((n_tiles - 1) & 1), ((n_tiles - 1) >> 1) & 1, 9, n_tiles);
    ptx::named_barrier_sync(4 + quarter, 64);      // the maxima of the last tile have been read
    row_max[g * kRows + r] = l_part;
    ptx::named_barrier_sync(4 + quarter, 64);
    if (ok && *fail == 0) {
      ptx::tc_fence_after();
      const float l = row_max[r] + row_max[kRows + r], inv = l > 0.0f ? 1.0f / l : 0.0f;
      __nv_bfloat16* dst = prm.out + (static_cast<int64_t>(tok0 + tok) * prm.heads + head) * 512 + half * 256 + g * 128;
#pragma unroll 1
      for (int c = 0; c < 4; ++c) {
        uint32_t v[32];
        ptx::tmem_ld_32x32(tmem + g * 128 + c * 32 + lanes, v);
        ptx::tc_wait_ld();
        if (tok < n_tok) {
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            uint4 pk;
            pk.x = ptx::pack_bf16x2(__uint_as_float(v[i * 8]) * inv, __uint_as_float(v[i * 8 + 1]) * inv);
            pk.y = ptx::pack_bf16x2(__uint_as_float(v[i * 8 + 2]) * inv, __uint_as_float(v[i * 8 + 3]) * inv);
            pk.z = ptx::pack_bf16x2(__uint_as_float(v[i * 8 + 4]) * inv, __uint_as_float(v[i * 8 + 5]) * inv);
            pk.w = ptx::pack_bf16x2(__uint_as_float(v[i * 8 + 6]) * inv, __uint_as_float(v[i * 8 + 7]) * inv);
            ptx::st_v4(dst + c * 32 + i * 8, pk);
          }
        }
      }
    }
  }
  ptx::tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    ptx::tc_fence_after();
    ptx::tmem_dealloc(tmem, 512);
  }
}

// Query rows [tokens, heads, columns] with `stride` elements between tokens: boxes of one 64-column piece of all heads of a row block.
bool query_map(CUtensorMap* out, const void* q, int64_t tokens, int heads, int cols, int64_t stride, int box_tokens) {
  auto enc = tensor_map_encoder();
  if (enc == nullptr || (reinterpret_cast<uintptr_t>(q) & 15) != 0 || stride % 8 != 0) return false;
  cuuint64_t dims[3] = {static_cast<cuuint64_t>(cols), static_cast<cuuint64_t>(heads), static_cast<cuuint64_t>(tokens)};
  cuuint64_t strides[2] = {static_cast<cuuint64_t>(cols) * 2, static_cast<cuuint64_t>(stride) * 2};
  cuuint32_t box[3] = {64, static_cast<cuuint32_t>(heads), static_cast<cuuint32_t>(box_tokens)}, estr[3] = {1, 1, 1};
  return enc(out, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void*>(q), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
             CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

}  // namespace
}  // namespace b2

using namespace b2;

// Prompt chunks of `batch` sequences: cu_q (absolute rows, batch + 1), ctx_lens and block_tables of these sequences; q_lat, q_rope and
// out hold all `total_rows` rows of the step. `heads` divides 128, pages are multiples of 64 tokens.
extern "C" int b2_mla_prefill_tc_bf16(const void* q_lat, const void* q_rope, const void* kv_cache, void* out, const int32_t* cu_q, const int32_t* ctx_lens,
                                      const int32_t* block_tables, int batch, int total_rows, int max_q_len, int max_blocks, int n_heads, int page_size,
                                      float scale, int64_t num_pages, int64_t q_lat_stride, int64_t q_rope_stride, Status* status, cudaStream_t stream) {
  if (batch <= 0 || total_rows <= 0 || max_q_len <= 0) return 0;
  if (n_heads <= 0 || n_heads > kRows || kRows % n_heads != 0 || page_size <= 0 || page_size % kKeys != 0 || batch > 65535 ||
      (reinterpret_cast<uintptr_t>(out) & 15) != 0 || num_pages * page_size > 0x7fffffff)
    return -kBadArgument;
  const int tokens = kRows / n_heads;
  CUtensorMap tq, tr, tk;
  if (!query_map(&tq, q_lat, total_rows, n_heads, 512, q_lat_stride, tokens) || !query_map(&tr, q_rope, total_rows, n_heads, 64, q_rope_stride, tokens) ||
      !make_tmap_2d(&tk, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, kv_cache, static_cast<uint64_t>(num_pages) * page_size, 576, 1152, kKeys, 64, CU_TENSOR_MAP_SWIZZLE_128B))
    return -kBadArgument;
  MlaTcParams prm{static_cast<const __nv_bfloat16*>(q_lat), static_cast<__nv_bfloat16*>(out), q_lat_stride, cu_q, ctx_lens, block_tables, max_blocks, n_heads,
                  tokens, page_size, num_pages, scale * ptx::kLog2e};
  static DeviceOnce attr_once;
  if (const int rc = attr_once.max_smem(mla_prefill_tc_kernel, kSmem)) return rc;
  launch_pdl(mla_prefill_tc_kernel, dim3(2 * ((max_q_len + tokens - 1) / tokens), batch), dim3(kThreads), kSmem, stream, tq, tr, tk, prm, status);
  return last_launch_rc();
}
