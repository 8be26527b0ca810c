// Causal GQA prefill attention on the 5th-generation tensor cores: S = Q K^T and O_j = P_j V_j are tcgen05.mma
// instructions with S and O_j in TMEM; Q, K and V tiles arrive by TMA; the online softmax runs in registers.
// Head dimension 128, KV pages of 128 tokens (one KV tile = one page of one KV head, a contiguous 32 KB block).
// The reference has no attention of any kind, and no tensor-core code (its newest gate is sm_90a,
// stdlib/src/sys/info.mojo:423-434).
//
// One CTA = 128 query rows of one query head, 320 threads:
//   warp 0      TMA producer: the Q tile once (two 128 x 64 boxes), then K and V of each KV tile into a 2-deep ring
//   warp 1      owns TMEM (512 columns: two S buffers, two O buffers); one lane issues the MMAs
//                 S_j   = Q K_j^T    A = Q  (K-major, 128-byte swizzle), B = K_j (K-major: head dim is contiguous)
//                 O_j   = P_j V_j    A = P_j (K-major, written by the softmax warps), B = V_j (MN-major: V rows are
//                                    KV tokens, so the N = head-dim index is the contiguous one)
//   warps 2-9   compute, two threads per query row (64 columns each): tcgen05.ld the half row of S_j, causal mask,
//               running max (halves exchanged through shared memory), exp2, row sum; write P_j as bf16 into shared
//               memory in the swizzled operand layout; then O = O * alpha_{j-1} + O_{j-1} for their 64 columns of
//               the accumulator (tcgen05.ld); at the end O / l as bf16
// S_{j+1} is issued before P_j V_j, so the softmax of tile j + 1 overlaps the second MMA of tile j, and the
// accumulation of O_j runs after the softmax of tile j + 1.
// Every mbarrier wait is bounded; a role that gives up records TIMEOUT, raises a CTA-wide flag and leaves its
// loop, the others follow at their next wait, and the CTA still frees TMEM and exits.
#include <cstdint>
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include "b2/api.h"
#include "b2/launch.h"
#include "b2/config.h"
#include "b2/f32x2.cuh"
#include "b2/gemm_tc.cuh"
#include "b2/ptx.cuh"
#include "b2/score_mods.cuh"
#include "b2/status.h"
#include "b2/tma.h"
#include "b2/vec.cuh"

namespace b2 {
namespace {

constexpr int kD = 128;            // head dimension
constexpr int kTile = 128;         // query rows per CTA = KV tokens per tile = page size
constexpr int kThreadsAttn = 320;
constexpr int kHalfBytes = kTile * 64 * 2;     // one 128 x 64 bf16 box: 16 KB
constexpr int kTileBytes = 2 * kHalfBytes;     // 128 x 128 bf16: 32 KB
constexpr int kStages = 2;
// shared memory: Q | P | K[2] | V[2] | barriers | alpha ring | l
constexpr int kOffQ = 0;
constexpr int kOffP = kOffQ + kTileBytes;
constexpr int kOffK = kOffP + kTileBytes;
constexpr int kOffV = kOffK + kStages * kTileBytes;
constexpr int kOffBar = kOffV + kStages * kTileBytes;      // 192 KB
constexpr int kNumBars = 1 + 4 * kStages + 2 + 2 + 2 + 2 + 1;  // q_full, k/v full+empty, s full/empty, p full/empty, o full/empty, drain
constexpr int kOffAlpha = kOffBar + 8 * kNumBars + 16;     // float [2][2][128]: partial row maxima
constexpr int kOffL = kOffAlpha + 4 * kTile * 4;           // float [2][128]
constexpr int kOffBias = kOffL + 2 * kTile * 4;            // float [2][256]: distance biases of a tile
constexpr int kOffFlags = kOffBias + 2 * 256 * 4;          // tmem holder, fail flag
constexpr int kSmemAttn = kOffFlags + 16 + 1024;           // + alignment slack

struct AttnTcParams {
  __nv_bfloat16* out;
  int64_t ld_out;
  const int* cu_q;
  const int* ctx_lens;
  const int* block_tables;
  int max_blocks, n_q, n_kv;
  int64_t num_pages;
  float scale_log2;   // softmax scale * log2(e)
  // descriptor of the MN-major V operand (bytes): stride between 64-column groups, stride between 8-row groups
  uint32_t v_lbo, v_sbo;
  // Optional work list: item i = (sequence, query tile) as two ints, for grids of (items, heads). `n_work` (device
  // memory) is the number of valid items, so that a captured launch with a fixed grid serves any batch; null means
  // every CTA of the grid has an item. Without a list the grid is (query tiles, heads, sequences).
  const int* work;
  const int* n_work;
  // Optional output gate, null: none. One factor sigmoid(gate[t * gate_stride + h]) for head h of row t, or with
  // `gate_elems` one per output element, sigmoid(gate[t * gate_stride + h * 128 + c]).
  const __nv_bfloat16* gate;
  int64_t gate_stride;
  int gate_elems;
  // Where the tile of (page, KV head) lies in the K and V matrices: row page * page_rows + head * head_rows, column
  // head * head_cols. Paged cache: {n_kv * 128, 128, 0}; rows of one token with its heads side by side: {128, 0, 128}.
  int page_rows, head_rows, head_cols;
  // Kernel of two heads to a block: items of the list (or of the grid q_tiles x sequences), and whether every block takes one head.
  int n_items, q_tiles, one_head;
  ScoreMods mods;
};

// Shared-memory descriptor with explicit leading / stride byte offsets, 128-byte swizzle.
__device__ __forceinline__ uint64_t smem_desc(uint32_t addr, uint32_t lbo_bytes, uint32_t sbo_bytes) {
  uint64_t d = 0;
  d |= static_cast<uint64_t>((addr & 0x3FFFF) >> 4);
  d |= static_cast<uint64_t>((lbo_bytes >> 4) & 0x3FFF) << 16;
  d |= static_cast<uint64_t>((sbo_bytes >> 4) & 0x3FFF) << 32;
  d |= static_cast<uint64_t>(1) << 46;
  d |= static_cast<uint64_t>(2) << 61;
  return d;
}

// MODS: AttnTcParams::mods. Tiles before the first position that the first row sees are never visited. A tile's distance bias
// depends on 255 distances only: they wait in shared memory, written while the tile before is worked on.
template <bool MODS>
__global__ void __launch_bounds__(kThreadsAttn, 1)
attn_prefill_tc_kernel(const __grid_constant__ CUtensorMap tmap_q, const __grid_constant__ CUtensorMap tmap_k,
                       const __grid_constant__ CUtensorMap tmap_v, AttnTcParams prm, Status* status) {
  ptx::grid_dep_sync();
  int seq = blockIdx.z, qt = blockIdx.x;
  const int head = blockIdx.y;
  if (prm.work != nullptr) {
    if (prm.n_work != nullptr && static_cast<int>(blockIdx.x) >= *prm.n_work) return;
    seq = prm.work[2 * blockIdx.x];
    qt = prm.work[2 * blockIdx.x + 1];
  }
  const int q_begin = prm.cu_q[seq], q_len = prm.cu_q[seq + 1] - q_begin;
  if (qt * kTile >= q_len) return;                       // uniform per CTA: before any barrier or allocation
  const int ctx = prm.ctx_lens[seq];
  const int pos0 = ctx - q_len + qt * kTile;              // absolute position of this tile's first query row
  const int rows = min(kTile, q_len - qt * kTile);
  const int first_tile = MODS ? prm.mods.first(pos0) / kTile : 0;
  const int n_tiles = min((pos0 + rows + kTile - 1) / kTile, (ctx + kTile - 1) / kTile) - first_tile;  // KV tiles with a visible token
  const int kvh = head / (prm.n_q / prm.n_kv);

  extern __shared__ uint8_t smem_raw[];
  const uint32_t base = (ptx::smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t* smem = smem_raw + (base - ptx::smem_u32(smem_raw));
  auto bar = [&](int i) { return base + kOffBar + 8u * i; };
  const uint32_t q_full = bar(0);
  auto k_full = [&](int s) { return bar(1 + s); };
  auto v_full = [&](int s) { return bar(1 + kStages + s); };
  auto k_empty = [&](int s) { return bar(1 + 2 * kStages + s); };
  auto v_empty = [&](int s) { return bar(1 + 3 * kStages + s); };
  auto s_full = [&](int a) { return bar(1 + 4 * kStages + a); };
  auto s_empty = [&](int a) { return bar(3 + 4 * kStages + a); };
  const uint32_t p_full = bar(5 + 4 * kStages), p_empty = bar(6 + 4 * kStages);
  auto o_full = [&](int a) { return bar(7 + 4 * kStages + a); };
  auto o_empty = [&](int a) { return bar(9 + 4 * kStages + a); };
  const uint32_t drain_bar = bar(11 + 4 * kStages);
  float* alpha_ring = reinterpret_cast<float*>(smem + kOffAlpha);
  float* l_final = reinterpret_cast<float*>(smem + kOffL);
  uint32_t* tmem_holder = reinterpret_cast<uint32_t*>(smem + kOffFlags);
  volatile uint32_t* fail = reinterpret_cast<volatile uint32_t*>(smem + kOffFlags + 4);

  const int warp = ptx::warp_id(), lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    ptx::prefetch_tensormap(&tmap_q);
    ptx::prefetch_tensormap(&tmap_k);
    ptx::prefetch_tensormap(&tmap_v);
    ptx::mbar_init(q_full, 1);
    for (int s = 0; s < kStages; ++s) {
      ptx::mbar_init(k_full(s), 1);
      ptx::mbar_init(v_full(s), 1);
      ptx::mbar_init(k_empty(s), 1);
      ptx::mbar_init(v_empty(s), 1);
    }
    for (int a = 0; a < 2; ++a) {
      ptx::mbar_init(s_full(a), 1);
      ptx::mbar_init(s_empty(a), 8);
      ptx::mbar_init(o_full(a), 1);
      ptx::mbar_init(o_empty(a), 8);
    }
    ptx::mbar_init(p_full, 8);
    ptx::mbar_init(p_empty, 1);
    ptx::mbar_init(drain_bar, 1);
    ptx::fence_mbar_init();
    *fail = 0;
  }
  if (warp == 1) {
    ptx::tmem_alloc(ptx::smem_u32(tmem_holder), 512);
    ptx::tmem_relinquish();
  }
  ptx::tc_fence_before();
  __syncthreads();
  ptx::tc_fence_after();
  const uint32_t tmem_base = *tmem_holder;
  auto give_up = [&](int site_a, int site_b) {
    status_record(status, kTimeout, kSiteAttn, site_a, site_b);
    *fail = 1;
  };

  if (warp == 0) {
    // ------------------------------------------------------------------ TMA producer
    if (ptx::elect_one()) {
      ptx::mbar_arrive_expect_tx(q_full, kTileBytes);
      ptx::tma_load_2d(base + kOffQ, &tmap_q, q_full, head * kD, q_begin + qt * kTile, ptx::kEvictFirst);
      ptx::tma_load_2d(base + kOffQ + kHalfBytes, &tmap_q, q_full, head * kD + 64, q_begin + qt * kTile, ptx::kEvictFirst);
      int issued_k = 0, issued_v = 0;
      bool ok = true;
      for (int j = 0; j < n_tiles && ok; ++j) {
        const int s = j % kStages;
        const uint32_t ph = static_cast<uint32_t>((j / kStages) & 1);
        int page = prm.block_tables[static_cast<int64_t>(seq) * prm.max_blocks + first_tile + j];
        if (page < 0 || page >= prm.num_pages) {
          status_record(status, kOutOfBounds, kSiteKvIndex, seq, page);
          page = 0;
        }
        const int row = page * prm.page_rows + kvh * prm.head_rows, col = kvh * prm.head_cols;
        if (!ptx::mbar_wait(k_empty(s), ph ^ 1u)) { give_up(1, j); ok = false; break; }
        ptx::mbar_arrive_expect_tx(k_full(s), kTileBytes);
        ptx::tma_load_2d(base + kOffK + s * kTileBytes, &tmap_k, k_full(s), col, row, ptx::kEvictLast);
        ptx::tma_load_2d(base + kOffK + s * kTileBytes + kHalfBytes, &tmap_k, k_full(s), col + 64, row, ptx::kEvictLast);
        ++issued_k;
        if (!ptx::mbar_wait(v_empty(s), ph ^ 1u)) { give_up(2, j); ok = false; break; }
        ptx::mbar_arrive_expect_tx(v_full(s), kTileBytes);
        ptx::tma_load_2d(base + kOffV + s * kTileBytes, &tmap_v, v_full(s), col, row, ptx::kEvictLast);
        ptx::tma_load_2d(base + kOffV + s * kTileBytes + kHalfBytes, &tmap_v, v_full(s), col + 64, row, ptx::kEvictLast);
        ++issued_v;
      }
      if (!ok) {
        // let the copies this thread started land before the CTA gives up its shared memory
        ptx::mbar_wait(q_full, 0, 200000000ull);
        for (int j = max(0, issued_k - kStages); j < issued_k; ++j) ptx::mbar_wait(k_full(j % kStages), (j / kStages) & 1, 200000000ull);
        for (int j = max(0, issued_v - kStages); j < issued_v; ++j) ptx::mbar_wait(v_full(j % kStages), (j / kStages) & 1, 200000000ull);
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    // ------------------------------------------------------------------ MMA issuer
    if (ptx::elect_one()) {
      constexpr uint32_t idesc_s = ptx::make_idesc(1, 1, 128, 128);                 // bf16 x bf16, both K-major
      constexpr uint32_t idesc_o = ptx::make_idesc(1, 1, 128, 128) | (1u << 16);    // B (= V) is MN-major
      bool ok = true;
      auto issue_s = [&](int j) -> bool {
        const int s = j % kStages, a = j & 1;
        if (!ptx::mbar_wait(k_full(s), (j / kStages) & 1)) { give_up(3, j); return false; }
        if (!ptx::mbar_wait(s_empty(a), ((j >> 1) & 1) ^ 1u)) { give_up(4, j); return false; }
        ptx::tc_fence_after();
        const uint32_t d = tmem_base + a * 128;
#pragma unroll
        for (int kb = 0; kb < 2; ++kb) {
          const uint64_t da = ptx::make_smem_desc_sw128(base + kOffQ + kb * kHalfBytes);
          const uint64_t db = ptx::make_smem_desc_sw128(base + kOffK + s * kTileBytes + kb * kHalfBytes);
#pragma unroll
          for (int k = 0; k < 4; ++k) ptx::tc_mma_f16(d, da + 2u * k, db + 2u * k, idesc_s, (kb | k) ? 1u : 0u);
        }
        ptx::tc_commit(k_empty(s));    // K_j can be overwritten once S_j has read it
        ptx::tc_commit(s_full(a));
        return true;
      };
      if (!ptx::mbar_wait(q_full, 0)) { give_up(5, 0); ok = false; }
      if (ok && n_tiles > 0) ok = issue_s(0);
      for (int j = 0; j < n_tiles && ok; ++j) {
        if (j + 1 < n_tiles && !issue_s(j + 1)) { ok = false; break; }
        const int s = j % kStages, a = j & 1;
        if (!ptx::mbar_wait(v_full(s), (j / kStages) & 1)) { give_up(6, j); ok = false; break; }
        if (!ptx::mbar_wait(p_full, j & 1)) { give_up(7, j); ok = false; break; }
        if (!ptx::mbar_wait(o_empty(a), ((j >> 1) & 1) ^ 1u)) { give_up(8, j); ok = false; break; }
        ptx::tc_fence_after();
        const uint32_t d = tmem_base + 256 + a * 128;
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          // A: 16 KV columns of P = 32 bytes inside the swizzled row (+2 per step, next 64-column block after four)
          const uint64_t da = ptx::make_smem_desc_sw128(base + kOffP + (k >> 2) * kHalfBytes) + 2u * (k & 3);
          // B: 16 KV rows of V = two 8-row groups of 1 KB each; the two 64-column halves of the head dim are v_lbo apart
          const uint64_t db = smem_desc(base + kOffV + s * kTileBytes + k * 2048, prm.v_lbo, prm.v_sbo);
          ptx::tc_mma_f16(d, da, db, idesc_o, k ? 1u : 0u);
        }
        ptx::tc_commit(v_empty(s));
        ptx::tc_commit(p_empty);
        ptx::tc_commit(o_full(a));
      }
      if (!ok) {
        ptx::tc_commit(drain_bar);
        ptx::mbar_wait(drain_bar, 0, 200000000ull);
      }
    }
    __syncwarp();
  } else {
    // ------------------------------------------------------------------ compute warps
    // Eight warps, two threads per query row: thread (r, g) owns columns [64 g, 64 g + 64) of the row's S tile and
    // the same columns of its O accumulator. Two warps per scheduler hide each other's dependency stalls, which one
    // warp per scheduler cannot. Per KV tile: softmax of S_j and the write of P_j, then (software pipelining) the
    // accumulation of O_{j-1}, whose MMA ran while this tile's softmax did.
    const int g = (warp - 2) >> 2;          // column half
    const int quarter = warp & 3;           // TMEM lane quarter this warp may access
    const int r = quarter * 32 + lane;
    const int qpos = pos0 + r;
    const uint32_t lane_bits = static_cast<uint32_t>(quarter * 32) << 16;
    float* pmax = alpha_ring;               // [2 tiles in flight][2 halves][128 rows]
    const float scale_log2 = MODS ? 1.0f : prm.scale_log2;      // MODS: the scores come scaled
    const bool sink = MODS && prm.mods.sink;                    // a score of zero that has been seen already
    float m_run = sink ? 0.0f : -INFINITY, l_part = sink && g == 0 ? 1.0f : 0.0f, alpha_prev = 1.0f;
    const int first_seen = MODS ? prm.mods.first(qpos) : 0, first_last = MODS ? prm.mods.first(pos0 + kTile - 1) : 0;
    const bool biased = MODS && prm.mods.bias != nullptr;
    float* bias_sm = reinterpret_cast<float*>(smem + kOffBias);
    float2 head_bias = make_float2(0.0f, 0.0f);
    // entry i of tile j: distance (row 0's to the tile's last column) + i; a row and column meet at r + 127 - column
    const auto fill_bias = [&](int j) {
      const int i = static_cast<int>(threadIdx.x) - 64;
      bias_sm[(j & 1) * 256 + i] = ScoreMods::distance(head_bias, max(0, pos0 - (first_tile + j) * kTile - (kTile - 1) + i));
    };
    if (biased) {
      head_bias = prm.mods.head_bias(head);
      fill_bias(0);
      ptx::named_barrier_sync(5, 256);
    }
    float o[64];
#pragma unroll
    for (int i = 0; i < 64; ++i) o[i] = 0.0f;
    // A warp that gives up keeps walking the loop (every compute warp must reach the named barrier of every tile)
    // but no longer waits, reads TMEM or arrives anywhere; the other roles then run into their own limits.
    bool ok = true;
    auto wait_all = [&](uint32_t bar_addr, uint32_t parity, int code, int j) -> bool {
      if (!ok || *fail != 0) return false;
      if (__all_sync(0xffffffffu, ptx::mbar_wait(bar_addr, parity))) return true;
      if (lane == 0) give_up(code, j);
      return false;
    };
    auto accumulate = [&](int j, float alpha) {
      const int a = j & 1;
      ok = wait_all(o_full(a), (j >> 1) & 1, 11, j);
      if (!ok) return;
      ptx::tc_fence_after();
      const uint32_t taddr = tmem_base + 256 + a * 128 + g * 64 + lane_bits;
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        uint32_t v[32];
        ptx::tmem_ld_32x32(taddr + c * 32, v);
        ptx::tc_wait_ld();
#pragma unroll
        for (int i = 0; i < 32; ++i) o[c * 32 + i] = fmaf(o[c * 32 + i], alpha, __uint_as_float(v[i]));
      }
      ptx::tc_fence_before();
      __syncwarp();
      if (lane == 0) ptx::mbar_arrive(o_empty(a));
    };
    for (int j = 0; j < n_tiles; ++j) {
      const int a = j & 1;
      float s[64];
      ok = wait_all(s_full(a), (j >> 1) & 1, 9, j);
      if (ok) {
        ptx::tc_fence_after();
        const uint32_t taddr = tmem_base + a * 128 + g * 64 + lane_bits;
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          uint32_t v[32];
          ptx::tmem_ld_32x32(taddr + c * 32, v);
          ptx::tc_wait_ld();
#pragma unroll
          for (int i = 0; i < 32; ++i) s[c * 32 + i] = __uint_as_float(v[i]);
        }
        ptx::tc_fence_before();
        __syncwarp();
        if (lane == 0) ptx::mbar_arrive(s_empty(a));     // S buffer free for tile j + 2
      } else {
#pragma unroll
        for (int c = 0; c < 64; ++c) s[c] = 0.0f;
      }
      const int kv0 = (first_tile + j) * kTile + g * 64;
      if constexpr (MODS) {
        prm.mods.scores<64>(s, prm.scale_log2);
        if (biased) {
          const float* b = bias_sm + (j & 1) * 256 + r + kTile - 1 - g * 64;
#pragma unroll
          for (int c = 0; c < 64; ++c) s[c] -= b[-c];
          if (j + 1 < n_tiles) fill_bias(j + 1);
        }
        if (kv0 < first_last) {                            // some row of this tile is past some of these columns
#pragma unroll
          for (int c = 0; c < 64; ++c)
            if (kv0 + c < first_seen) s[c] = -INFINITY;
        }
      }
      if (kv0 + 63 > pos0) {                             // some row of this tile masks some of these columns
#pragma unroll
        for (int c = 0; c < 64; ++c)
          if (kv0 + c > qpos) s[c] = -INFINITY;
      }
      // row maximum of the raw scores: eight independent chains, then the partner's half through shared memory
      float mx[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) mx[i] = s[i];
#pragma unroll
      for (int c = 8; c < 64; ++c) mx[c & 7] = fmaxf(mx[c & 7], s[c]);
      const float mloc = fmaxf(fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3])), fmaxf(fmaxf(mx[4], mx[5]), fmaxf(mx[6], mx[7])));
      pmax[(a * 2 + g) * kTile + r] = mloc;
      ptx::named_barrier_sync(5, 256);
      const float m_new = fmaxf(m_run, fmaxf(mloc, pmax[(a * 2 + (g ^ 1)) * kTile + r]));
      const float m_use = m_new == -INFINITY ? 0.0f : m_new;   // a row with nothing visible yet
      const float alpha = ptx::ex2((m_run - m_use) * scale_log2);
      const float neg_m = -m_use * scale_log2;
      m_run = m_new;
      if (j > 0) ok = wait_all(p_empty, (j - 1) & 1, 10, j);
      if (ok) {
        float sum[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll
        for (int ch = 0; ch < 8; ++ch) {
          float p[8];
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            p[i] = ptx::ex2(fmaf(s[ch * 8 + i], scale_log2, neg_m));
            sum[i & 3] += p[i];
          }
          uint4 pk;
          pk.x = ptx::pack_bf16x2(p[0], p[1]);
          pk.y = ptx::pack_bf16x2(p[2], p[3]);
          pk.z = ptx::pack_bf16x2(p[4], p[5]);
          pk.w = ptx::pack_bf16x2(p[6], p[7]);
          *reinterpret_cast<uint4*>(smem + kOffP + g * kHalfBytes + gemm::sw128_offset(r, ch)) = pk;
        }
        l_part = l_part * alpha + ((sum[0] + sum[1]) + (sum[2] + sum[3]));
        ptx::fence_proxy_async_smem();   // generic-proxy writes of P -> visible to the tensor core's async proxy
        __syncwarp();
        if (lane == 0) ptx::mbar_arrive(p_full);
      }
      // O_{j-1} = P_{j-1} V_{j-1} has had this tile's softmax to finish in
      if (j > 0) accumulate(j - 1, alpha_prev);
      alpha_prev = alpha;
    }
    if (n_tiles > 0) accumulate(n_tiles - 1, alpha_prev);
    l_final[g * kTile + r] = l_part;
    ptx::named_barrier_sync(5, 256);
    if (ok && *fail == 0 && r < rows) {
      const float l = l_final[r] + l_final[kTile + r];
      float inv = l > 0.0f ? 1.0f / l : 0.0f;
      if constexpr (MODS) inv *= prm.mods.out_scale;
      if (prm.gate != nullptr && prm.gate_elems) {
        const __nv_bfloat16* z = prm.gate + static_cast<int64_t>(q_begin + qt * kTile + r) * prm.gate_stride + head * kD + g * 64;
#pragma unroll
        for (int c = 0; c < 8; ++c) {
          float f[8];
          bf16x8_to_f32(ptx::ld_v4(z + c * 8), f);
#pragma unroll
          for (int i = 0; i < 8; ++i) o[c * 8 + i] *= ptx::rcp(1.0f + ptx::ex2(-f[i] * ptx::kLog2e));
        }
      } else if (prm.gate != nullptr) {
        const float z = __bfloat162float(prm.gate[static_cast<int64_t>(q_begin + qt * kTile + r) * prm.gate_stride + head]);
        inv /= 1.0f + ptx::ex2(-z * ptx::kLog2e);
      }
      __nv_bfloat16* dst = prm.out + static_cast<int64_t>(q_begin + qt * kTile + r) * prm.ld_out + head * kD + g * 64;
#pragma unroll
      for (int c = 0; c < 8; ++c) {
        uint4 pk;
        pk.x = ptx::pack_bf16x2(o[c * 8 + 0] * inv, o[c * 8 + 1] * inv);
        pk.y = ptx::pack_bf16x2(o[c * 8 + 2] * inv, o[c * 8 + 3] * inv);
        pk.z = ptx::pack_bf16x2(o[c * 8 + 4] * inv, o[c * 8 + 5] * inv);
        pk.w = ptx::pack_bf16x2(o[c * 8 + 6] * inv, o[c * 8 + 7] * inv);
        ptx::st_v4(dst + c * 8, pk);
      }
    }
  }
  ptx::tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    ptx::tc_fence_after();
    ptx::tmem_dealloc(tmem_base, 512);
  }
}

// ------------------------------------------------------------------------------------------------------------
// Two heads of one KV head to a CTA
// ------------------------------------------------------------------------------------------------------------
// Where scores are only masked, not changed, and with an even number of query heads per KV head, a CTA takes the same 128 rows of two heads:
// every K and V tile is fetched once for both, and while one head's softmax runs the tensor cores work for the other. That is what
// the kernel above lacks: its one S tile at a time leaves the tensor pipe idle for most of the softmax (669 TFLOP/s).
//
//   TMEM   head t: S / P of even blocks at 128 t, of odd blocks at 128 t + 64, O at 256 + 128 t
//   shared memory   Q_0, Q_1 (64 KB), five 32 KB places for K and V tiles in the order K_0 V_0 K_1 V_1 ...
//
// Keys go in blocks of 64, so that a head has two places for scores: those of block i + 1 are there when the softmax of block i ends.
// Warp 0 loads; warps 1 and 2 each issue one head's products, S of i + 2 behind P_i V_i, and one head's wait does not hold up the other's;
// warps 3-6 and 7-10 do one head each, a thread per row. P is written over S (a thread's own lane: no one else reads it) and read from
// TMEM by the second product. O is accumulated in TMEM and rescaled where a row's maximum has grown, so that the largest weight is
// always 1, which bf16 holds exactly: letting the weights grow to 2^8 first took 656 us for the case below where this took 700, and its
// error against 64 bits was 0.00235, this one's 0.0023 like that of the kernel above. The rescaling comes behind the weights, when the
// product of the block before, which it has to wait for, has had their time to finish (in front of them: 739 us against 700).
//
// A block may also take one head, whose keys its two groups of softmax warps share (CUT): each takes one half of every tile, and maxima, sums and O are brought
// together at the end. That is half of the time, for launches and last waves that have too few units of two heads.
//
// Two sequences of 1000 - 2048 rows behind up to 14000, 32 heads on 8 key heads (us): the kernel above 820 a call, this 615 (0.90 PFLOP/s). The other
// figures here are of a graph that replays the launch back to back, which takes 529. The
// tensor pipe needs some 1250 cycles for a pair of blocks (S of 64 columns reads its operands at the rate of shared memory), the
// special-function unit 1024 for its exponentials: the barrier, TMEM and exponential instructions of a scheduler's two softmax
// warps share one queue. Two threads per row, exponentials on the FMA pipe and scores requested a block ahead were no faster.
constexpr int kThreadsTwo = 96 + 256;
constexpr int kBlock = 64;      // keys to a softmax step
constexpr int kPlaces = 5;
constexpr int kOffRing2 = 2 * kTileBytes;
constexpr int kOffBar2 = kOffRing2 + kPlaces * kTileBytes;
constexpr int kNumBars2 = 1 + 2 * kPlaces + 4 + 4 + 4 + 2;      // q_full, ring full + empty, s_full, p_full, o_done, drain
constexpr int kOffFlags2 = kOffBar2 + 8 * kNumBars2;
constexpr int kSmemPair = kOffFlags2 + 16;
static_assert(kSmemPair <= kMaxSmemPerCta, "shared memory");

__device__ __forceinline__ float max3(float a, float b, float c) {
  float r;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
  return r;
}
__device__ __forceinline__ uint64_t add2(uint64_t a, uint64_t b) {
  uint64_t d;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}

// Units of two heads that the last wave shares out as blocks of one head, cut in two, where that fills it no further than once: 368 units leave
// 72 to a third wave, 144 blocks of half the time (two sequences of 1000 - 2048 rows behind up to 14000, 32 heads: 680 -> 575 us; 16 heads:
// 395 -> 256 us, where 184 units took two waves).
__host__ __device__ __forceinline__ int last_wave_units(int units) {
  const int rest = units % kNumSMs;
  return 2 * rest <= kNumSMs ? rest : 0;
}

// What a block works on: `rows` query rows from row qt * 128 of a sequence on, which is at position pos0, and n_blocks blocks of keys from
// tile first_tile on; heads head0 and head0 + 1, or (`one`) head0 alone.
struct TwoUnit {
  int one, seq, qt, q_begin, pos0, rows, first_tile, n_blocks, head0;
};

// RANGE: rows do not see all that came before (a window, chunks): tiles below the first row's range are left out, the edge is masked.
// CUT: one head, whose keys the two groups of softmax warps share.
template <bool RANGE, bool CUT>
__device__ __forceinline__ void attn_prefill_two(const CUtensorMap& tmap_q, const CUtensorMap& tmap_k, const CUtensorMap& tmap_v, const AttnTcParams& prm,
                                                 const TwoUnit& u, Status* status) {
  const int one = u.one, seq = u.seq, qt = u.qt, q_begin = u.q_begin, pos0 = u.pos0, rows = u.rows, first_tile = u.first_tile, n_blocks = u.n_blocks;
  const int n_tiles = (n_blocks + 1) / 2, head0 = u.head0, kvh = head0 / (prm.n_q / prm.n_kv);
  extern __shared__ __align__(1024) uint8_t smem_two[];
  const uint32_t base = ptx::smem_u32(smem_two);
  auto bar = [&](int i) { return base + kOffBar2 + 8u * i; };
  const uint32_t q_full = bar(0);
  auto drain = [&](int t) { return bar(kNumBars2 - 2 + t); };
  auto full = [&](int s) { return bar(1 + s); };
  auto empty = [&](int s) { return bar(1 + kPlaces + s); };
  // a head's two places for S: blocks take them in turn
  auto s_full = [&](int t, int i) { return bar(1 + 2 * kPlaces + t * 2 + (i & 1)); };
  auto p_full = [&](int t, int i) { return bar(5 + 2 * kPlaces + t * 2 + (i & 1)); };
  auto o_done = [&](int t, int i) { return bar(9 + 2 * kPlaces + t * 2 + (i & 1)); };
  uint32_t* tmem_holder = reinterpret_cast<uint32_t*>(smem_two + kOffFlags2);
  volatile uint32_t* fail = reinterpret_cast<volatile uint32_t*>(smem_two + kOffFlags2 + 4);

  const int warp = ptx::warp_id(), lane = threadIdx.x & 31;      // as threadIdx.x >> 5: 575 us for the case above
  if (threadIdx.x == 0) {
    ptx::prefetch_tensormap(&tmap_q);
    ptx::prefetch_tensormap(&tmap_k);
    ptx::prefetch_tensormap(&tmap_v);
    ptx::mbar_init(q_full, 1);
    for (int s = 0; s < kPlaces; ++s) {
      ptx::mbar_init(full(s), 1);
      ptx::mbar_init(empty(s), 2);      // both heads have read the place
    }
    for (int t = 0; t < 2; ++t) {
      for (int i = 0; i < 2; ++i) {
        ptx::mbar_init(s_full(t, i), 1);
        ptx::mbar_init(p_full(t, i), 4);
        ptx::mbar_init(o_done(t, i), 1);
      }
      ptx::mbar_init(drain(t), 1);
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
  const bool aligned = *fail == 0;
  auto give_up = [&](int a, int b) {
    status_record(status, kTimeout, kSiteAttn, a, b);
    *fail = 1;
  };
  // Block i of group t: the number of its K tile below (V follows), which half of the tile it is, and how many there are. CUT: t = 0 takes
  // the first halves of the tiles and t = 1 the second, each with sums of its own.
  auto k_tile = [](int i) { return CUT ? 2 * i : i & ~1; };
  auto half_of = [](int t, int i) { return CUT ? t : i & 1; };
  auto blocks_of = [&](int t) { return CUT ? (u.n_blocks + 1 - t) / 2 : u.n_blocks; };
  const bool idle = !CUT && u.one;      // group 1 is
  // tile number i of the sequence K_0 V_0 K_1 V_1 ...: its place and its turn there
  auto place = [](int i) { return i % kPlaces; };
  auto turn = [](int i) { return static_cast<uint32_t>((i / kPlaces) & 1); };

  if (!aligned) {
    if (threadIdx.x == 0) status_record(status, kBadArgument, kSiteAttn, 20, 0);
  } else if (warp == 0) {
    if (ptx::elect_one()) {
      ptx::mbar_arrive_expect_tx(q_full, (2 - one) * kTileBytes);
      for (int t = 0; t < 2 - one; ++t)
        for (int h = 0; h < 2; ++h)
          ptx::tma_load_2d(base + t * kTileBytes + h * kHalfBytes, &tmap_q, q_full, (head0 + t) * kD + h * 64, q_begin + qt * kTile, ptx::kEvictFirst);
      int issued = 0;
      bool ok = true;
      for (int j = 0; j < n_tiles && ok; ++j) {
        int page = prm.block_tables[static_cast<int64_t>(seq) * prm.max_blocks + first_tile + j];
        if (page < 0 || page >= prm.num_pages) {
          status_record(status, kOutOfBounds, kSiteKvIndex, seq, page);
          page = 0;
        }
        const int row = page * prm.page_rows + kvh * prm.head_rows, col = kvh * prm.head_cols;
        for (int v = 0; v < 2; ++v) {
          const int i = 2 * j + v, s = place(i);
          if (!ptx::mbar_wait(empty(s), turn(i) ^ 1u)) { give_up(1, i); ok = false; break; }
          ptx::mbar_arrive_expect_tx(full(s), kTileBytes);
          const uint32_t at = base + kOffRing2 + s * kTileBytes;
          ptx::tma_load_2d(at, v ? &tmap_v : &tmap_k, full(s), col, row, ptx::kEvictLast);
          ptx::tma_load_2d(at + kHalfBytes, v ? &tmap_v : &tmap_k, full(s), col + 64, row, ptx::kEvictLast);
          ++issued;
        }
      }
      if (!ok) {
        // let the copies this thread started land before the CTA gives up its shared memory
        ptx::mbar_wait(q_full, 0, 200000000ull);
        for (int i = max(0, issued - kPlaces); i < issued; ++i) ptx::mbar_wait(full(place(i)), turn(i), 200000000ull);
      }
    }
    __syncwarp();
  } else if (warp <= 2) {
    if (ptx::elect_one() && !(idle && warp == 2)) {
      const int t = warp - 1, n = blocks_of(t);
      const uint32_t q_at = base + (one ? 0 : t * kTileBytes);
      constexpr uint32_t idesc_s = ptx::make_idesc(1, 1, 128, kBlock);              // both K-major
      constexpr uint32_t idesc_o = ptx::make_idesc(1, 1, 128, 128) | (1u << 16);    // B (= V) is MN-major
      bool ok = true;
      auto wait_tile = [&](int i) -> bool {
        if (ptx::mbar_wait(full(place(i)), turn(i))) return true;
        give_up(2, i);
        return false;
      };
      auto issue_s = [&](int i) {      // its K tile has arrived
        const uint32_t k_at = base + kOffRing2 + place(k_tile(i)) * kTileBytes + half_of(t, i) * (kBlock * 128);
#pragma unroll
        for (int kb = 0; kb < 2; ++kb) {
          const uint64_t da = ptx::make_smem_desc_sw128(q_at + kb * kHalfBytes), db = ptx::make_smem_desc_sw128(k_at + kb * kHalfBytes);
#pragma unroll
          for (int k = 0; k < 4; ++k) ptx::tc_mma_f16(tmem + t * 128 + (i & 1) * kBlock, da + 2u * k, db + 2u * k, idesc_s, (kb | k) ? 1u : 0u);
        }
        ptx::tc_commit(s_full(t, i));
      };
      if (!ptx::mbar_wait(q_full, 0)) { give_up(3, 0); ok = false; }
      // S of block i; its K tile is done with behind the last block in it
      auto next_s = [&](int i) -> bool {
        const int tile = k_tile(i);
        if ((CUT || (i & 1) == 0) && !wait_tile(tile)) return false;
        ptx::tc_fence_after();
        issue_s(i);
        if (CUT || (i & 1)) ptx::tc_commit(empty(place(tile)));
        return true;
      };
      for (int i = 0; i < min(n, 2) && ok; ++i) ok = next_s(i);
      for (int i = 0; i < n && ok; ++i) {
        const int v_tile = k_tile(i) + 1;
        const uint32_t v_at = base + kOffRing2 + place(v_tile) * kTileBytes + half_of(t, i) * (kBlock * 128);
        if ((CUT || (i & 1) == 0) && !(ok = wait_tile(v_tile))) break;
        if (!ptx::mbar_wait(p_full(t, i), (i >> 1) & 1)) { give_up(4, i); ok = false; break; }
        ptx::tc_fence_after();
#pragma unroll
        for (int k = 0; k < kBlock / 16; ++k)
          ptx::mma_tmem_a(tmem + 256 + t * 128, tmem + t * 128 + (i & 1) * kBlock + k * 8, smem_desc(v_at + k * 2048, prm.v_lbo, prm.v_sbo), idesc_o,
                     (i | k) ? 1u : 0u);
        ptx::tc_commit(o_done(t, i));
        if (CUT || (i & 1)) ptx::tc_commit(empty(place(v_tile)));
        // goes where P of this block is, which the product before it in the order of issue has read
        if (i + 2 < n) ok = next_s(i + 2);
      }
      if (!ok) {
        ptx::tc_commit(drain(t));
        ptx::mbar_wait(drain(t), 0, 200000000ull);
      }
    }
    __syncwarp();
  } else if (!idle || warp < 7) {
    const int t = (warp - 3) >> 2, quarter = warp & 3, r = quarter * 32 + lane, n = blocks_of(t);
    const uint32_t lanes = static_cast<uint32_t>(quarter * 32) << 16;
    const uint32_t s_at = tmem + t * 128 + lanes, o_at = tmem + 256 + t * 128 + lanes;
    const int qpos = pos0 + r, low = RANGE ? prm.mods.first(qpos) : 0, low_last = RANGE ? prm.mods.first(pos0 + kTile - 1) : 0;
    const float scale = prm.scale_log2;
    float m_used = -INFINITY, l = 0.0f;
    bool ok = true;
    // no barrier joins the warps of a head: one that gives up leaves, the other roles run into their limits
    auto wait_all = [&](uint32_t b, uint32_t parity, int code, int j) -> bool {
      if (*fail != 0) return false;
      if (__all_sync(0xffffffffu, ptx::mbar_wait(b, parity))) return true;
      if (lane == 0) give_up(code, j);
      return false;
    };
    for (int i = 0; i < n; ++i) {
      if (!(ok = wait_all(s_full(t, i), (i >> 1) & 1, 5, i))) break;
      ptx::tc_fence_after();
      const uint32_t at = s_at + (i & 1) * kBlock;
      uint32_t x[kBlock];
      ptx::tmem_ld_32x32(at, *reinterpret_cast<uint32_t(*)[32]>(x));
      ptx::tmem_ld_32x32(at + 32, *reinterpret_cast<uint32_t(*)[32]>(x + 32));
      ptx::tc_wait_ld();
      const int kv0 = first_tile * kTile + (CUT ? 2 * i + t : i) * kBlock;
      if (kv0 + kBlock - 1 > pos0 || (RANGE && kv0 < low_last)) {      // some row masks some of these columns
#pragma unroll
        for (int c = 0; c < kBlock; ++c)
          if (kv0 + c > qpos || (RANGE && kv0 + c < low)) x[c] = 0xff800000u;
      }
      float mx[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
      for (int c = 0; c < kBlock; c += 2) mx[(c >> 1) & 3] = max3(mx[(c >> 1) & 3], __uint_as_float(x[c]), __uint_as_float(x[c + 1]));
      const float m_new = fmaxf(m_used, fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3])));
      const bool rescale = __any_sync(0xffffffffu, m_new > m_used);
      float alpha = 1.0f;
      if (rescale) {
        alpha = m_used == -INFINITY ? 0.0f : ptx::ex2((m_used - m_new) * scale);
        l *= alpha;
        m_used = m_new;
      }
      const float neg_m = m_used == -INFINITY ? 0.0f : -m_used * scale;
      const uint64_t scale2 = pack2(scale, scale), neg2 = pack2(neg_m, neg_m);
      uint64_t sum[2] = {0, 0};
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        uint32_t p[16];
#pragma unroll
        for (int k = 0; k < 16; ++k) {
          const float2 e = unpack2(fma2(pack2(__uint_as_float(x[c * 32 + 2 * k]), __uint_as_float(x[c * 32 + 2 * k + 1])), scale2, neg2));
          p[k] = ptx::pack_bf16x2(ptx::ex2(e.x), ptx::ex2(e.y));
          sum[k & 1] = add2(sum[k & 1], pack2(ptx::bf16_lo(p[k]), ptx::bf16_hi(p[k])));      // as the product uses them: the rounding of large weights cancels
        }
        ptx::tmem_st_32x16(at + c * 16, p);
      }
      l += half_sum(sum[0]) + half_sum(sum[1]);
      if (rescale && i > 0) {      // behind the weights: P V of the block before has had their time to finish
        if (!(ok = wait_all(o_done(t, i - 1), ((i - 1) >> 1) & 1, 6, i))) break;
        ptx::tc_fence_after();
#pragma unroll 1
        for (int c = 0; c < 2; ++c) {
          uint32_t v[2][32];
#pragma unroll
          for (int k = 0; k < 2; ++k) ptx::tmem_ld_32x32(o_at + c * 64 + k * 32, v[k]);
          ptx::tc_wait_ld();
#pragma unroll
          for (int k = 0; k < 2; ++k) {
#pragma unroll
            for (int e = 0; e < 32; ++e) v[k][e] = __float_as_uint(__uint_as_float(v[k][e]) * alpha);
            ptx::tmem_st_32x32(o_at + c * 64 + k * 32, v[k]);
          }
        }
      }
      ptx::tc_wait_st();
      ptx::tc_fence_before();
      __syncwarp();
      if (lane == 0) ptx::mbar_arrive(p_full(t, i));
    }
    if (ok && n > 0) ok = wait_all(o_done(t, n - 1), ((n - 1) >> 1) & 1, 7, n);
    // One head cut in two: each group hands the other half of its columns over (through the ring, which nothing reads any more once both have come
    // here), and both bring the two sums to the larger maximum. All eight warps meet, whether they gave up or not.
    float* other = reinterpret_cast<float*>(smem_two + kOffRing2);      // [receiver][16 x float4][row]
    float* other_ml = other + 2 * 64 * kTile;                           // [sender][maximum, sum][row]
    float own_part = 1.0f, other_part = 0.0f;
    if constexpr (CUT) {
      ptx::tc_fence_after();
      ok = ptx::named_barrier_and(1, 256, ok);
      if (ok) {
        other_ml[(t * 2 + 0) * kTile + r] = m_used;
        other_ml[(t * 2 + 1) * kTile + r] = l;
        uint32_t v[64];      // both groups have blocks
        ptx::tmem_ld_32x32(o_at + (1 - t) * 64, *reinterpret_cast<uint32_t(*)[32]>(v));
        ptx::tmem_ld_32x32(o_at + (1 - t) * 64 + 32, *reinterpret_cast<uint32_t(*)[32]>(v + 32));
        ptx::tc_wait_ld();
#pragma unroll
        for (int g = 0; g < 16; ++g)
          *reinterpret_cast<uint4*>(other + (1 - t) * 64 * kTile + (g * kTile + r) * 4) = make_uint4(v[4 * g], v[4 * g + 1], v[4 * g + 2], v[4 * g + 3]);
      }
      ok = ptx::named_barrier_and(1, 256, ok);
      if (ok) {
        const float m_other = other_ml[((1 - t) * 2 + 0) * kTile + r], l_other = other_ml[((1 - t) * 2 + 1) * kTile + r], m = fmaxf(m_used, m_other);
        own_part = m_used == -INFINITY ? 0.0f : ptx::ex2((m_used - m) * scale);
        other_part = m_other == -INFINITY ? 0.0f : ptx::ex2((m_other - m) * scale);
        l = l * own_part + l_other * other_part;
      }
    }
    if (ok) {
      ptx::tc_fence_after();
      const int head = head0 + (one ? 0 : t);
      const int64_t row = q_begin + qt * kTile + r;
      float inv = l > 0.0f ? 1.0f / l : 0.0f;
      const bool live = r < rows;
      if (live && prm.gate != nullptr && !prm.gate_elems) inv /= 1.0f + ptx::ex2(-__bfloat162float(prm.gate[row * prm.gate_stride + head]) * ptx::kLog2e);
      __nv_bfloat16* dst = prm.out + row * prm.ld_out + head * kD;
#pragma unroll 1
      for (int c = CUT ? 2 * t : 0; c < (CUT ? 2 * t + 2 : 4); ++c) {
        uint32_t v[32];
        if (n > 0) {
          ptx::tmem_ld_32x32(o_at + c * 32, v);
          ptx::tc_wait_ld();
        } else {
#pragma unroll
          for (int i = 0; i < 32; ++i) v[i] = 0;
        }
        if constexpr (CUT) {
#pragma unroll
          for (int g = 0; g < 8; ++g) {
            const float4 w = *reinterpret_cast<const float4*>(other + (t * 64 * kTile) + (((c & 1) * 8 + g) * kTile + r) * 4);
            v[4 * g + 0] = __float_as_uint(fmaf(w.x, other_part, __uint_as_float(v[4 * g + 0]) * own_part));
            v[4 * g + 1] = __float_as_uint(fmaf(w.y, other_part, __uint_as_float(v[4 * g + 1]) * own_part));
            v[4 * g + 2] = __float_as_uint(fmaf(w.z, other_part, __uint_as_float(v[4 * g + 2]) * own_part));
            v[4 * g + 3] = __float_as_uint(fmaf(w.w, other_part, __uint_as_float(v[4 * g + 3]) * own_part));
          }
        }
        if (live) {
#pragma unroll
          for (int g = 0; g < 4; ++g) {
            float o[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) o[i] = __uint_as_float(v[g * 8 + i]) * inv;
            if (prm.gate != nullptr && prm.gate_elems) {
              float f[8];
              bf16x8_to_f32(ptx::ld_v4(prm.gate + row * prm.gate_stride + head * kD + c * 32 + g * 8), f);
#pragma unroll
              for (int i = 0; i < 8; ++i) o[i] *= ptx::rcp(1.0f + ptx::ex2(-f[i] * ptx::kLog2e));
            }
            ptx::st_v4(dst + c * 32 + g * 8, f32_to_bf16x8(o));
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

template <bool RANGE>
__global__ void __launch_bounds__(kThreadsTwo, 1)
attn_prefill_two_kernel(const __grid_constant__ CUtensorMap tmap_q, const __grid_constant__ CUtensorMap tmap_k, const __grid_constant__ CUtensorMap tmap_v,
                        const __grid_constant__ AttnTcParams prm, Status* status) {
  ptx::grid_dep_sync();
  const int pairs = prm.n_q / 2, units = (prm.n_work != nullptr ? min(*prm.n_work, prm.n_items) : prm.n_items) * pairs;
  const int alone = prm.one_head ? units : last_wave_units(units), unit0 = units - alone;
  int unit = blockIdx.x, one = 0;      // `one`: this block has one head
  if (unit >= unit0) {
    one = 1;
    unit = unit0 + ((static_cast<int>(blockIdx.x) - unit0) >> 1);
    if (unit >= units) return;
  }
  // Item by item, longest first, so that the last blocks to start are short ones. Where all start at once, head by head: blocks side by side then
  // share keys (eight tiles behind 14000, 32 heads: 232 us, 237 the other way).
  const int n_items = units / pairs, by_head = units <= kNumSMs && !prm.one_head;
  const int item = by_head ? unit % n_items : unit / pairs, head0 = 2 * (by_head ? unit / n_items : unit % pairs) + (one ? (blockIdx.x - unit0) & 1 : 0);
  int seq, qt;
  if (prm.work != nullptr) {
    seq = prm.work[2 * item];
    qt = prm.work[2 * item + 1];
  } else {
    seq = item / prm.q_tiles;
    qt = item - seq * prm.q_tiles;
  }
  const int q_begin = prm.cu_q[seq], q_len = prm.cu_q[seq + 1] - q_begin;
  if (qt * kTile >= q_len) return;                       // uniform per CTA: before any barrier or allocation
  const int ctx = prm.ctx_lens[seq];
  const int pos0 = ctx - q_len + qt * kTile, rows = min(kTile, q_len - qt * kTile);
  const int first_tile = RANGE ? prm.mods.first(pos0) / kTile : 0;
  const int n_blocks = (pos0 + rows + kBlock - 1) / kBlock - 2 * first_tile;      // pos0 + rows <= ctx

  const TwoUnit u{one, seq, qt, q_begin, pos0, rows, first_tile, n_blocks, head0};
  if (one && n_blocks > 2) attn_prefill_two<RANGE, true>(tmap_q, tmap_k, tmap_v, prm, u, status);
  else attn_prefill_two<RANGE, false>(tmap_q, tmap_k, tmap_v, prm, u, status);
}

}  // namespace
}  // namespace b2

using namespace b2;

// Whether a launch takes two heads to a block throughout (for heads whose scores are only masked; b2_attn_prefill_tc_bf16 may cut the last
// wave's blocks, and those of a launch of one head, into smaller ones). A block of two heads takes 1.6 times as long as a
// block of one (100 rows behind 1400, one wave either way: 42 and 27 us), so it pays where it saves more than that in waves. Measured, us with
// one / two heads: 8 x 128 rows, 32 heads 16.5 / 12.5; 4 x 1024 rows, 32 heads 96 / 86; 640 rows, 64 heads 30.9 / 33.1. The list of a
// captured launch has room for more items than most steps fill, one for every chunk beside those of whole tiles: only the whole
// tiles of the captured rows count (one chunk of 100 rows behind 1400 in a graph for 128 rows and four chunks, 32 heads: 42 us when
// the room counted). `work_items` 0: a grid of max_q_len x batch.
// `keys`: as many as a row can see. O stays in TMEM for all of them, where every step cuts off what does not fit; the kernel of one head adds
// tiles up in rounded arithmetic. Relative drift of sums of one sign: 8e-5 at 16384 keys, where a result's own rounding to bf16 is
// 1.4e-3 and the error against 64 bits the same for both kernels, 1.8e-4 at 32768, 7.9e-4 at 131072 (error 0.00162 instead of 0.00142).
extern "C" int b2_attn_prefill_tc_two_heads(int work_items, int captured, int64_t q_rows, int max_q_len, int batch, int n_q, int n_kv, int64_t keys) {
  if (n_kv <= 0 || (n_q / n_kv) % 2 != 0 || keys > 16384) return 0;
  int64_t tiles = work_items > 0 ? work_items : static_cast<int64_t>((max_q_len + kTile - 1) / kTile) * batch;
  if (captured && q_rows / kTile < tiles) tiles = q_rows / kTile;
  const auto waves = [](int64_t blocks) { return (blocks + kNumSMs - 1) / kNumSMs; };
  return 8 * waves(tiles * n_q / 2) < 5 * waves(tiles * n_q) ? 1 : 0;
}

// Same contract as b2_attn_prefill_bf16 with head_dim = 128 and page_size = 128 fixed; out rows 16-byte aligned.
// `token_stride` 0: paged caches [pages, n_kv, 128, 128]; otherwise the elements between two tokens' rows of keys (and of
// values) that hold all heads side by side, 128 such rows to a page. With `work` (device memory, `work_items` pairs of (sequence, query tile)) the grid is one
// CTA per item and head; `n_work` (device memory, may be null) bounds the valid items, for launches whose grid is
// fixed ahead of the batch (CUDA graphs). The caller orders the items, longest context first for an even finish.
extern "C" int b2_attn_prefill_tc_bf16(const void* q, const void* k_cache, const void* v_cache, void* out, const int32_t* cu_q,
                                       const int32_t* ctx_lens, const int32_t* block_tables, int batch, int max_blocks, int n_q,
                                       int n_kv, int max_q_len, float scale, int64_t q_rows, int64_t q_stride, int64_t out_stride,
                                       int64_t num_pages, int64_t token_stride, const int32_t* work, const int32_t* n_work, int work_items,
                                       const void* gate, int64_t gate_stride, int gate_elems, const B2AttnMods* mods,
                                       Status* status, cudaStream_t stream) {
  if (batch <= 0 || max_q_len <= 0) return 0;
  if (work != nullptr && work_items <= 0) return 0;
  if (n_q <= 0 || n_kv <= 0 || n_q % n_kv != 0 || q_stride % 8 != 0 || out_stride % 8 != 0 ||
      (reinterpret_cast<uintptr_t>(q) & 15) != 0 || (reinterpret_cast<uintptr_t>(out) & 15) != 0 || token_stride % 8 != 0 ||
      (gate != nullptr && gate_elems && (gate_stride % 8 != 0 || (reinterpret_cast<uintptr_t>(gate) & 15) != 0)))
    return -kBadArgument;
  CUtensorMap tq, tk, tv;
  const bool by_token = token_stride != 0;
  const int64_t kv_rows = num_pages * (by_token ? 1 : n_kv) * kTile, kv_cols = by_token ? static_cast<int64_t>(n_kv) * kD : kD;
  const int64_t kv_ld = (by_token ? token_stride : kD) * 2;
  if (!make_tmap_2d(&tq, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, q, q_rows, static_cast<int64_t>(n_q) * kD, q_stride * 2, kTile, 64,
                    CU_TENSOR_MAP_SWIZZLE_128B) ||
      !make_tmap_2d(&tk, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, k_cache, kv_rows, kv_cols, kv_ld, kTile, 64, CU_TENSOR_MAP_SWIZZLE_128B) ||
      !make_tmap_2d(&tv, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, v_cache, kv_rows, kv_cols, kv_ld, kTile, 64, CU_TENSOR_MAP_SWIZZLE_128B))
    return -kBadArgument;
  AttnTcParams prm{};
  prm.out = static_cast<__nv_bfloat16*>(out);
  prm.ld_out = out_stride;
  prm.cu_q = cu_q;
  prm.ctx_lens = ctx_lens;
  prm.block_tables = block_tables;
  prm.max_blocks = max_blocks;
  prm.n_q = n_q;
  prm.n_kv = n_kv;
  prm.num_pages = num_pages;
  prm.scale_log2 = scale * 1.4426950408889634f;
  prm.v_lbo = kHalfBytes;   // the second 64 columns of the head dimension are the second TMA box
  prm.v_sbo = 1024;         // 8 KV rows of 128 bytes
  prm.work = work;
  prm.n_work = work != nullptr ? n_work : nullptr;
  prm.gate = static_cast<const __nv_bfloat16*>(gate);
  prm.gate_stride = gate_stride;
  prm.gate_elems = gate_elems;
  prm.page_rows = by_token ? kTile : n_kv * kTile;
  prm.head_rows = by_token ? 0 : kTile;
  prm.head_cols = by_token ? kD : 0;
  prm.mods = make_score_mods(mods, n_q, scale);
  int64_t keys = static_cast<int64_t>(max_blocks) * kTile;
  if (prm.mods.window < keys) keys = prm.mods.window;
  if (prm.mods.chunk > 0 && prm.mods.chunk < keys) keys = prm.mods.chunk;
  prm.one_head = !b2_attn_prefill_tc_two_heads(work != nullptr ? work_items : 0, n_work != nullptr, q_rows, max_q_len, batch, n_q, n_kv, keys);
  // One head to a block is cut in two where there are keys enough to pay for bringing the parts together (16 heads, 64 rows behind 500: 12.3 us
  // cut, 11.7 by the other kernel; 300 rows behind 1000 17.0 and 18.0; 1000 behind 14000 110 and 133). A captured step only knows how many its tables
// hold: few keys under tables for 2048 are slower cut (16 heads, 64 rows behind 200 7.0 and 6.4, 128 behind 300 9.2 and 8.9), more are faster.
  if (prm.mods.masks_only() && (n_q / n_kv) % 2 == 0 && keys <= 16384 && (!prm.one_head || keys > 640)) {
    prm.q_tiles = (max_q_len + kTile - 1) / kTile;
    prm.n_items = work != nullptr ? work_items : prm.q_tiles * batch;
    static DeviceOnce two_once[2];
    const bool all = prm.mods.plain();
    auto two = all ? attn_prefill_two_kernel<false> : attn_prefill_two_kernel<true>;
    if (const int rc = two_once[all].max_smem(two, kSmemPair)) return rc;
    // with `n_work` the number of units is known on the device only, and with it how many blocks the last wave has
    const int64_t units = static_cast<int64_t>(prm.n_items) * (n_q / 2);
    if (units > (1 << 29)) return -kTooLarge;
    const int64_t more = prm.one_head ? units : n_work != nullptr ? kNumSMs / 2 : last_wave_units(static_cast<int>(units));
    const dim3 grid(static_cast<unsigned>(units + more));
    launch_pdl(two, grid, dim3(kThreadsTwo), kSmemPair, stream, tq, tk, tv, prm, status);
    return last_launch_rc();
  }
  static DeviceOnce attr_once[2];
  auto kern = prm.mods.plain() ? attn_prefill_tc_kernel<false> : attn_prefill_tc_kernel<true>;
  if (const int rc = attr_once[prm.mods.plain()].max_smem(kern, kSmemAttn)) return rc;
  dim3 grid((max_q_len + kTile - 1) / kTile, n_q, batch);
  if (work != nullptr) grid = dim3(work_items, n_q, 1);
  launch_pdl(kern, dim3(grid), dim3(kThreadsAttn), kSmemAttn, stream, tq, tk, tv, prm, status);
  return last_launch_rc();
}
