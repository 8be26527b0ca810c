// Block-scaled fp8 GEMM on CTA pairs (tcgen05 cta_group::2, kind::f8f6f4), the same product as gemm_fp8.cu:
//   Y[M, N] = sum over 128-wide K blocks kb of  sx[m, kb] * sw[n / 128, kb] * (Xq[m, kb-block] . Wq[n, kb-block])
//
// Every k-block goes into a fresh TMEM slab, which the promotion warps scale and add to f32 registers. For a 128 x 128 tile of one CTA
// that is, per k-block, 256 cycles of the tensor pipe, 256 of shared memory for its operands, as many for TMA to write them, and a chain of
// barrier, tcgen05.ld, multiply-adds and barrier that takes some 700. Two CTAs that share a 256 x BN tile read each operand byte from L2 and
// shared memory half as often for the same work, and the chain (550 cycles for 128 columns, 1000 for 256) covers two or four times
// the multiply-adds: 4096 rows through 8192 x 8192 take 237 us (2.32 PFLOP/s), 319 with tiles of one CTA. The chain still binds.
//
// Per CTA: eight promotion warps, each 32 rows x BN / 2 columns, a TMA warp and an MMA warp (the even CTA's issues for both). A promotion
// thread holds up to 128 accumulators and 64 columns of the slab. Barriers as in gemm_bf16_pair.cu; a slab is free again
// when the sixteen promotion warps of the pair have read it, before they multiply. Results leave through shared memory by TMA, so that the promotion
// warps go on to the next tile after a few hundred cycles. Loads carry no cluster broadcast. Every wait is bounded.
#include <cstdint>
#include <cuda.h>
#include <cuda_bf16.h>
#include "b2/api.h"
#include "b2/f32x2.cuh"
#include "b2/gemm_fp8.h"
#include "b2/launch.h"
#include "b2/ptx.cuh"
#include "b2/tma.h"

namespace b2 {
namespace {

constexpr int kPromotionWarps = 8;
constexpr int kFp8PairThreads = 32 * (kPromotionWarps + 4);      // TMA and MMA warps share a warpgroup with two that idle
// Registers: 384 threads are launched with 168 each; the two warpgroups of promotion warps go up to 216, the third down to 72.
constexpr int kLaunchRegs = 168, kPromotionRegs = 216, kIssueRegs = 72;
static_assert(128 * (2 * kPromotionRegs + kIssueRegs) <= kFp8PairThreads * kLaunchRegs && kFp8PairThreads * kLaunchRegs <= 65536, "register shares");

// BN = UMMA N of the pair; each CTA stages 128 rows of X and BN / 2 rows of W per k-block.
template <int BN>
struct Fp8PairCfg {
  static constexpr int kCols = BN / 2;                                 // accumulator columns of a promotion thread
  static constexpr int kABytes = 128 * 128, kBBytes = (BN / 2) * 128, kStageBytes = kABytes + kBBytes;
  static constexpr int kOutBytes = 128 * BN * 2;
  static constexpr int kSlabs = kTmemColumns / BN;
  static constexpr int kStages = (224 * 1024 - kOutBytes) / kStageBytes;      // 5 (BN 256) or 8 (BN 128)
  static constexpr int kBars = 2 * kStages + 2 * kSlabs;
  static constexpr int kSmem = kStages * kStageBytes + kOutBytes + 8 * kBars + 16 + 1024;
  static_assert(kSmem <= kMaxSmemPerCta, "ring and staged results must fit");
};

struct Fp8PairParams {
  const float *sx, *sw;
  int M, N, KB;
  int m_tiles, n_tiles;
};

// Groups of eight row tiles, column tiles varying slowest inside a group: pairs that run at the same time share both operands through L2.
__device__ __forceinline__ void fp8_pair_tile(const Fp8PairParams& p, int t, int& mt, int& nt) {
  const int group_size = 8 * p.n_tiles, group = t / group_size, first = group * 8;
  const int gm = min(p.m_tiles - first, 8), r = t - group * group_size;
  mt = first + r % gm;
  nt = r / gm;
}

template <int BN>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kFp8PairThreads, 1)
gemm_fp8_pair_kernel(const __grid_constant__ CUtensorMap tmap_x, const __grid_constant__ CUtensorMap tmap_w, const __grid_constant__ CUtensorMap tmap_y,
                     const Fp8PairParams p, Status* status) {
  using Cfg = Fp8PairCfg<BN>;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t base = (ptx::smem_u32(smem_raw) + 1023u) & ~1023u;
  const uint32_t out_base = base + Cfg::kStages * Cfg::kStageBytes, bar_base = out_base + Cfg::kOutBytes;
  auto full_bar = [&](int s) { return bar_base + 8u * s; };
  auto empty_bar = [&](int s) { return bar_base + 8u * (Cfg::kStages + s); };
  auto slab_full = [&](int s) { return bar_base + 8u * (2 * Cfg::kStages + s); };
  auto slab_empty = [&](int s) { return bar_base + 8u * (2 * Cfg::kStages + Cfg::kSlabs + s); };
  const uint32_t holder = bar_base + 8u * Cfg::kBars;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t rank = ptx::cluster_ctarank();        // 0 = the CTA that issues the MMAs
  const int pair = static_cast<int>(blockIdx.x >> 1), num_pairs = static_cast<int>(gridDim.x >> 1);
  const int total = p.m_tiles * p.n_tiles;

  if (threadIdx.x == 0) {
    ptx::prefetch_tensormap(&tmap_x);
    ptx::prefetch_tensormap(&tmap_w);
    ptx::prefetch_tensormap(&tmap_y);
    for (int s = 0; s < Cfg::kStages; ++s) {
      ptx::mbar_init(full_bar(s), 1);      // used in the even CTA only
      ptx::mbar_init(empty_bar(s), 1);
    }
    for (int s = 0; s < Cfg::kSlabs; ++s) {
      ptx::mbar_init(slab_full(s), 1);
      ptx::mbar_init(slab_empty(s), 2 * kPromotionWarps);      // used in the even CTA only: the promotion warps of both
    }
    ptx::fence_mbar_init();
  }
  if (warp == kPromotionWarps + 1) {
    ptx::tmem_alloc_pair(holder, kTmemColumns);
    ptx::tmem_relinquish_pair();
  }
  ptx::tc_fence_before();
  __syncthreads();
  ptx::cluster_sync();   // the peer's barriers are initialised before anything is signalled across the pair
  ptx::tc_fence_after();
  const uint32_t tmem_base = *reinterpret_cast<const uint32_t*>(smem_raw + (holder - ptx::smem_u32(smem_raw)));
  ptx::grid_dep_sync();   // the set-up above overlapped the previous kernel's tail

  if (warp >= kPromotionWarps) {
    ptx::setmaxnreg_dec<kIssueRegs>();
    if (warp == kPromotionWarps) {
      // ---------------------------------------------------------------- TMA producer (both CTAs)
      if (ptx::elect_one()) {
        int stage = 0;
        uint32_t phase = 0;
        bool ok = true, issued = false;
        for (int t = pair; ok && t < total; t += num_pairs) {
          int mt, nt;
          fp8_pair_tile(p, t, mt, nt);
          const int row_x = mt * 256 + static_cast<int>(rank) * 128, row_w = nt * BN + static_cast<int>(rank) * (BN / 2);
          for (int kb = 0; kb < p.KB; ++kb) {
            if (!ptx::mbar_wait(empty_bar(stage), phase ^ 1u)) {
              status_record(status, kTimeout, kSiteGemmEmpty, t, kb);
              ok = false;
              break;
            }
            const uint32_t sp = base + stage * Cfg::kStageBytes, leader_full = ptx::mapa(full_bar(stage), 0);
            if (rank == 0) ptx::mbar_arrive_expect_tx(full_bar(stage), 2 * Cfg::kStageBytes);      // both CTAs' bytes
            ptx::tma_load_2d_pair(sp, &tmap_x, leader_full, kb * 128, row_x, ptx::kEvictNormal);
            ptx::tma_load_2d_pair(sp + Cfg::kABytes, &tmap_w, leader_full, kb * 128, row_w, ptx::kEvictNormal);
            issued = true;
            if (++stage == Cfg::kStages) { stage = 0; phase ^= 1u; }
          }
        }
        // A copy of this CTA reports to the even CTA's barrier, so it cannot be waited for here: after a failed
        // wait give the copies in flight time to land before the pair meets at the closing cluster barrier.
        if (!ok && issued) ptx::nanosleep(100000);
      }
      __syncwarp();
    } else if (warp == kPromotionWarps + 1) {
      // ---------------------------------------------------------------- MMA issuer (even CTA only)
      if (rank == 0 && ptx::elect_one()) {
        constexpr uint32_t idesc = ptx::make_idesc(0, 0, 256, BN);      // e4m3 x e4m3 -> f32
        int stage = 0, slab = 0;
        uint32_t phase = 0, slab_phase = 0;
        bool ok = true;
        for (int t = pair; ok && t < total; t += num_pairs) {
          for (int kb = 0; kb < p.KB; ++kb) {
            if (!ptx::mbar_wait(slab_empty(slab), slab_phase ^ 1u)) {
              status_record(status, kTimeout, kSiteGemmTmemEmpty, t, kb);
              ok = false;
              break;
            }
            if (!ptx::mbar_wait(full_bar(stage), phase)) {
              status_record(status, kTimeout, kSiteGemmFull, t, kb);
              ok = false;
              break;
            }
            ptx::tc_fence_after();
            const uint32_t sp = base + stage * Cfg::kStageBytes;
            const uint64_t da = ptx::make_smem_desc_sw128(sp), db = ptx::make_smem_desc_sw128(sp + Cfg::kABytes);
#pragma unroll
            for (int k = 0; k < 4; ++k) ptx::tc_mma_f8_pair(tmem_base + slab * BN, da + 2u * k, db + 2u * k, idesc, k > 0 ? 1u : 0u);
            ptx::tc_commit_pair(slab_full(slab));
            ptx::tc_commit_pair(ptx::mapa(slab_full(slab), 1));
            // the stage is free in both CTAs once these MMAs have read it
            ptx::tc_commit_pair(empty_bar(stage));
            ptx::tc_commit_pair(ptx::mapa(empty_bar(stage), 1));
            if (++stage == Cfg::kStages) { stage = 0; phase ^= 1u; }
            if (++slab == Cfg::kSlabs) { slab = 0; slab_phase ^= 1u; }
          }
        }
      }
      __syncwarp();
    }
  } else {
    // ------------------------------------------------------------------ promotion and results (both CTAs, 128 rows each)
    ptx::setmaxnreg_inc<kPromotionRegs>();
    constexpr int COLS = Cfg::kCols, BOX = 64;      // BOX: columns of a TMA store
    const int quarter = warp & 3, col_base = (warp >> 2) * COLS;
    const uint32_t taddr0 = tmem_base + col_base + (static_cast<uint32_t>(quarter * 32) << 16);
    const uint32_t out_st = out_base + warp * (32 * COLS * 2);      // this warp's 32 rows, as the TMA boxes read them
    const bool by4 = p.KB % 4 == 0 && ((reinterpret_cast<uintptr_t>(p.sx) | reinterpret_cast<uintptr_t>(p.sw)) & 15) == 0;
    int slab = 0;
    uint32_t slab_phase = 0;
    bool ok = true;
    for (int t = pair; t < total; t += num_pairs) {
      int mt, nt;
      fp8_pair_tile(p, t, mt, nt);
      const int row0 = mt * 256 + static_cast<int>(rank) * 128 + quarter * 32, row = row0 + lane, col0 = nt * BN + col_base;
      const float* sx = p.sx + static_cast<int64_t>(row) * p.KB;
      const float* sw = p.sw + static_cast<int64_t>(col0 >> 7) * p.KB;
      // scales come four k-blocks at a time, requested one k-block ahead; rows and columns outside have none
      float n_row[4] = {}, n_col[4] = {};
      auto fetch = [&](int kb) {
        const bool has_row = row < p.M, has_col = col0 < p.N;
        if (by4) {
          const float4 zero = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
          const float4 a = has_row ? *reinterpret_cast<const float4*>(sx + kb) : zero, b = has_col ? *reinterpret_cast<const float4*>(sw + kb) : zero;
          n_row[0] = a.x; n_row[1] = a.y; n_row[2] = a.z; n_row[3] = a.w;
          n_col[0] = b.x; n_col[1] = b.y; n_col[2] = b.z; n_col[3] = b.w;
        } else {
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            if (has_row && kb + i < p.KB) n_row[i] = sx[kb + i];
            if (has_col && kb + i < p.KB) n_col[i] = sw[kb + i];
          }
        }
      };
      auto pick = [](const float (&v)[4], int i) { return i < 2 ? (i == 0 ? v[0] : v[1]) : (i == 2 ? v[2] : v[3]); };
      uint64_t acc[COLS / 2];
#pragma unroll
      for (int j = 0; j < COLS / 2; ++j) acc[j] = 0;
      fetch(0);
      for (int kb = 0; kb < p.KB; ++kb) {
        if (!__all_sync(0xffffffffu, ptx::mbar_wait(slab_full(slab), slab_phase))) {
          if (lane == 0) status_record(status, kTimeout, kSiteGemmTmemFull, t, kb);
          ok = false;
          break;
        }
        ptx::tc_fence_after();
        const float s = pick(n_row, kb & 3) * pick(n_col, kb & 3);
        const uint64_t s2 = pack2(s, s);
        const uint32_t taddr = taddr0 + slab * BN;
        const auto next_scales = [&] {
          if ((kb & 3) == 3 && kb + 1 < p.KB) fetch(kb + 1);
        };
        const auto give_back = [&] {      // the slab has been read
          ptx::tc_fence_before();
          __syncwarp();
          if (lane == 0) ptx::mbar_arrive_cluster_tmem(ptx::mapa(slab_empty(slab), 0));
        };
        if constexpr (COLS == 64) {
          uint32_t r[2][32];      // the second chunk of the slab is on its way while the first is added
          ptx::tmem_ld_32x32(taddr, r[0]);
          next_scales();
#pragma unroll
          for (int c = 0; c < 2; ++c) {
            ptx::tc_wait_ld();
            if (c == 0) ptx::tmem_ld_32x32(taddr + 32, r[1]);
            else give_back();
            const uint32_t(&x)[32] = r[c];
#pragma unroll
            for (int j = 0; j < 16; ++j) acc[c * 16 + j] = fma2(pack2(__uint_as_float(x[2 * j]), __uint_as_float(x[2 * j + 1])), s2, acc[c * 16 + j]);
          }
        } else {
          uint32_t r[64];      // half a slab at a time: with a chunk of 32 on its way while one is added 4096 rows through 28672 x 4096 took 452 us, this way 437
          next_scales();
#pragma unroll
          for (int c = 0; c < COLS / 64; ++c) {
            ptx::tmem_ld_32x32(taddr + c * 64, *reinterpret_cast<uint32_t(*)[32]>(r));
            ptx::tmem_ld_32x32(taddr + c * 64 + 32, *reinterpret_cast<uint32_t(*)[32]>(r + 32));
            ptx::tc_wait_ld();
            if (c == COLS / 64 - 1) give_back();
#pragma unroll
            for (int j = 0; j < 32; ++j) acc[c * 32 + j] = fma2(pack2(__uint_as_float(r[2 * j]), __uint_as_float(r[2 * j + 1])), s2, acc[c * 32 + j]);
          }
        }
        if (++slab == Cfg::kSlabs) { slab = 0; slab_phase ^= 1u; }
      }
      if (!ok) break;
      // results: bf16, boxes of 32 rows x 64 columns in the swizzled order in which TMA reads them
      if (lane == 0) ptx::tma_store_wait_read<0>();      // the tile before has left
      __syncwarp();
#pragma unroll
      for (int g = 0; g < COLS / 8; ++g) {
        uint32_t v[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const float2 f = unpack2(acc[g * 4 + i]);
          v[i] = ptx::pack_bf16x2(f.x, f.y);
        }
        const uint32_t at = out_st + (g / 8) * (32 * BOX * 2) + lane * 128 + (((g & 7) ^ (lane & 7)) << 4);
        asm volatile("st.shared.v4.u32 [%0], {%1, %2, %3, %4};" ::"r"(at), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]) : "memory");
      }
      ptx::fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0 && row0 < p.M) {
#pragma unroll
        for (int b = 0; b < COLS / BOX; ++b)
          if (col0 + b * BOX < p.N) ptx::tma_store_2d(&tmap_y, out_st + b * (32 * BOX * 2), col0 + b * BOX, row0);
        ptx::tma_store_commit();
      }
    }
    if (lane == 0) ptx::tma_store_wait<0>();
    __syncwarp();
  }

  ptx::tc_fence_before();
  __syncthreads();
  ptx::cluster_sync();   // neither CTA frees TMEM or leaves while the other may still read its shared memory / TMEM
  if (warp == kPromotionWarps + 1) {
    ptx::tc_fence_after();
    ptx::tmem_dealloc_pair(tmem_base, kTmemColumns);
  }
}

template <int BN>
int launch_fp8_pair(const void* xq, const float* xs, const void* wq, const float* ws, void* y, int M, int N, int K, int64_t ldy, Status* status,
                    cudaStream_t stream) {
  using Cfg = Fp8PairCfg<BN>;
  CUtensorMap tx, tw, ty;
  if (!make_tmap_2d(&tx, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, xq, M, K, K, 128, 128, CU_TENSOR_MAP_SWIZZLE_128B) ||
      !make_tmap_2d(&tw, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, wq, N, K, K, BN / 2, 128, CU_TENSOR_MAP_SWIZZLE_128B) ||
      !make_tmap_2d(&ty, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, y, M, N, ldy * 2, 32, 64, CU_TENSOR_MAP_SWIZZLE_128B))
    return -kBadArgument;
  const Fp8PairParams p{xs, ws, M, N, K / 128, (M + 255) / 256, (N + BN - 1) / BN};
  static DeviceOnce attr_once;
  if (const int rc = attr_once.max_smem(gemm_fp8_pair_kernel<BN>, Cfg::kSmem)) return rc;
  const int64_t total = static_cast<int64_t>(p.m_tiles) * p.n_tiles;
  const int pairs = static_cast<int>(total < kNumSMs / 2 ? total : kNumSMs / 2);
  launch_pdl(gemm_fp8_pair_kernel<BN>, dim3(2 * pairs), dim3(kFp8PairThreads), Cfg::kSmem, stream, tx, tw, ty, p, status);
  return last_launch_rc();
}

}  // namespace

int gemm_fp8_pair(const void* xq, const float* xs, const void* wq, const float* ws, void* y, int M, int N, int K, int64_t ldy, int bn, Status* status,
                  cudaStream_t stream) {
  if (bn == 256) return launch_fp8_pair<256>(xq, xs, wq, ws, y, M, N, K, ldy, status, stream);
  if (bn == 128) return launch_fp8_pair<128>(xq, xs, wq, ws, y, M, N, K, ldy, status, stream);
  return -kBadArgument;
}

}  // namespace b2
