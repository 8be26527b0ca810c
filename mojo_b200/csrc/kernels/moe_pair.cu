// Grouped expert products on CTA pairs (tcgen05 cta_group::2) for experts with more rows than a lone CTA feeds well.
//
// The two CTAs of a cluster work on 256 weight rows x up to 256 token rows of one expert: each stages 128 rows of the weights and
// half of the tokens, so a 64-wide k-block costs 32 KB per SM at the full tile where a lone CTA with a 128 x 256 tile needs 48 KB
// for the same multiplications. That path from L2 is what binds the lone kernel. The number of token rows that are
// loaded and multiplied follows the tile's own count in steps of 32 (the instruction descriptor is made per tile): the short last
// tile of an expert costs what it holds. Measured, 3001 rows x 6 of 64 experts, 2048 -> 2 x 1408 -> 2048: both
// products together 377 us (528 with lone CTAs whose last tile of an expert multiplied all 256 rows). The epilogue of the gated product is long: eight warps
// share it, and of two tokens either half of a warp works out one; with four warps and half of the lanes idle it took 447.
//
// Roles, barriers and the behaviour of a wait that runs out are those of gemm_bf16_pair.cu.
#include <cstdint>
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include "b2/act.cuh"
#include "b2/api.h"
#include "b2/config.h"
#include "b2/launch.h"
#include "b2/latent.h"
#include "b2/moe_gemm.cuh"
#include "b2/ptx.cuh"
#include "b2/status.h"
#include "b2/tma.h"

namespace b2 {
namespace {

constexpr int kEpiWarps = 8, kThreads = 64 + 32 * kEpiWarps, kStages = 6;
constexpr int kABytes = 128 * 64 * 2, kBoxRows = 32, kBoxBytes = kBoxRows * 64 * 2, kStageBytes = 2 * kABytes;      // up to 128 token rows per CTA
constexpr int kRing = kStages * kStageBytes, kBars = 2 * kStages + 4, kSmem = kRing + 8 * kBars + 16 + 1024;

struct PairTiles {
  const int4* tiles;      // (expert, first row, rows, place among the expert's tiles << 16 | their number)
  const int32_t* n_tiles;
  int n_rows, num_kb, p_blocks;      // weight rows of an expert, 64-wide k-blocks, blocks of 256 weight rows
  // Unit number w of `count` tiles. The tiles of an expert take a block of weight rows one after the other, so that it crosses HBM once: tile by
  // tile, the first product of the case above read 1.33 GB of which 0.74 are weights. The fourth word orders work and nothing else: a list that
  // b2_moe_gather did not make, or of which a part was left out, goes tile by tile, whatever that word holds.
  __device__ __forceinline__ int4 unit(int w, int count, int& pb) const {
    const int q = w / p_blocks;
    const int4 t = tiles[q];
    const int n = t.w & 0xffff, first = q - (t.w >> 16);
    if (n <= 1 || t.w < 0 || first < 0 || first + n > count || tiles[first].w != n || tiles[first + n - 1].w != ((n - 1) << 16 | n)) {
      pb = w - q * p_blocks;
      return t;
    }
    const int r = w - first * p_blocks;
    pb = r / n;
    return tiles[first + r - pb * n];
  }
};

__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kThreads, 1)
moe_pair_kernel(const __grid_constant__ CUtensorMap tmap_w, const __grid_constant__ CUtensorMap tmap_x, PairTiles p, GroupedEpiParams ep, Status* status) {
  extern __shared__ uint8_t smem_raw[];
  const uint32_t base = (ptx::smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t* smem = smem_raw + (base - ptx::smem_u32(smem_raw));
  const uint32_t bar_base = base + kRing;
  auto full_bar = [&](int s) { return bar_base + 8u * s; };
  auto empty_bar = [&](int s) { return bar_base + 8u * (kStages + s); };
  auto tmem_full = [&](int a) { return bar_base + 8u * (2 * kStages + a); };
  auto tmem_empty = [&](int a) { return bar_base + 8u * (2 * kStages + 2 + a); };
  uint32_t* holder = reinterpret_cast<uint32_t*>(smem + kRing + 8 * kBars);

  const int warp = ptx::warp_id(), lane = threadIdx.x & 31;
  const uint32_t rank = ptx::cluster_ctarank();
  const int pair = static_cast<int>(blockIdx.x >> 1), num_pairs = static_cast<int>(gridDim.x >> 1);

  if (threadIdx.x == 0) {
    ptx::prefetch_tensormap(&tmap_w);
    ptx::prefetch_tensormap(&tmap_x);
    for (int s = 0; s < kStages; ++s) {
      ptx::mbar_init(full_bar(s), 1);
      ptx::mbar_init(empty_bar(s), 1);
    }
    for (int a = 0; a < 2; ++a) {
      ptx::mbar_init(tmem_full(a), 1);
      ptx::mbar_init(tmem_empty(a), 2 * kEpiWarps);
    }
    ptx::fence_mbar_init();
  }
  if (warp == 1) {
    ptx::tmem_alloc_pair(ptx::smem_u32(holder), 512);
    ptx::tmem_relinquish_pair();
  }
  ptx::tc_fence_before();
  __syncthreads();
  ptx::cluster_sync();
  ptx::tc_fence_after();
  const uint32_t tmem_base = *holder;
  ptx::grid_dep_sync();
  const int count = *p.n_tiles, total = count * p.p_blocks;
  // token rows of a tile that take part, a multiple of 32: half of them in each CTA
  auto tile_n = [](const int4& t) { return min(256, max(32, (t.z + 31) & ~31)); };

  if (warp == 0) {
    if (ptx::elect_one()) {
      int stage = 0;
      uint32_t phase = 0;
      long issued = 0;
      bool ok = true;
      for (int w = pair; ok && w < total; w += num_pairs) {
        int pb;
        const int4 t = p.unit(w, count, pb);
        const int half = tile_n(t) / 2, boxes = (half + kBoxRows - 1) / kBoxRows;
        const int row_w = t.x * p.n_rows + pb * 256 + static_cast<int>(rank) * 128;
        const int row_x = t.y + static_cast<int>(rank) * half;
        for (int kb = 0; kb < p.num_kb; ++kb) {
          if (!ptx::mbar_wait(empty_bar(stage), phase ^ 1u)) {
            status_record(status, kTimeout, kSiteGemmEmpty, w, kb);
            ok = false;
            break;
          }
          const uint32_t sp = base + stage * kStageBytes, leader_full = ptx::mapa(full_bar(stage), 0);
          if (rank == 0) ptx::mbar_arrive_expect_tx(full_bar(stage), 2 * (kABytes + boxes * kBoxBytes));      // both CTAs' bytes
          ptx::tma_load_2d_pair(sp, &tmap_w, leader_full, kb * 64, row_w, (t.w & 0xffff) > 1 ? ptx::kEvictNormal : ptx::kEvictFirst);      // another tile may want it
          for (int b = 0; b < boxes; ++b)
            ptx::tma_load_2d_pair(sp + kABytes + b * kBoxBytes, &tmap_x, leader_full, kb * 64, row_x + b * kBoxRows, ptx::kEvictLast);
          ++issued;
          if (++stage == kStages) { stage = 0; phase ^= 1u; }
        }
      }
      if (!ok && issued > 0) ptx::nanosleep(100000);      // let copies in flight land (they report to the even CTA)
    }
    __syncwarp();
  } else if (warp == 1) {
    if (rank == 0 && ptx::elect_one()) {
      int stage = 0, acc = 0;
      uint32_t phase = 0, acc_phase = 0;
      bool ok = true;
      for (int w = pair; ok && w < total; w += num_pairs) {
        int pb;
        const int4 t = p.unit(w, count, pb);
        const uint32_t idesc = ptx::make_idesc(1, 1, 256, tile_n(t));
        if (!ptx::mbar_wait(tmem_empty(acc), acc_phase ^ 1u)) {
          status_record(status, kTimeout, kSiteGemmTmemEmpty, w, acc);
          ok = false;
          break;
        }
        ptx::tc_fence_after();
        const uint32_t d_tmem = tmem_base + acc * 256;
        for (int kb = 0; kb < p.num_kb; ++kb) {
          if (!ptx::mbar_wait(full_bar(stage), phase)) {
            status_record(status, kTimeout, kSiteGemmFull, w, kb);
            ok = false;
            break;
          }
          ptx::tc_fence_after();
          const uint32_t sp = base + stage * kStageBytes;
          const uint64_t da = ptx::make_smem_desc_sw128(sp), db = ptx::make_smem_desc_sw128(sp + kABytes);
#pragma unroll
          for (int k = 0; k < 4; ++k) ptx::tc_mma_f16_pair(d_tmem, da + 2u * k, db + 2u * k, idesc, (kb > 0 || k > 0) ? 1u : 0u);
          ptx::tc_commit_pair(empty_bar(stage));
          ptx::tc_commit_pair(ptx::mapa(empty_bar(stage), 1));
          if (++stage == kStages) { stage = 0; phase ^= 1u; }
        }
        if (!ok) break;
        ptx::tc_commit_pair(tmem_full(acc));
        ptx::tc_commit_pair(ptx::mapa(tmem_full(acc), 1));
        acc ^= 1;
        if (acc == 0) acc_phase ^= 1u;
      }
    }
    __syncwarp();
  } else {
    const int quarter = warp & 3;
    const uint32_t leader_empty0 = ptx::mapa(tmem_empty(0), 0), leader_empty1 = ptx::mapa(tmem_empty(1), 0);
    const GroupedEpilogue<256> epi{ep, (warp - 2) >> 2, kEpiWarps / 4};
    int acc = 0;
    uint32_t acc_phase = 0;
    for (int w = pair; w < total; w += num_pairs) {
      int pb;
      const int4 t = p.unit(w, count, pb);
      if (!__all_sync(0xffffffffu, ptx::mbar_wait(tmem_full(acc), acc_phase))) {
        if (lane == 0) status_record(status, kTimeout, kSiteGemmTmemFull, w, acc);
        break;
      }
      ptx::tc_fence_after();
      gemm::WorkUnit u{};
      u.pb = pb * 2 + static_cast<int>(rank);
      u.q_coord = t.y;
      u.nsplit = t.z;
      epi(u, tmem_base + acc * 256 + (static_cast<uint32_t>(quarter * 32) << 16), quarter, lane, nullptr, status);
      ptx::tc_fence_before();
      __syncwarp();
      if (lane == 0) ptx::mbar_arrive_cluster_tmem(acc == 0 ? leader_empty0 : leader_empty1);
      acc ^= 1;
      if (acc == 0) acc_phase ^= 1u;
    }
  }

  ptx::tc_fence_before();
  __syncthreads();
  ptx::cluster_sync();      // neither CTA frees TMEM or leaves while the other may still use its shared memory / TMEM
  if (warp == 1) {
    ptx::tc_fence_after();
    ptx::tmem_dealloc_pair(tmem_base, 512);
  }
}

// Tiles of up to 512 token rows, so that most experts of a long prompt have one: with two, the second read the weights again and took more
// than half of the first one's time for a few rows (281 rows an expert: 411 us a layer, 385 with one tile). Tensor memory is a ring of 16 places
// of 32 columns: a tile takes as many as its rows fill, in at most three runs of neighbouring places (one MMA each per k-step, all
// on the same weights), and the next tile starts as soon as the places it wraps into have been read.
constexpr int kPlaces = 16, kWideStages = 4, kWideStageBytes = kABytes + 256 * 128, kWideBoxRows = 16;
constexpr int kWideRing = kWideStages * kWideStageBytes, kWideBars = 2 * kWideStages + 3 * kPlaces, kWideSmem = kWideRing + 8 * kWideBars + 16 + 1024;
static_assert(kWideSmem <= kMaxSmemPerCta, "shared memory");

struct WideTile {      // the places of a tile, and how the ring goes on behind it
  int places;
  __device__ __forceinline__ explicit WideTile(const int4& t) : places(min(kPlaces, max(1, (t.z + 31) >> 5))) {}
  // f(first place of the run, places in it, places of the tile before it)
  template <class F>
  __device__ __forceinline__ void runs(int at, F&& f) const {
    for (int off = 0; off < places;) {
      const int len = min(min(8, places - off), kPlaces - at);
      f(at, len, off);
      off += len;
      at = (at + len) % kPlaces;
    }
  }
};

__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kThreads, 1)
moe_pair_wide_kernel(const __grid_constant__ CUtensorMap tmap_w, const __grid_constant__ CUtensorMap tmap_x, const __grid_constant__ CUtensorMap tmap_x64, PairTiles p,
                     GroupedEpiParams ep, Status* status) {
  extern __shared__ uint8_t smem_raw[];
  const uint32_t base = (ptx::smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t* smem = smem_raw + (base - ptx::smem_u32(smem_raw));
  const uint32_t bar_base = base + kWideRing;
  auto full_bar = [&](int s) { return bar_base + 8u * s; };
  auto empty_bar = [&](int s) { return bar_base + 8u * (kWideStages + s); };
  // No more than 16 tiles are on their way, one barrier each: a tile has at least one place, and tile n + 16 waits for all warps to have found
  // tile n. Those of the first group (places 0, 2, ...) read a place of every tile and show it by giving that back; those of the
  // second have nothing to read in a tile of one place, so they say so.
  auto tile_full = [&](int i) { return bar_base + 8u * (2 * kWideStages + i % kPlaces); };
  auto place_empty = [&](int i) { return bar_base + 8u * (2 * kWideStages + kPlaces + i); };
  auto tile_seen = [&](int i) { return bar_base + 8u * (2 * kWideStages + 2 * kPlaces + i % kPlaces); };
  uint32_t* holder = reinterpret_cast<uint32_t*>(smem + kWideRing + 8 * kWideBars);

  const int warp = ptx::warp_id(), lane = threadIdx.x & 31;
  const uint32_t rank = ptx::cluster_ctarank();
  const int pair = static_cast<int>(blockIdx.x >> 1), num_pairs = static_cast<int>(gridDim.x >> 1);

  if (threadIdx.x == 0) {
    ptx::prefetch_tensormap(&tmap_w);
    ptx::prefetch_tensormap(&tmap_x);
    for (int s = 0; s < kWideStages; ++s) {
      ptx::mbar_init(full_bar(s), 1);
      ptx::mbar_init(empty_bar(s), 1);
    }
    for (int i = 0; i < kPlaces; ++i) {
      ptx::mbar_init(tile_full(i), 1);
      ptx::mbar_init(place_empty(i), 8);      // used in the even CTA only: the four warps of either CTA that read the place
      ptx::mbar_init(tile_seen(i), 8);        // likewise: the second group of either CTA
    }
    ptx::fence_mbar_init();
  }
  if (warp == 1) {
    ptx::tmem_alloc_pair(ptx::smem_u32(holder), 512);
    ptx::tmem_relinquish_pair();
  }
  ptx::tc_fence_before();
  __syncthreads();
  ptx::cluster_sync();
  ptx::tc_fence_after();
  const uint32_t tmem_base = *holder;
  ptx::grid_dep_sync();
  const int count = *p.n_tiles, total = count * p.p_blocks;

  if (warp == 0) {
    if (ptx::elect_one()) {
      int stage = 0, at = 0;
      uint32_t phase = 0;
      bool ok = true, issued = false;
      for (int w = pair; ok && w < total; w += num_pairs) {
        int pb;
        const int4 t = p.unit(w, count, pb);
        const WideTile tile(t);
        const int row_w = t.x * p.n_rows + pb * 256 + static_cast<int>(rank) * 128;
        for (int kb = 0; kb < p.num_kb; ++kb) {
          if (!ptx::mbar_wait(empty_bar(stage), phase ^ 1u)) {
            status_record(status, kTimeout, kSiteGemmEmpty, w, kb);
            ok = false;
            break;
          }
          const uint32_t sp = base + stage * kWideStageBytes, leader_full = ptx::mapa(full_bar(stage), 0);
          if (rank == 0) ptx::mbar_arrive_expect_tx(full_bar(stage), 2 * (kABytes + tile.places * kWideBoxRows * 128));      // both CTAs' bytes
          ptx::tma_load_2d_pair(sp, &tmap_w, leader_full, kb * 64, row_w, (t.w & 0xffff) > 1 ? ptx::kEvictNormal : ptx::kEvictFirst);
          tile.runs(at, [&](int, int len, int off) {      // either CTA has one half of a run's rows
            const int row_x = t.y + off * 32 + static_cast<int>(rank) * len * kWideBoxRows;
            for (int b = 0; b < len;) {
              const bool four = len - b >= 4;
              ptx::tma_load_2d_pair(sp + kABytes + (off + b) * kWideBoxRows * 128, four ? &tmap_x64 : &tmap_x, leader_full, kb * 64, row_x + b * kWideBoxRows, ptx::kEvictLast);
              b += four ? 4 : 1;
            }
          });
          issued = true;
          if (++stage == kWideStages) { stage = 0; phase ^= 1u; }
        }
        at = (at + tile.places) % kPlaces;
      }
      if (!ok && issued) ptx::nanosleep(100000);      // let copies in flight land (they report to the even CTA)
    }
    __syncwarp();
  } else if (warp == 1) {
    if (rank == 0 && ptx::elect_one()) {
      int stage = 0, at = 0, n = 0;
      uint32_t phase = 0, used = 0;      // `used`: a bit per place, how often it has been filled, modulo 2
      bool ok = true;
      for (int w = pair; ok && w < total; w += num_pairs, ++n) {
        int pb;
        const int4 t = p.unit(w, count, pb);
        const WideTile tile(t);
        for (int i = 0; i < tile.places && ok; ++i) {
          const int place = (at + i) % kPlaces;
          if (!ptx::mbar_wait(place_empty(place), ((used >> place) & 1u) ^ 1u)) {
            status_record(status, kTimeout, kSiteGemmTmemEmpty, w, place);
            ok = false;
          }
          used ^= 1u << place;
        }
        if (ok && !ptx::mbar_wait(tile_seen(n), ((n / kPlaces) & 1) ^ 1u)) {
          status_record(status, kTimeout, kSiteGemmTmemEmpty, w, kPlaces);
          ok = false;
        }
        if (!ok) break;
        ptx::tc_fence_after();
        for (int kb = 0; kb < p.num_kb; ++kb) {
          if (!ptx::mbar_wait(full_bar(stage), phase)) {
            status_record(status, kTimeout, kSiteGemmFull, w, kb);
            ok = false;
            break;
          }
          ptx::tc_fence_after();
          const uint32_t sp = base + stage * kWideStageBytes;
          const uint64_t da = ptx::make_smem_desc_sw128(sp);
          tile.runs(at, [&](int place, int len, int off) {
            const uint32_t idesc = ptx::make_idesc(1, 1, 256, 32 * len);
            const uint64_t db = ptx::make_smem_desc_sw128(sp + kABytes + off * kWideBoxRows * 128);
#pragma unroll
            for (int k = 0; k < 4; ++k) ptx::tc_mma_f16_pair(tmem_base + place * 32, da + 2u * k, db + 2u * k, idesc, (kb > 0 || k > 0) ? 1u : 0u);
          });
          ptx::tc_commit_pair(empty_bar(stage));
          ptx::tc_commit_pair(ptx::mapa(empty_bar(stage), 1));
          if (++stage == kWideStages) { stage = 0; phase ^= 1u; }
        }
        if (!ok) break;
        ptx::tc_commit_pair(tile_full(n));
        ptx::tc_commit_pair(ptx::mapa(tile_full(n), 1));
        at = (at + tile.places) % kPlaces;
      }
    }
    __syncwarp();
  } else {
    const int quarter = warp & 3, group = (warp - 2) >> 2;
    const GroupedEpilogue<512> epi{ep};
    int at = 0, n = 0;
    for (int w = pair; w < total; w += num_pairs, ++n) {
      int pb;
      const int4 t = p.unit(w, count, pb);
      const WideTile tile(t);
      if (!__all_sync(0xffffffffu, ptx::mbar_wait(tile_full(n), (n / kPlaces) & 1))) {
        if (lane == 0) status_record(status, kTimeout, kSiteGemmTmemFull, w, n);
        break;
      }
      if (group == 1 && lane == 0) ptx::mbar_arrive_cluster_tmem(ptx::mapa(tile_seen(n), 0));
      ptx::tc_fence_after();
      gemm::WorkUnit u{};
      u.pb = pb * 2 + static_cast<int>(rank);
      u.q_coord = t.y;
      u.nsplit = t.z;
      for (int c = group; c < tile.places; c += kEpiWarps / 4) {
        const int place = (at + c) % kPlaces;
        if (c * 32 < t.z) epi.chunk(u, tmem_base + place * 32 + (static_cast<uint32_t>(quarter * 32) << 16), c * 32, quarter, lane);
        ptx::tc_fence_before();
        __syncwarp();
        if (lane == 0) ptx::mbar_arrive_cluster_tmem(ptx::mapa(place_empty(place), 0));
      }
      at = (at + tile.places) % kPlaces;
    }
  }

  ptx::tc_fence_before();
  __syncthreads();
  ptx::cluster_sync();      // neither CTA frees TMEM or leaves while the other may still use its shared memory / TMEM
  if (warp == 1) {
    ptx::tc_fence_after();
    ptx::tmem_dealloc_pair(tmem_base, 512);
  }
}

}  // namespace

int launch_moe_pair(const void* x, const void* w, const int32_t* tiles, const int32_t* n_tiles, void* y, int rows, int experts, int n, int k, int epilogue,
                    const B2EpiAct* act, bool wide, Status* status, cudaStream_t stream) {
  CUtensorMap tw, tx;
  if (!make_tmap_2d(&tw, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, w, static_cast<uint64_t>(experts) * n, k, static_cast<uint64_t>(k) * 2, 128, 64, CU_TENSOR_MAP_SWIZZLE_128B) ||
      !make_tmap_2d(&tx, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, x, rows, k, static_cast<uint64_t>(k) * 2, wide ? kWideBoxRows : kBoxRows, 64, CU_TENSOR_MAP_SWIZZLE_128B))
    return -kBadArgument;
  const PairTiles p{reinterpret_cast<const int4*>(tiles), n_tiles, n, (k + 63) / 64, (n + 255) / 256};
  const GroupedEpiParams ep{static_cast<__nv_bfloat16*>(y), epilogue == B2_EPI_SWIGLU ? n / 2 : n, n, epilogue, act != nullptr ? *act : kPlainAct};
  static DeviceOnce attr_once[2];
  if (wide) {
    CUtensorMap tx64;
    if (!make_tmap_2d(&tx64, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, x, rows, k, static_cast<uint64_t>(k) * 2, 4 * kWideBoxRows, 64, CU_TENSOR_MAP_SWIZZLE_128B)) return -kBadArgument;
    if (const int rc = attr_once[1].max_smem(moe_pair_wide_kernel, kWideSmem)) return rc;
    launch_pdl(moe_pair_wide_kernel, dim3(kNumSMs), dim3(kThreads), kWideSmem, stream, tw, tx, tx64, p, ep, status);
    return last_launch_rc();
  }
  if (const int rc = attr_once[0].max_smem(moe_pair_kernel, kSmem)) return rc;
  launch_pdl(moe_pair_kernel, dim3(kNumSMs), dim3(kThreads), kSmem, stream, tw, tx, p, ep, status);
  return last_launch_rc();
}

}  // namespace b2
