// GGUF k-quant weights: standalone dequantisation and the product with packed weights
//   Y[M, N] = X[M, K] * dequant(Wq)[N, K]^T     Wq: Q4_K or Q6_K super-blocks, row-major [N][K / 256].
// The product is for decode-sized M, where the packed weights (4.5 / 6.56 bits each) are what has to cross HBM. The quants
// themselves, small integers and exact in bf16, go to the tensor cores; the scales of their groups are applied to the 32-bit
// partial sums. That costs less than expanding every weight (a shift and a mask for two weights instead of a conversion, a
// multiply-add and a rounding each) and rounds nothing.
#include <algorithm>
#include <cstdint>
#include <cuda.h>
#include <type_traits>
#include <cuda_bf16.h>
#include "b2/api.h"
#include "b2/launch.h"
#include "b2/gguf.cuh"
#include "b2/ptx.cuh"
#include "b2/tma.h"

namespace b2 {
namespace {

// One thread per 64 weights, wide loads (tensor 16-byte aligned).
__global__ void dequant64_kernel(const uint8_t* __restrict__ wq, int ggml_type, __nv_bfloat16* __restrict__ out, int64_t n_pairs) {
  const int64_t pidx = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (pidx >= n_pairs) return;
  const int64_t blk = pidx >> 2;
  const int g0 = static_cast<int>(pidx & 3) * 2;
  float v[64];
  if (ggml_type == gguf::kTypeQ4K) gguf::q4k_dequant64(wq + blk * gguf::kQ4KBytes, g0, v);
  else gguf::q6k_dequant64(wq + blk * gguf::kQ6KBytes, g0, v);
  uint4* dst = reinterpret_cast<uint4*>(out + pidx * 64);
#pragma unroll
  for (int c = 0; c < 8; ++c) {
    uint4 pk;
    pk.x = ptx::pack_bf16x2(v[c * 8 + 0], v[c * 8 + 1]);
    pk.y = ptx::pack_bf16x2(v[c * 8 + 2], v[c * 8 + 3]);
    pk.z = ptx::pack_bf16x2(v[c * 8 + 4], v[c * 8 + 5]);
    pk.w = ptx::pack_bf16x2(v[c * 8 + 6], v[c * 8 + 7]);
    dst[c] = pk;
  }
}

__global__ void dequant_kernel(const uint8_t* __restrict__ wq, int ggml_type, __nv_bfloat16* __restrict__ out, int64_t n_groups) {
  // one thread per 32 weights
  const int64_t gidx = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (gidx >= n_groups) return;
  const int64_t blk = gidx >> 3;
  const int g = static_cast<int>(gidx & 7);
  float v[32];
  if (ggml_type == gguf::kTypeQ4K) gguf::q4k_dequant32(wq + blk * gguf::kQ4KBytes, g, v);
  else gguf::q6k_dequant32(wq + blk * gguf::kQ6KBytes, g, v);
  uint4* dst = reinterpret_cast<uint4*>(out + gidx * 32);
#pragma unroll
  for (int c = 0; c < 4; ++c) {
    uint4 pk;
    pk.x = ptx::pack_bf16x2(v[c * 8 + 0], v[c * 8 + 1]);
    pk.y = ptx::pack_bf16x2(v[c * 8 + 2], v[c * 8 + 3]);
    pk.z = ptx::pack_bf16x2(v[c * 8 + 4], v[c * 8 + 5]);
    pk.w = ptx::pack_bf16x2(v[c * 8 + 6], v[c * 8 + 7]);
    dst[c] = pk;
  }
}

// ------------------------------------------------------------------------------------------------------
// Product with packed weights
// ------------------------------------------------------------------------------------------------------
// A CTA of four warps takes 64 weight rows and one slice of K, a warp 16 of the rows. Every warp streams its rows by itself: a
// stage is two super-blocks of 16 rows, one TMA box into a two-stage ring of its own, so that no warp waits for another and an SM has
// more than 100 KB on the way. (A bulk copy for every row's 288 or 432 bytes bound the kernel: 229000 of them in 28672 x 4096.) mma.sync m16n8k16 with the weights as the 16-row operand: tcgen05 would need the operand in
// shared memory as bf16, a store and a fence for every 64 weights, and at these M the tensor work is small either way. Where the
// rows alone do not fill the machine, the CTAs of a cluster share 64 rows and split K; the first one adds up the partial sums
// in a fixed order. The order of k inside a group is the order in which the bytes hold the quants: x is permuted to match.
// Measured, 4 rows through the 28672 x 4096 (Q4_K) and 4096 x 14336 (Q6_K) products of a feed-forward: 34 and 23 us, with bulk copies 39 and 25 in a
// profile and 84 us for both and the activation between them; the packed bytes are 17 us of HBM time. The integer pipe that takes the
// quants apart is busy for half of the time, and 448 blocks of rows over 148 SMs leave a fifth of them idle at the end.
constexpr int kRows = 64, kQWarps = 4, kQThreads = 128, kMaxTokens = 32, kMaxSplit = 8;
constexpr float kExtreme = 1e27f;      // times 32 columns, 143 and the largest factor (63 times a half): well inside 32 bits

template <int TYPE>
struct Pack;
template <>
struct Pack<gguf::kTypeQ4K> {
  static constexpr int kBytes = gguf::kQ4KBytes, kStages = 2;
  // two super-blocks of a row, 288 bytes = 72 words: the 8-byte reads of 4 rows x 4 lanes fall on different banks
  static constexpr int kRowStride = 288;
};
template <>
struct Pack<gguf::kTypeQ6K> {
  static constexpr int kBytes = gguf::kQ6KBytes, kStages = 2;
  // 420 bytes of a row from the 16-byte boundary below them, 432 bytes = 108 words: 4-byte reads of 8 rows x 4 lanes likewise
  static constexpr int kRowStride = 432;
};

struct PackedArgs {
  const __nv_bfloat16* x;
  const uint8_t* wq;
  __nv_bfloat16* y;
  int M, N, K;
  int blocks_per_row;      // K / 256
  int pairs;               // pairs of super-blocks in a row
  int splits;              // CTAs of a cluster that share K
  int tma;                 // rows lie on 16-byte boundaries: TMA; otherwise the lanes copy
};

__device__ __forceinline__ void mma_bf16(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
               : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
// the first product of a sum: no accumulator registers to clear
__device__ __forceinline__ void mma_bf16_first(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
               : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
               : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "f"(0.0f));
}
// (w & mask) | 0x4300 in both halves: bf16 numbers 128 + q for q < 128
__device__ __forceinline__ uint32_t biased(uint32_t w, uint32_t mask) { return (w & mask) | 0x43004300u; }
__device__ __forceinline__ uint32_t minus(uint32_t v, uint32_t bias) {
  const __nv_bfloat162 r = __hsub2(*reinterpret_cast<const __nv_bfloat162*>(&v), *reinterpret_cast<const __nv_bfloat162*>(&bias));
  return *reinterpret_cast<const uint32_t*>(&r);
}

// Shared memory behind the rings: sums of x over groups of 32 columns (Q4_K only), [group of the slice][token].
template <int TYPE>
__host__ __device__ constexpr int packed_ring_bytes() {
  return kQWarps * Pack<TYPE>::kStages * 16 * Pack<TYPE>::kRowStride;
}

// groups of 32 columns of the longest slice
__host__ __device__ constexpr int packed_groups(int pairs, int splits) { return (pairs + splits - 1) / splits * 16; }
template <int TYPE, int NT>
__host__ __device__ constexpr int packed_table_offset(int pairs, int splits) {
  return packed_ring_bytes<TYPE>() + (TYPE == gguf::kTypeQ4K ? packed_groups(pairs, splits) * NT * 8 * 4 : 0);
}
template <int TYPE, int NT>
__host__ __device__ constexpr int packed_smem(int pairs, int splits) {
  return packed_table_offset<TYPE, NT>(pairs, splits) + (TYPE == gguf::kTypeQ4K ? kQWarps * 128 * 8 : 0);
}

template <int TYPE, int NT>
__global__ void __launch_bounds__(kQThreads, 4) packed_gemm_kernel(const __grid_constant__ CUtensorMap tmap_w, const PackedArgs a, Status* status) {
  constexpr bool Q4 = TYPE == gguf::kTypeQ4K;
  constexpr int kStages = Pack<TYPE>::kStages, kStride = Pack<TYPE>::kRowStride, kBlk = Pack<TYPE>::kBytes, kStage = 16 * kStride;
  extern __shared__ __align__(128) uint4 packed_smem[];
  __shared__ uint64_t bars[kQWarps * kStages];
  uint8_t* smem = reinterpret_cast<uint8_t*>(packed_smem);
  const int warp = ptx::warp_id(), lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const int rank = blockIdx.x % a.splits, n0 = blockIdx.x / a.splits * kRows + warp * 16;
  const int p0 = static_cast<int>(static_cast<int64_t>(a.pairs) * rank / a.splits), p1 = static_cast<int>(static_cast<int64_t>(a.pairs) * (rank + 1) / a.splits);
  uint8_t* ring = smem + warp * kStages * kStage;
  const uint32_t bar0 = ptx::smem_u32(&bars[warp * kStages]);
  if (lane == 0) {
    for (int s = 0; s < kStages; ++s) ptx::mbar_init(bar0 + 8 * s, 1);
    ptx::fence_mbar_init();
  }
  __syncwarp();
  ptx::grid_dep_sync();

  const int64_t row_bytes = static_cast<int64_t>(a.blocks_per_row) * kBlk;
  // A stage: super-blocks 2p and 2p + 1 (the last pair may be one) of 16 rows.
  auto fill = [&](int p, int s) {
    uint8_t* to = ring + s * kStage;
    if (a.tma) {      // what lies past a row's end or the last row arrives as zeros
      if (lane == 0) {
        ptx::mbar_arrive_expect_tx(bar0 + 8 * s, kStage);
        ptx::tma_load_2d(ptx::smem_u32(to), &tmap_w, bar0 + 8 * s, ((2 * p * kBlk) & ~15) / 4, n0, ptx::kEvictNormal);
      }
    } else {      // rows past N repeat the last one
      const int blocks = min(2, a.blocks_per_row - 2 * p);
      for (int r = 0; r < 16; ++r) {
        const uint8_t* src = a.wq + min(n0 + r, a.N - 1) * row_bytes + static_cast<int64_t>(2 * p) * kBlk;
        uint8_t* dst = to + r * kStride + ((2 * p * kBlk) & 15);
        for (int i = lane; i < blocks * kBlk; i += 32) dst[i] = src[i];
      }
      __syncwarp();
      if (lane == 0) ptx::mbar_arrive(bar0 + 8 * s);
    }
  };
  const bool active = n0 < a.N;
  if (active)
    for (int s = 0; s < kStages && p0 + s < p1; ++s) fill(p0 + s, s);

  // ---- sums of x per group of 32, for the minima of Q4_K: y += a (S - 128 X) - b X with S the products of 128 + q ----
  // An infinite x, or one whose S could overflow where the product does not, must not meet that difference: the sum is marked by a
  // NaN and the group takes the weights as they are.
  bool extreme = false;
  float* xsum = reinterpret_cast<float*>(smem + packed_ring_bytes<TYPE>());
  if (Q4) {
    const int g0 = p0 * 16, groups = min(p1 * 16, a.K / 32) - g0;
    const int items = groups * a.M;      // sums of rows past M are never used
    for (int i0 = threadIdx.x; i0 < items; i0 += 4 * kQThreads) {
      uint4 q[4][4];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int i = min(i0 + u * kQThreads, items - 1), tok = i / groups, gr = i - tok * groups;
        const uint4* src = reinterpret_cast<const uint4*>(a.x + static_cast<int64_t>(tok) * a.K + (g0 + gr) * 32);
#pragma unroll
        for (int j = 0; j < 4; ++j) q[u][j] = src[j];
      }
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int i = i0 + u * kQThreads, tok = i / groups, gr = i - tok * groups;
        float sum = 0.0f;
        __nv_bfloat162 most = __float2bfloat162_rn(0.0f);      // largest magnitude, NaN if there is one
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          sum += (ptx::bf16_lo(q[u][j].x) + ptx::bf16_hi(q[u][j].x)) + (ptx::bf16_lo(q[u][j].y) + ptx::bf16_hi(q[u][j].y));
          sum += (ptx::bf16_lo(q[u][j].z) + ptx::bf16_hi(q[u][j].z)) + (ptx::bf16_lo(q[u][j].w) + ptx::bf16_hi(q[u][j].w));
          const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&q[u][j]);
          most = __hmax2_nan(most, __hmax2_nan(__hmax2_nan(__habs2(h[0]), __habs2(h[1])), __hmax2_nan(__habs2(h[2]), __habs2(h[3]))));
        }
        const bool far = !(fmaxf(__low2float(most), __high2float(most)) < kExtreme) || __hisnan(most.x) || __hisnan(most.y);
        extreme = extreme || far;
        if (i < items) xsum[gr * (NT * 8) + tok] = far ? __int_as_float(0x7fffffff) : sum;
      }
    }
    extreme = __syncthreads_or(extreme) != 0;
  }

  float acc[NT][4];
#pragma unroll
  for (int i = 0; i < NT; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = 0.0f;

  if (active) {
    const __nv_bfloat16* xrow[NT];      // this lane's piece of a token's row
#pragma unroll
    for (int i = 0; i < NT; ++i) xrow[i] = a.x + static_cast<int64_t>(min(i * 8 + g, a.M - 1)) * a.K + t * (Q4 ? 8 : 4);
    // the B operands of 32 columns from column k on: two k16 steps
    const auto frag = [&](int i, int k) {
      if constexpr (Q4) {
        const uint4 xv = *reinterpret_cast<const uint4*>(xrow[i] + k);
        return make_uint4(__byte_perm(xv.x, xv.y, 0x5410), __byte_perm(xv.x, xv.y, 0x7632), __byte_perm(xv.z, xv.w, 0x5410), __byte_perm(xv.z, xv.w, 0x7632));
      } else {
        const uint2 x0 = *reinterpret_cast<const uint2*>(xrow[i] + k), x1 = *reinterpret_cast<const uint2*>(xrow[i] + k + 16);
        return make_uint4(__byte_perm(x0.x, x0.y, 0x5410), __byte_perm(x0.x, x0.y, 0x7632), __byte_perm(x1.x, x1.y, 0x5410), __byte_perm(x1.x, x1.y, 0x7632));
      }
    };
    float2* tab = reinterpret_cast<float2*>(smem + packed_table_offset<TYPE, NT>(a.pairs, a.splits)) + warp * 128;      // Q4_K: factor and minimum, [group][row]
    bool ok = true;
    const auto walk = [&](auto marked) {      // `marked`: some sum is
      for (int p = p0; p < p1; ++p) {
        const int it = p - p0, s = it % kStages;
        if (!ptx::mbar_wait(bar0 + 8 * s, (it / kStages) & 1)) ok = false;
        if (!__all_sync(0xffffffffu, ok)) {
          if (lane == 0) status_record(status, kTimeout, kSiteGemmFull, blockIdx.x, p);
          break;
        }
        const int blocks = min(2, a.blocks_per_row - 2 * p);
        const uint8_t* base = ring + s * kStage + ((2 * p * kBlk) & 15);
#pragma unroll(Q4 ? 1 : 2)      // Q6_K: how its words are read depends on b
        for (int b = 0; b < 2; ++b) {
          if (b == blocks) break;
          const uint8_t* r0 = base + b * kBlk + g * kStride;       // rows g and g + 8 of the warp's 16
          const uint8_t* r1 = r0 + 8 * kStride;
          const int k0 = (2 * p + b) * 256;
          if constexpr (Q4) {
            // lane t of a row's four works out the scales of groups t and t + 4, for all lanes: factor, and what goes with the sum of
            // x (where sums are marked, the minimum)
            __syncwarp();
#pragma unroll
            for (int r = 0; r < 2; ++r) {
              const uint4 h = *reinterpret_cast<const uint4*>(r ? r1 : r0);
              const float d = __half2float(__ushort_as_half(static_cast<uint16_t>(h.x & 0xffff)));
              const float dmin = __half2float(__ushort_as_half(static_cast<uint16_t>(h.x >> 16)));
              const uint32_t c0 = (h.y >> (8 * t)) & 0xffu, c1 = (h.z >> (8 * t)) & 0xffu, c2 = (h.w >> (8 * t)) & 0xffu;
              const float a0 = d * static_cast<float>(c0 & 63u), b0 = dmin * static_cast<float>(c1 & 63u);
              const float a1 = d * static_cast<float>((c2 & 15u) | ((c0 >> 6) << 4)), b1 = dmin * static_cast<float>((c2 >> 4) | ((c1 >> 6) << 4));
              tab[t * 16 + g + 8 * r] = make_float2(a0, decltype(marked)::value ? b0 : fmaf(-128.0f, a0, -b0));
              tab[(t + 4) * 16 + g + 8 * r] = make_float2(a1, decltype(marked)::value ? b1 : fmaf(-128.0f, a1, -b1));
            }
            __syncwarp();
#pragma unroll
            for (int c = 0; c < 4; ++c) {      // 32 bytes: groups 2c (low nibbles) and 2c + 1 (high nibbles)
              const uint2 q0 = *reinterpret_cast<const uint2*>(r0 + 16 + c * 32 + t * 8), q1 = *reinterpret_cast<const uint2*>(r1 + 16 + c * 32 + t * 8);
#pragma unroll
              for (int hi = 0; hi < 2; ++hi) {
                const int j = 2 * c + hi;
                const float2 s0 = tab[j * 16 + g], s1 = tab[j * 16 + g + 8];
                const float a0 = s0.x, a1 = s1.x, b0 = s0.y, b1 = s1.y;      // b only where sums are marked
                const float m0 = decltype(marked)::value ? fmaf(-128.0f, a0, -b0) : b0, m1 = decltype(marked)::value ? fmaf(-128.0f, a1, -b1) : b1;
                const uint32_t w00 = q0.x >> (4 * hi), w01 = q0.y >> (4 * hi), w10 = q1.x >> (4 * hi), w11 = q1.y >> (4 * hi);
                const uint32_t mk = 0x000f000fu;
                const uint32_t f00 = biased(w00, mk), f01 = biased(w00 >> 8, mk), f02 = biased(w01, mk), f03 = biased(w01 >> 8, mk);
                const uint32_t f10 = biased(w10, mk), f11 = biased(w10 >> 8, mk), f12 = biased(w11, mk), f13 = biased(w11 >> 8, mk);
                const float* xs = xsum + ((2 * (p - p0) + b) * 8 + j) * (NT * 8) + 2 * t;
#pragma unroll
                for (int i = 0; i < NT; ++i) {
                  const uint4 xv = frag(i, k0 + j * 32);
                  float d[4];
                  mma_bf16_first(d, f00, f10, f01, f11, xv.x, xv.y);
                  mma_bf16(d, f02, f12, f03, f13, xv.z, xv.w);
                  const float2 X = *reinterpret_cast<const float2*>(xs + i * 8);
                  if constexpr (decltype(marked)::value) {
                    // the group's weights themselves, rounded to bf16, for the tokens whose sum is marked
                    const auto real = [](uint32_t f, float sc, float mn) {
                      return ptx::pack_bf16x2(fmaf(sc, ptx::bf16_lo(f) - 128.0f, -mn), fmaf(sc, ptx::bf16_hi(f) - 128.0f, -mn));
                    };
                    float e[4];
                    mma_bf16_first(e, real(f00, a0, b0), real(f10, a1, b1), real(f01, a0, b0), real(f11, a1, b1), xv.x, xv.y);
                    mma_bf16(e, real(f02, a0, b0), real(f12, a1, b1), real(f03, a0, b0), real(f13, a1, b1), xv.z, xv.w);
                    acc[i][0] = X.x == X.x ? fmaf(a0, d[0], fmaf(m0, X.x, acc[i][0])) : acc[i][0] + e[0];
                    acc[i][1] = X.y == X.y ? fmaf(a0, d[1], fmaf(m0, X.y, acc[i][1])) : acc[i][1] + e[1];
                    acc[i][2] = X.x == X.x ? fmaf(a1, d[2], fmaf(m1, X.x, acc[i][2])) : acc[i][2] + e[2];
                    acc[i][3] = X.y == X.y ? fmaf(a1, d[3], fmaf(m1, X.y, acc[i][3])) : acc[i][3] + e[3];
                  } else {
                    acc[i][0] = fmaf(a0, d[0], fmaf(m0, X.x, acc[i][0]));
                    acc[i][1] = fmaf(a0, d[1], fmaf(m0, X.y, acc[i][1]));
                    acc[i][2] = fmaf(a1, d[2], fmaf(m1, X.x, acc[i][2]));
                    acc[i][3] = fmaf(a1, d[3], fmaf(m1, X.y, acc[i][3]));
                  }
                }
              }
            }
          } else {
            // the first block of a pair starts on a 4-byte boundary, the second 210 bytes later between two
            auto word = [b](const uint8_t* q) {
              if (b == 0) return *reinterpret_cast<const uint32_t*>(q);
              const uint32_t* w = reinterpret_cast<const uint32_t*>(q - 2);
              return __byte_perm(w[0], w[1], 0x5432);
            };
            auto scale_d = [](const uint8_t* r) { return __half2float(__ushort_as_half(*reinterpret_cast<const uint16_t*>(r + 208))); };
            const float d0 = scale_d(r0), d1 = scale_d(r1);
#pragma unroll
            for (int half = 0; half < 2; ++half) {
              // lane t holds the scales of quarter t (two groups of 16) of this half
              const uint16_t s0 = *reinterpret_cast<const uint16_t*>(r0 + 192 + half * 8 + t * 2), s1 = *reinterpret_cast<const uint16_t*>(r1 + 192 + half * 8 + t * 2);
              const float sc[2][2] = {{d0 * static_cast<int8_t>(s0 & 0xff), d0 * static_cast<int8_t>(s0 >> 8)},
                                      {d1 * static_cast<int8_t>(s1 & 0xff), d1 * static_cast<int8_t>(s1 >> 8)}};
              // columns 16 grp .. + 15 of every quarter: lane t has bytes 4t .. 4t + 3
              uint32_t high[2][2], low[2][2][2];      // [grp][row], [grp][row][even / odd quarters]
#pragma unroll
              for (int grp = 0; grp < 2; ++grp)
#pragma unroll
                for (int r = 0; r < 2; ++r) {
                  const uint8_t* rr = (r ? r1 : r0) + grp * 16 + t * 4;
                  high[grp][r] = word(rr + 128 + half * 32);
                  low[grp][r][0] = word(rr + half * 64);
                  low[grp][r][1] = word(rr + half * 64 + 32);
                }
#pragma unroll
              for (int qt = 0; qt < 4; ++qt) {
                const int owner = (lane & ~3) | qt;
                uint4 xv[NT];
#pragma unroll
                for (int i = 0; i < NT; ++i) xv[i] = frag(i, k0 + half * 128 + qt * 32);
#pragma unroll
                for (int grp = 0; grp < 2; ++grp) {
                  const float a0 = __shfl_sync(0xffffffffu, sc[0][grp], owner), a1 = __shfl_sync(0xffffffffu, sc[1][grp], owner);
                  uint32_t f[2][2];
#pragma unroll
                  for (int r = 0; r < 2; ++r) {
                    const uint32_t l = low[grp][r][qt & 1] >> (4 * (qt >> 1)), h = high[grp][r];
                    const uint32_t hs = qt < 2 ? h << (4 - 2 * qt) : h >> (2 * qt - 4);      // the two high bits to bits 4 and 5
                    const uint32_t q = (l & 0x0f0f0f0fu) | (hs & 0x30303030u);
                    f[r][0] = minus(biased(q, 0x003f003fu), 0x43204320u);                     // 128 + q - 160: exact
                    f[r][1] = minus(biased(q >> 8, 0x003f003fu), 0x43204320u);
                  }
#pragma unroll
                  for (int i = 0; i < NT; ++i) {
                    float d[4];
                    mma_bf16_first(d, f[0][0], f[1][0], f[0][1], f[1][1], grp ? xv[i].z : xv[i].x, grp ? xv[i].w : xv[i].y);
                    acc[i][0] = fmaf(a0, d[0], acc[i][0]);
                    acc[i][1] = fmaf(a0, d[1], acc[i][1]);
                    acc[i][2] = fmaf(a1, d[2], acc[i][2]);
                    acc[i][3] = fmaf(a1, d[3], acc[i][3]);
                  }
                }
              }
            }
          }
        }
        __syncwarp();      // every lane has read the stage
        if (p + kStages < p1) fill(p + kStages, s);
      }
    };
    if constexpr (Q4) {
      if (extreme) walk(std::true_type{});
      else walk(std::false_type{});
    } else {
      walk(std::false_type{});
    }
    if (!__all_sync(0xffffffffu, ok)) {
      // copies in flight must land before the shared memory is given up
      for (int s = 0; s < kStages; ++s)
        for (int ph = 0; ph < 2; ++ph) ptx::mbar_wait(bar0 + 8 * s, ph, 100000000ull);
    }
  }

  // ---- partial sums of the cluster's CTAs, in order of rank ----
  float* part = reinterpret_cast<float*>(smem);      // [rank - 1][thread][NT * 4] in the first CTA; the rings are done with
  if (a.splits > 1) {
    ptx::cluster_sync();
    if (rank > 0) {
      const uint32_t to = ptx::mapa(ptx::smem_u32(part + (rank - 1) * kQThreads * NT * 4), 0);
#pragma unroll
      for (int i = 0; i < NT; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) ptx::st_cluster_f32(to + ((i * 4 + j) * kQThreads + threadIdx.x) * 4, acc[i][j]);
    }
    ptx::cluster_sync();
    if (rank > 0) return;
    for (int r = 0; r + 1 < a.splits; ++r)
#pragma unroll
      for (int i = 0; i < NT; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] += part[(r * NT * 4 + i * 4 + j) * kQThreads + threadIdx.x];
  }
#pragma unroll
  for (int i = 0; i < NT; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int n = n0 + g + (j >> 1) * 8, m = i * 8 + 2 * t + (j & 1);
      if (n < a.N && m < a.M) a.y[static_cast<int64_t>(m) * a.N + n] = __float2bfloat16(acc[i][j]);
    }
}

// What a CTA may take: ring and sums 200 KB, as many columns of a row as before there were tables, which come on top.
template <int TYPE>
constexpr int kMostSmem = 200 * 1024 + (TYPE == gguf::kTypeQ4K ? kQWarps * 128 * 8 : 0);
static_assert(kMostSmem<gguf::kTypeQ4K> + 1024 <= kMaxSmemPerCta, "shared memory");

// K is split until every SM has some CTAs. Two of them fill it for up to eight tokens (4 tokens, us by splits 1 / 2 / 4 / 8: 28672 x 4096 Q4_K
// 34 / 35 / 40 / 53, 4096 x 14336 Q6_K 62 / 33 / 23 / 25); more tokens hold a warp of Q4_K longer, and three per SM in four rounds is what
// one without splits gets (32 tokens 123 / 91 / 97 / 125, Q6_K 150 / 72 / 49 / 79). Rows that lanes copy (`tma` false) wait for every word of
// theirs: two CTAs per SM or more, in one wave if that will do (1 token, Q6_K, splits 2 / 4 / 8: 4096 x 11008 338 / 185 / 95, 5120 x 13824
// 445 / 229 / 248, 13824 x 5120 155 / 183). Where that leaves the fullest SM with more than its share, or slices are long, splits go on up to four
// CTAs per SM (172 blocks of rows, 11008 x 4096: Q6_K, 32 tokens, two splits 50.0, four 45.0; 344 blocks, Q4_K, 1 token, one / two 30.5 / 26.8;
// 8192 x 28672, Q6_K, 16 tokens, two / four / eight 124 / 96 / 100, 24 tokens 202 / 143 / 172). An eighth off the fullest SM is not enough: more than four CTAs per SM
// are not launched ahead of the kernel before (448 blocks, Q4_K, a feed-forward of 4096 x 14336 with 4 tokens 61.4 us with one split, 65.3 with two), except
// for five to eight tokens, whose longer reads of x take more warps to hide (8 tokens 68.5 / 65.2). A slice keeps at least two stages.
template <int TYPE, int NT>
int packed_splits(int M, int N, int pairs, bool tma) {
  const int tiles = (N + kRows - 1) / kRows, ctas = TYPE == gguf::kTypeQ4K && NT > 1 ? 4 * kNumSMs : tma ? 3 * kNumSMs / 2 : 2 * kNumSMs;
  int splits = 1;
  const auto load = [&](int n) { return static_cast<double>((tiles * n + kNumSMs - 1) / kNumSMs) / n; };      // of the fullest SM
  const auto more = [&] {
    if (tiles * splits < ctas) return true;
    if (!tma || tiles * splits >= 4 * kNumSMs) return false;
    return load(2 * splits) < (TYPE == gguf::kTypeQ4K && NT == 1 && M > 4 ? 0.9 : 0.85) * load(splits) || pairs >= 24 * splits || (NT == 4 && splits == 1 && load(2) <= load(1));
  };
  while (splits < kMaxSplit && pairs >= 4 * splits && more()) splits *= 2;
  while (splits < kMaxSplit && packed_smem<TYPE, NT>(pairs, splits) > kMostSmem<TYPE>) splits *= 2;      // a very long K
  return splits;
}

template <int TYPE, int NT>
int launch_packed(PackedArgs a, Status* status, cudaStream_t stream) {
  CUtensorMap tmap{};
  constexpr int kRow = Pack<TYPE>::kRowStride;
  const int64_t row_bytes = static_cast<int64_t>(a.blocks_per_row) * Pack<TYPE>::kBytes;
  if (a.tma && !make_tmap_2d(&tmap, CU_TENSOR_MAP_DATA_TYPE_UINT32, 4, a.wq, a.N, row_bytes / 4, row_bytes, 16, kRow / 4, CU_TENSOR_MAP_SWIZZLE_NONE)) a.tma = 0;
  const int tiles = (a.N + kRows - 1) / kRows;
  a.splits = packed_splits<TYPE, NT>(a.M, a.N, a.pairs, a.tma != 0);
  const int smem = std::max(packed_smem<TYPE, NT>(a.pairs, a.splits), (a.splits - 1) * kQThreads * NT * 4 * 4);
  if (smem > kMostSmem<TYPE>) return -kTooLarge;
  auto kern = packed_gemm_kernel<TYPE, NT>;
  static DeviceOnce attr_once;
  if (const int rc = attr_once.max_smem(kern, kMostSmem<TYPE>)) return rc;
  const cudaError_t e = launch_cluster(kern, dim3(static_cast<unsigned>(tiles * a.splits)), dim3(kQThreads), a.splits, smem, stream, tmap, a, status);
  return e != cudaSuccess ? cuda_rc(e) : last_launch_rc();
}

template <int TYPE>
int launch_packed_type(const PackedArgs& a, Status* status, cudaStream_t stream) {
  if (a.M <= 8) return launch_packed<TYPE, 1>(a, status, stream);
  if (a.M <= 16) return launch_packed<TYPE, 2>(a, status, stream);
  return launch_packed<TYPE, 4>(a, status, stream);
}

}  // namespace
}  // namespace b2

using namespace b2;

extern "C" int b2_dequant_gguf(const void* wq, int ggml_type, void* out_bf16, int64_t n_elems, cudaStream_t stream) {
  if (n_elems <= 0) return 0;
  if (n_elems % gguf::kQK != 0 || gguf::block_bytes(ggml_type) == 0) return -kBadArgument;
  if ((reinterpret_cast<uintptr_t>(wq) & 15) == 0 && (reinterpret_cast<uintptr_t>(out_bf16) & 15) == 0) {
    const int64_t pairs = n_elems / 64;
    dequant64_kernel<<<static_cast<unsigned>((pairs + 127) / 128), 128, 0, stream>>>(static_cast<const uint8_t*>(wq), ggml_type,
                                                                                    static_cast<__nv_bfloat16*>(out_bf16), pairs);
    return last_launch_rc();
  }
  const int64_t groups = n_elems / 32;
  dequant_kernel<<<static_cast<unsigned>((groups + 127) / 128), 128, 0, stream>>>(static_cast<const uint8_t*>(wq), ggml_type,
                                                                                  static_cast<__nv_bfloat16*>(out_bf16), groups);
  return last_launch_rc();
}

extern "C" int b2_gemm_gguf_splits(int ggml_type, int M, int N, int K, int aligned) {
  const int blocks = K / gguf::kQK, pairs = (blocks + 1) / 2;
  const bool tma = aligned && static_cast<int64_t>(blocks) * gguf::block_bytes(ggml_type) % 16 == 0;
  const auto of = [&](auto type) {
    constexpr int T = decltype(type)::value;
    return M <= 8 ? packed_splits<T, 1>(M, N, pairs, tma) : M <= 16 ? packed_splits<T, 2>(M, N, pairs, tma) : packed_splits<T, 4>(M, N, pairs, tma);
  };
  return ggml_type == gguf::kTypeQ4K ? of(std::integral_constant<int, gguf::kTypeQ4K>{}) : of(std::integral_constant<int, gguf::kTypeQ6K>{});
}

extern "C" int b2_gemm_gguf(const void* x, const void* wq, int ggml_type, void* y, int M, int N, int K, b2::Status* status,
                            cudaStream_t stream) {
  if (M <= 0 || N <= 0) return 0;
  if (K <= 0 || K % gguf::kQK != 0 || gguf::block_bytes(ggml_type) == 0) return -kBadArgument;
  if ((reinterpret_cast<uintptr_t>(x) & 15) != 0) return -kBadArgument;
  PackedArgs a{};
  a.wq = static_cast<const uint8_t*>(wq);
  a.N = N;
  a.K = K;
  a.blocks_per_row = K / gguf::kQK;
  a.pairs = (a.blocks_per_row + 1) / 2;
  const int64_t row_bytes = static_cast<int64_t>(a.blocks_per_row) * gguf::block_bytes(ggml_type);
  a.tma = (reinterpret_cast<uintptr_t>(wq) & 15) == 0 && row_bytes % 16 == 0 ? 1 : 0;
  for (int m = 0, most = kMaxTokens; m < M;) {      // the weights are read once for every 32 tokens (fewer if the sums of a very long K do not fit)
    a.x = static_cast<const __nv_bfloat16*>(x) + static_cast<int64_t>(m) * K;
    a.y = static_cast<__nv_bfloat16*>(y) + static_cast<int64_t>(m) * N;
    a.M = std::min(M - m, most);
    const int rc = ggml_type == gguf::kTypeQ4K ? launch_packed_type<gguf::kTypeQ4K>(a, status, stream) : launch_packed_type<gguf::kTypeQ6K>(a, status, stream);
    if (rc == -kTooLarge && most > 8) {
      most /= 2;
      continue;
    }
    if (rc) return rc;
    m += a.M;
  }
  return 0;
}
