// Token sampling: greedy argmax and temperature / top-k / top-p sampling over a [rows, vocab] logits matrix.
//
// Selection of the k-th largest logit is an MSB-first radix select on order-preserving integer keys: the
// GPU form of the quick-select `partition(span, k)` the reference offers on the CPU
// (stdlib/src/builtin/sort.mojo:373-506 - first k elements = k largest, unordered). Top-p reuses the same
// digit walk with probability mass instead of counts. The uniform draw is Philox4x32-10 keyed by
// (seed; step, row), replacing the reference's closed host RNG (stdlib/src/random/random.mojo:32-92).
// bf16 rows (what the models produce) go to a cluster of CTAs that reads a row once into shared memory; the digit walk, one CTA
// per row with the row in L2 across passes, serves f32 rows and bf16 rows too long for that.
#include <algorithm>
#include <cstdint>
#include <cuda_bf16.h>
#include "b2/api.h"
#include "b2/launch.h"
#include "b2/ptx.cuh"
#include "b2/vec.cuh"

namespace b2 {
namespace {

constexpr int kThreads = 1024;

template <bool BF16>
__device__ __forceinline__ float load_logit(const void* row, int i) {
  if (BF16) return __bfloat162float(static_cast<const __nv_bfloat16*>(row)[i]);
  return static_cast<const float*>(row)[i];
}
__device__ __forceinline__ uint32_t float_key(float x) {
  const uint32_t u = __float_as_uint(x);
  return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}

struct Philox {
  uint32_t c[4];
  uint32_t k[2];
  __device__ __forceinline__ void round() {
    const uint32_t M0 = 0xD2511F53u, M1 = 0xCD9E8D57u;
    const uint32_t hi0 = __umulhi(M0, c[0]), lo0 = M0 * c[0];
    const uint32_t hi1 = __umulhi(M1, c[2]), lo1 = M1 * c[2];
    const uint32_t n0 = hi1 ^ c[1] ^ k[0], n1 = lo1, n2 = hi0 ^ c[3] ^ k[1], n3 = lo0;
    c[0] = n0; c[1] = n1; c[2] = n2; c[3] = n3;
  }
  __device__ __forceinline__ void run10() {
#pragma unroll
    for (int i = 0; i < 10; ++i) {
      round();
      if (i < 9) { k[0] += 0x9E3779B9u; k[1] += 0xBB67AE85u; }
    }
  }
};
__device__ __forceinline__ float philox_uniform(uint64_t seed, uint64_t step, uint32_t row) {
  Philox p;
  p.c[0] = static_cast<uint32_t>(step);
  p.c[1] = static_cast<uint32_t>(step >> 32);
  p.c[2] = row;
  p.c[3] = 0;
  p.k[0] = static_cast<uint32_t>(seed);
  p.k[1] = static_cast<uint32_t>(seed >> 32);
  p.run10();
  return static_cast<float>(p.c[0] >> 8) * (1.0f / 16777216.0f);
}

struct ArgMax {
  float v;
  int i;
};
__device__ __forceinline__ ArgMax better(ArgMax a, ArgMax b) {
  return (b.v > a.v || (b.v == a.v && b.i < a.i)) ? b : a;
}
template <bool BF16>
__device__ ArgMax block_argmax(const void* row, int vocab, ArgMax* scratch) {
  ArgMax best{-INFINITY, 0x7fffffff};
  for (int i = threadIdx.x; i < vocab; i += blockDim.x) {
    const float x = load_logit<BF16>(row, i);
    if (x > best.v || (x == best.v && i < best.i)) best = ArgMax{x, i};
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    ArgMax other{__shfl_xor_sync(0xffffffffu, best.v, o), __shfl_xor_sync(0xffffffffu, best.i, o)};
    best = better(best, other);
  }
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  if (lane == 0) scratch[warp] = best;
  __syncthreads();
  if (warp == 0) {
    ArgMax b = lane < nw ? scratch[lane] : ArgMax{-INFINITY, 0x7fffffff};
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      ArgMax other{__shfl_xor_sync(0xffffffffu, b.v, o), __shfl_xor_sync(0xffffffffu, b.i, o)};
      b = better(b, other);
    }
    if (lane == 0) scratch[32] = b;
  }
  __syncthreads();
  const ArgMax r = scratch[32];
  __syncthreads();
  if (r.i == 0x7fffffff) return ArgMax{r.v, 0};  // all -inf / NaN row
  return r;
}

// Visit every logit of a row with its index: 16-byte loads (8 bf16 / 4 f32 per load, consecutive threads on
// consecutive vectors) when the row is 16-byte aligned, scalar loads otherwise and for the tail.
template <bool BF16, class F>
__device__ __forceinline__ void for_each_logit(const void* row, int vocab, F&& f) {
  constexpr int V = BF16 ? 8 : 4;
  const bool aligned = (reinterpret_cast<uintptr_t>(row) & 15u) == 0;
  const int nvec = aligned ? vocab / V : 0;
  const uint4* rv = static_cast<const uint4*>(row);
  for (int v = threadIdx.x; v < nvec; v += blockDim.x) {
    const uint4 q = rv[v];
    if (BF16) {
      float x[8];
      bf16x8_to_f32(q, x);
#pragma unroll
      for (int j = 0; j < 8; ++j) f(x[j], v * 8 + j);
    } else {
      f(__uint_as_float(q.x), v * 4 + 0);
      f(__uint_as_float(q.y), v * 4 + 1);
      f(__uint_as_float(q.z), v * 4 + 2);
      f(__uint_as_float(q.w), v * 4 + 3);
    }
  }
  for (int i = nvec * V + threadIdx.x; i < vocab; i += blockDim.x) f(load_logit<BF16>(row, i), i);
}

constexpr int kWarps = kThreads / 32;

// MSB-first radix walk. MASS = false: find the key of the `want`-th largest element (counts).
// MASS = true: find the key at which the mass of strictly larger keys first reaches `want`.
// Only keys >= floor_key participate. Returns the selected key.
// Every warp accumulates into its own 256-bin histogram (logits crowd into a few exponent buckets: one shared
// histogram serialises all 1024 threads on the same two or three words), and the warps' histograms are added up
// afterwards. bf16 logits have 16 significant key bits, so their walk is two digits long instead of four.
template <bool BF16, bool MASS>
__device__ uint32_t radix_select(const void* row, int vocab, float want, uint32_t floor_key, float mx, float inv_t,
                                 float* hist /* [kWarps + 1][256] */, float* bcast) {
  uint32_t prefix = 0, mask = 0;
  const int warp = threadIdx.x >> 5;
  float* mine = hist + warp * 256;
  float* total = hist + kWarps * 256;
  constexpr int kLastPass = BF16 ? 2 : 0;
  for (int pass = 3; pass >= kLastPass; --pass) {
    for (int b = threadIdx.x; b < (kWarps + 1) * 256; b += blockDim.x) hist[b] = 0.0f;
    __syncthreads();
    const int shift = pass * 8;
    for_each_logit<BF16>(row, vocab, [&](float x, int) {
      const uint32_t key = float_key(x);
      if (key >= floor_key && (key & mask) == prefix) {
        const float w = MASS ? ptx::ex2((x - mx) * inv_t) : 1.0f;
        atomicAdd(&mine[(key >> shift) & 0xffu], w);
      }
    });
    __syncthreads();
    if (threadIdx.x < 256) {
      float acc = 0.0f;
#pragma unroll 4
      for (int w2 = 0; w2 < kWarps; ++w2) acc += hist[w2 * 256 + threadIdx.x];
      total[threadIdx.x] = acc;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
      float acc = 0.0f;
      int b = 255;
      for (; b > 0; --b) {
        if (acc + total[b] >= want) break;
        acc += total[b];
      }
      bcast[0] = acc;
      bcast[1] = __int_as_float(b);
    }
    __syncthreads();
    want -= bcast[0];
    const uint32_t b = static_cast<uint32_t>(__float_as_int(bcast[1]));
    prefix |= b << shift;
    mask |= 0xffu << shift;
    __syncthreads();
  }
  return prefix;
}

template <bool BF16>
__global__ void __launch_bounds__(kThreads) sample_kernel(const void* logits, int64_t* ids, const float* temperature,
                                                           const int32_t* top_k, const float* top_p,
                                                           const float* uniforms, uint64_t seed, uint64_t step,
                                                           int vocab, int64_t row_stride) {
  ptx::grid_dep_sync();
  __shared__ ArgMax scratch[33];
  __shared__ float fscratch[33];
  __shared__ float hist[(kWarps + 1) * 256];
  __shared__ float bcast[2];
  __shared__ float sums[kThreads];
  const int row = blockIdx.x;
  const void* base = static_cast<const char*>(logits) + static_cast<int64_t>(row) * row_stride * (BF16 ? 2 : 4);
  const float temp = temperature != nullptr ? temperature[row] : 1.0f;
  const ArgMax best = block_argmax<BF16>(base, vocab, scratch);
  if (temp <= 0.0f) {
    if (threadIdx.x == 0) ids[row] = best.i;
    return;
  }
  const float mx = best.v;
  const float inv_t = ptx::kLog2e / temp;  // exp((x - mx)/T) = 2^((x - mx) * log2e / T)
  const int k = top_k != nullptr ? top_k[row] : 0;
  const float pp = top_p != nullptr ? top_p[row] : 1.0f;

  uint32_t floor_key = 0;
  if (k > 0 && k < vocab)
    floor_key = radix_select<BF16, false>(base, vocab, static_cast<float>(k), 0u, mx, inv_t, hist, bcast);
  if (pp < 1.0f) {
    float z = 0.0f;
    for_each_logit<BF16>(base, vocab, [&](float x, int) {
      if (float_key(x) >= floor_key) z += ptx::ex2((x - mx) * inv_t);
    });
    z = block_sum(z, fscratch);
    const uint32_t pkey = radix_select<BF16, true>(base, vocab, pp * z, floor_key, mx, inv_t, hist, bcast);
    floor_key = max(floor_key, pkey);
  }
  // inverse-CDF draw in index order over the kept set
  const int chunk = (vocab + blockDim.x - 1) / blockDim.x;
  const int i0 = threadIdx.x * chunk, i1 = min(vocab, i0 + chunk);
  float local = 0.0f;
  for (int i = i0; i < i1; ++i) {
    const float x = load_logit<BF16>(base, i);
    if (float_key(x) >= floor_key) local += ptx::ex2((x - mx) * inv_t);
  }
  sums[threadIdx.x] = local;
  __syncthreads();
  // inclusive scan (Hillis-Steele over 1024 entries)
  for (int o = 1; o < kThreads; o <<= 1) {
    const float add = threadIdx.x >= o ? sums[threadIdx.x - o] : 0.0f;
    __syncthreads();
    sums[threadIdx.x] += add;
    __syncthreads();
  }
  const float total = sums[kThreads - 1];
  const float u = uniforms != nullptr ? uniforms[row] : philox_uniform(seed, step, static_cast<uint32_t>(row));
  const float target = u * total;
  const float before = threadIdx.x > 0 ? sums[threadIdx.x - 1] : 0.0f;
  const float after = sums[threadIdx.x];
  if (threadIdx.x == 0) bcast[0] = __int_as_float(-1);
  __syncthreads();
  if (local > 0.0f && before <= target && target < after) {
    float acc = before;
    int pick = -1;
    for (int i = i0; i < i1; ++i) {
      const float x = load_logit<BF16>(base, i);
      if (float_key(x) >= floor_key) {
        acc += ptx::ex2((x - mx) * inv_t);
        pick = i;
        if (acc > target) break;
      }
    }
    bcast[0] = __int_as_float(pick);
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    const int pick = __float_as_int(bcast[0]);
    ids[row] = pick >= 0 ? pick : best.i;  // rounding fell off the end: the mode is always in the kept set
  }
}

// ------------------------------------------------------------------------------------------------------
// Rows spread over a cluster of CTAs
// ------------------------------------------------------------------------------------------------------
// A row of 128256 logits is 256 KB: one CTA cannot pull it in faster than about 100 GB/s, and a decode step has few rows. A
// cluster of up to eight CTAs shares a row, so that 148 SMs have work from 37 rows on.
constexpr int kRowThreads = 512;
constexpr int kRowWarps = kRowThreads / 32;
constexpr int kMaxCluster = 8;

// CTAs per row: the widest cluster that keeps the launch within `ctas` thread blocks and gives each 2048 logits. Shorter runs, and more
// blocks than SMs, cost more in exchanges than they save in reading (the choice among 1000 logits, 64 rows: 2.2 us with one CTA a row, 3.3
// with four; among 128256, 64 rows: 5.7 us with two, 6.8 with four).
int cluster_for(int rows, int vocab, int ctas) {
  int c = kMaxCluster;
  while (c > 1 && (rows > ctas / c || vocab < 2048 * c)) c >>= 1;
  return c;
}

// The kernel has called `cluster_started`.
__device__ __forceinline__ ArgMax cluster_argmax(ArgMax best, ArgMax* scratch /* [kRowWarps] */, ArgMax* all /* [kMaxCluster] */, int rank, int cluster) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1)
    best = better(best, ArgMax{__shfl_xor_sync(0xffffffffu, best.v, o), __shfl_xor_sync(0xffffffffu, best.i, o)});
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (lane == 0) scratch[warp] = best;
  __syncthreads();
  ptx::cluster_wait_started();
  if (warp == 0) {
    best = lane < kRowWarps ? scratch[lane] : ArgMax{-INFINITY, 0x7fffffff};
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
      best = better(best, ArgMax{__shfl_xor_sync(0xffffffffu, best.v, o), __shfl_xor_sync(0xffffffffu, best.i, o)});
    if (lane < cluster) {
      const uint32_t to = ptx::mapa(ptx::smem_u32(&all[rank]), lane);
      ptx::st_cluster_f32(to, best.v);
      ptx::st_cluster_u32(to + 4, static_cast<uint32_t>(best.i));
    }
  }
  ptx::cluster_sync();
  best = all[0];
  for (int q = 1; q < cluster; ++q) best = better(best, all[q]);
  if (best.i == 0x7fffffff) best.i = 0;      // nothing but -inf and NaN
  return best;
}

// Greedy choice. Bound by the latency of one pass over the row: 16-byte loads, four in flight per thread. 1 x 32000 bf16:
// 9.7 us with one CTA and 2-byte loads.
template <bool BF16>
__global__ void __launch_bounds__(kRowThreads) argmax_kernel(const void* logits, int64_t* ids, float* max_out, int vocab, int64_t row_stride, int cluster) {
  ptx::cluster_started();
  ptx::grid_dep_sync();
  __shared__ ArgMax scratch[kRowWarps], all[kMaxCluster];
  constexpr int V = BF16 ? 8 : 4;
  const int rank = blockIdx.x % cluster, row = blockIdx.x / cluster;
  const char* base = static_cast<const char*>(logits) + static_cast<int64_t>(row) * row_stride * (BF16 ? 2 : 4);
  ArgMax best{-INFINITY, 0x7fffffff};
  auto see = [&](float x, int i) {
    if (x > best.v || (x == best.v && i < best.i)) best = ArgMax{x, i};
  };
  // single logits up to the first 16-byte boundary and behind the last, vectors between them
  const int head = min(vocab, static_cast<int>((16u - (reinterpret_cast<uintptr_t>(base) & 15u)) & 15u) / (BF16 ? 2 : 4));
  const int nvec = (vocab - head) / V;
  const uint4* rv = reinterpret_cast<const uint4*>(base + head * (BF16 ? 2 : 4));
  const int stride = cluster * kRowThreads;
  auto use = [&](const uint4& q, int v) {
    if (BF16) {
      float x[8];
      bf16x8_to_f32(q, x);
#pragma unroll
      for (int j = 0; j < 8; ++j) see(x[j], head + v * 8 + j);
    } else {
      see(__uint_as_float(q.x), head + v * 4);
      see(__uint_as_float(q.y), head + v * 4 + 1);
      see(__uint_as_float(q.z), head + v * 4 + 2);
      see(__uint_as_float(q.w), head + v * 4 + 3);
    }
  };
  for (int v = rank * kRowThreads + threadIdx.x; v < nvec; v += 4 * stride) {
    uint4 q[4];
#pragma unroll
    for (int j = 0; j < 4; ++j)
      if (v + j * stride < nvec) q[j] = rv[v + j * stride];
#pragma unroll
    for (int j = 0; j < 4; ++j)
      if (v + j * stride < nvec) use(q[j], v + j * stride);
  }
  if (rank == 0) {
    const int i = static_cast<int>(threadIdx.x) < head ? threadIdx.x : nvec * V + threadIdx.x;      // fewer than V on either side
    if (i < vocab) see(load_logit<BF16>(base, i), i);
  }
  best = cluster_argmax(best, scratch, all, rank, cluster);
  if (rank == 0 && threadIdx.x == 0) {
    ids[row] = best.i;
    if (max_out != nullptr) max_out[row] = best.v;
  }
}

// Sampling from a bf16 row. The row is read from memory once, into the cluster's shared memory; everything after that works on
// the copy. A bf16 logit has 16 significant bits, so equal values are counted, not sorted: a histogram over the distinct values
// from the maximum down gives the k-th largest by counts, and probability mass as count x weight, with no floating-point
// atomics. Values below a bound that provably keeps the answer above it never enter the histogram (the atomics are what it
// costs). What bounds it is the chain of passes over the copy and of exchanges between its CTAs, not the 16 MB. Measured, 64 rows x 128256,
// mixed top-k / top-p: 22.9 us a call, against 213 us for the digit walk with one CTA per row. 26.4 with bins by way of keys, a pass of its own
// for the sum of weights, the draw's scans one after the other and each row's parameters read behind the row.
constexpr int kBins = 8192;                 // distinct values from the maximum down
constexpr int kChunk = 4 * kRowThreads;     // bins that are summed over the cluster at once
constexpr int kMaxSegs = 1024;              // (round, warp) runs of a CTA's slice in index order: 64 rounds of 4096 logits
// Keys of |x| < 2^-20 share one place on the line of bins, so that the bins reach from the maximum to large negative values.
constexpr uint32_t kGapLo = 0x4A80u, kGapHi = 0xB580u;

__device__ __forceinline__ uint32_t key16(uint32_t bits) { return (bits & 0x8000u) ? (~bits & 0xffffu) : (bits | 0x8000u); }
__device__ __forceinline__ int line_of(uint32_t key) {
  return static_cast<int>(key >= kGapHi ? key - kGapHi + kGapLo + 1u : key >= kGapLo ? kGapLo : key);
}
__device__ __forceinline__ uint32_t key_at(int line) {      // not for the gap's place
  const uint32_t l = static_cast<uint32_t>(line);
  return l > kGapLo ? l - kGapLo - 1u + kGapHi : l;
}
__device__ __forceinline__ float value_of(uint32_t key) {
  return __uint_as_float(((key & 0x8000u) ? (key & 0x7fffu) : (~key & 0xffffu)) << 16);
}

struct RowShared {
  float vmax[kMaxCluster];
  uint32_t nan[kMaxCluster];      // whether a slice holds one
  uint32_t where[kMaxCluster];    // first place of the maximum in a slice
  float seg[kMaxSegs];
  float part[2][kMaxCluster];      // sums handed from rank to rank, alternating
  float slice_mass[kMaxCluster];
  float warp_f[kRowWarps + 1];
  int warp_i[kRowWarps + 1];
  float found_mass;
  int found;
};

__device__ __forceinline__ float row_block_sum(float v, RowShared& sh) {
  v = warp_sum(v);
  if ((threadIdx.x & 31) == 0) sh.warp_f[threadIdx.x >> 5] = v;
  __syncthreads();
  float t = 0.0f;
#pragma unroll
  for (int w = 0; w < kRowWarps; ++w) t += sh.warp_f[w];
  __syncthreads();
  return t;
}
// Sum of the CTAs' numbers over the cluster; every thread of every CTA gets the same bits.
__device__ __forceinline__ float row_cluster_total(float v, RowShared& sh, int rank, int cluster, int& turn) {
  if (static_cast<int>(threadIdx.x) < cluster) ptx::st_cluster_f32(ptx::mapa(ptx::smem_u32(&sh.part[turn][rank]), threadIdx.x), v);
  ptx::cluster_sync();
  float t = 0.0f;
  for (int q = 0; q < cluster; ++q) t += sh.part[turn][q];
  turn ^= 1;
  return t;
}
__device__ __forceinline__ float row_cluster_sum(float v, RowShared& sh, int rank, int cluster, int& turn) {
  return row_cluster_total(row_block_sum(v, sh), sh, rank, cluster, turn);
}

__global__ void __launch_bounds__(kRowThreads, 2) sample_row_kernel(const __nv_bfloat16* logits, int64_t* ids, const float* temperature, const int32_t* top_k,
                                                                    const float* top_p, const float* uniforms, uint64_t seed, uint64_t step, int vocab,
                                                                    int64_t row_stride, int cluster, int slice_vecs) {
  ptx::cluster_started();
  ptx::grid_dep_sync();
  extern __shared__ uint4 row_smem[];
  __shared__ RowShared sh;
  uint4* vals = row_smem;
  uint32_t* hist = reinterpret_cast<uint32_t*>(row_smem + slice_vecs);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int rank = blockIdx.x % cluster, row = blockIdx.x / cluster;
  const __nv_bfloat16* base = logits + static_cast<int64_t>(row) * row_stride;
  const bool aligned = (reinterpret_cast<uintptr_t>(base) & 15u) == 0;
  // asked for ahead of the row: their latency would stand between it and the histogram
  const float temp = temperature != nullptr ? temperature[row] : 1.0f, pp = top_p != nullptr ? top_p[row] : 1.0f;
  const int k = top_k != nullptr ? top_k[row] : 0;
  const int total_vecs = (vocab + 7) / 8, v0 = rank * slice_vecs;
  const int nv = max(0, min(slice_vecs, total_vecs - v0));

  // ---- the row into shared memory, its maximum on the way (two at a time; where it stands is looked up only if needed) ----
  __nv_bfloat162 top = __halves2bfloat162(__ushort_as_bfloat16(0xff80), __ushort_as_bfloat16(0xff80)), seen_nan = top;
  auto fetch = [&](int v) {
    const int i0 = (v0 + v) * 8;
    if (aligned && i0 + 8 <= vocab) return ptx::ld_nc_v4(base + i0);
    uint32_t w[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const uint32_t lo = i0 + 2 * j < vocab ? __bfloat16_as_ushort(base[i0 + 2 * j]) : 0xff80u;      // past the end: -inf
      const uint32_t hi = i0 + 2 * j + 1 < vocab ? __bfloat16_as_ushort(base[i0 + 2 * j + 1]) : 0xff80u;
      w[j] = lo | (hi << 16);
    }
    return make_uint4(w[0], w[1], w[2], w[3]);
  };
  auto take = [&](const uint4& q, int v) {
    vals[v] = q;
    const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&q);
    top = __hmax2(top, __hmax2(__hmax2(h[0], h[1]), __hmax2(h[2], h[3])));
    seen_nan = __hmax2_nan(seen_nan, __hmax2_nan(__hmax2_nan(h[0], h[1]), __hmax2_nan(h[2], h[3])));
  };
  // eight loads at once, also where the slice ends in between: one after the other each would wait for memory by itself
  for (int lv = tid; lv < nv; lv += 8 * kRowThreads) {
    uint4 q[8];
#pragma unroll
    for (int j = 0; j < 8; ++j)
      if (lv + j * kRowThreads < nv) q[j] = fetch(lv + j * kRowThreads);
#pragma unroll
    for (int j = 0; j < 8; ++j)
      if (lv + j * kRowThreads < nv) take(q[j], lv + j * kRowThreads);
  }
  const uint32_t my_max = max(key16(__bfloat16_as_ushort(top.x)), key16(__bfloat16_as_ushort(top.y)));
  for (int b = tid; b < kBins / 4; b += kRowThreads) reinterpret_cast<uint4*>(hist)[b] = make_uint4(0, 0, 0, 0);
  {
    const float m = warp_max(fmaxf(__bfloat162float(top.x), __bfloat162float(top.y)));
    const bool any = __any_sync(0xffffffffu, __hisnan(seen_nan.x) || __hisnan(seen_nan.y));
    if (lane == 0) {
      sh.warp_f[warp] = m;
      sh.warp_i[warp] = any;
    }
    __syncthreads();
    ptx::cluster_wait_started();
    if (warp == 0) {
      const float t = warp_max(lane < kRowWarps ? sh.warp_f[lane] : -INFINITY);
      const bool n = __any_sync(0xffffffffu, lane < kRowWarps && sh.warp_i[lane] != 0);
      if (lane < cluster) {
        ptx::st_cluster_f32(ptx::mapa(ptx::smem_u32(&sh.vmax[rank]), lane), t);
        ptx::st_cluster_u32(ptx::mapa(ptx::smem_u32(&sh.nan[rank]), lane), n ? 1u : 0u);
      }
    }
    ptx::cluster_sync();
  }
  float mx = sh.vmax[0];
  bool careful = sh.nan[0] != 0;      // a NaN somewhere: no vector is passed over for its maximum
  for (int q = 1; q < cluster; ++q) {
    mx = fmaxf(mx, sh.vmax[q]);
    careful = careful || sh.nan[q] != 0;
  }
  // First place of the maximum in the row. Every CTA of the cluster calls it or none; the first one stores the id.
  auto store_mode = [&]() {
    uint32_t at = 0xffffffffu;
    for (int v = tid; v < nv && at == 0xffffffffu; v += kRowThreads) {
      float x[8];
      bf16x8_to_f32(vals[v], x);
#pragma unroll
      for (int j = 7; j >= 0; --j)
        if (x[j] == mx) at = static_cast<uint32_t>((v0 + v) * 8 + j);
    }
    at = __reduce_min_sync(0xffffffffu, at);
    __syncthreads();
    if (lane == 0) sh.warp_i[warp] = static_cast<int>(at);
    __syncthreads();
    if (warp == 0) {
      const uint32_t t = __reduce_min_sync(0xffffffffu, lane < kRowWarps ? static_cast<uint32_t>(sh.warp_i[lane]) : 0xffffffffu);
      if (lane == 0) ptx::st_cluster_u32(ptx::mapa(ptx::smem_u32(&sh.where[rank]), 0), t);
    }
    ptx::cluster_sync();
    if (rank == 0 && tid == 0) {
      uint32_t t = sh.where[0];
      for (int q = 1; q < cluster; ++q) t = min(t, sh.where[q]);
      ids[row] = t < static_cast<uint32_t>(vocab) ? t : 0;      // nothing but NaN: 0
    }
  };
  if (temp <= 0.0f || isinf(mx)) {      // greedy; or a maximum that no finite weight can be taken against
    store_mode();
    return;
  }
  const float inv_t = ptx::kLog2e / temp;      // exp((x - mx) / T) = 2^((x - mx) log2e / T)
  const bool by_count = k > 0 && k < vocab, by_mass = pp < 1.0f;
  auto weight = [&](float x) { return ptx::ex2((x - mx) * inv_t); };
  // Whether a vector may hold a logit with a key of at least `key`.
  auto reaches = [&](const uint4& q, uint32_t key) {
    const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&q);
    const __nv_bfloat162 m = __hmax2(__hmax2(h[0], h[1]), __hmax2(h[2], h[3]));
    return careful || max(key16(__bfloat16_as_ushort(m.x)), key16(__bfloat16_as_ushort(m.y))) >= key;
  };
  auto each = [&](uint32_t least, auto&& f) {      // the logits of this CTA's slice, without vectors that stay below `least`
    for (int v = tid; v < nv; v += kRowThreads) {
      const uint4 q = vals[v];
      if (!reaches(q, least)) continue;
      const uint32_t w[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        f(w[j] & 0xffffu);
        f(w[j] >> 16);
      }
    }
  };

  uint32_t floor_key = 0;
  if (by_count || by_mass) {
    // ---- histogram of the values that may decide ----
    uint32_t cut = 0;
    float z = 0.0f;
    if (by_count) {
      // k threads whose own maxima reach a value prove that the k-th largest logit does: the largest such value. (128 groups of four threads,
      // which a warp can rank without a barrier, give a lower one, and what it lets into the histogram costs more: 18 -> 20 us for 64 rows.)
      if (k <= kRowThreads) {
#pragma unroll 1
        for (uint32_t bit = 0x8000u; bit; bit >>= 1)
          if (__syncthreads_count(my_max >= (cut | bit)) >= k) cut |= bit;
      }
    } else {
      // logits whose weight is below (1 - p) / vocab together weigh less than (1 - p) times the maximum's weight alone: the
      // mass p is reached above them. (The sum of weights first, for a bound by that: a third of the logits, and 2 us more for 64 rows.)
      const float x = mx + ptx::lg2((1.0f - pp) / static_cast<float>(vocab)) / inv_t;
      const uint32_t bits = __float_as_uint(x) >> 16;      // towards zero: below x where x < 0 needs one more step
      cut = x == x ? key16(bits) : 0u;
      if (cut > 0) --cut;
    }
    const int top_line = line_of(key16(__float_as_uint(mx) >> 16));
    // Bins of a logit straight from its bits, as top_line - line_of(key16(bits)) gives them: positive ones up to the gap's place, negative ones
    // from there on. Bins behind that of `cut` are left out; so is a NaN, whose bin is negative or far behind.
    constexpr int kAcross = static_cast<int>(kGapHi - kGapLo) - 1;
    const int gap_bin = top_line - static_cast<int>(kGapLo), above = top_line - 0x8000 + kAcross, below = 0xffff - top_line;
    const uint32_t bins = static_cast<uint32_t>(max(0, min(top_line - line_of(cut) + 1, kBins)));      // none where a mass below zero puts the cut above the maximum
    const auto count = [&](uint32_t bits) {
      const int pos = min(above - static_cast<int>(bits), gap_bin), neg = max(static_cast<int>(bits) - below, gap_bin);
      const uint32_t b = static_cast<uint32_t>(bits & 0x8000u ? neg : pos);
      if (b < bins) atomicAdd(&hist[b], 1u);
    };
    for (int v = tid; v < nv; v += kRowThreads) {
      const uint4 q = vals[v];
      if (!by_count) {
        float x[8];
        bf16x8_to_f32(q, x);
#pragma unroll
        for (int j = 0; j < 8; ++j) x[j] = weight(x[j]);
        z += ((x[0] + x[1]) + (x[2] + x[3])) + ((x[4] + x[5]) + (x[6] + x[7]));
      }
      if (!reaches(q, cut)) continue;
      const uint32_t w[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        count(w[j] & 0xffffu);
        count(w[j] >> 16);
      }
    }
    if (!by_count) z = row_block_sum(z, sh);
    int turn = 0;
    z = row_cluster_total(z, sh, rank, cluster, turn);      // its cluster barrier also completes the histograms

    // First bin at which the running count (or mass) reaches `want`; -1: not among the bins. `mass` gets the mass up to and
    // with that bin. Every CTA of the cluster adds up the same numbers in the same order.
    auto find = [&](bool mass_search, float want, float& mass) {
      int carry_n = 0;
      float carry_m = 0.0f;
      if (tid == 0) sh.found = -1;
      for (int c0 = 0; c0 < kBins; c0 += kChunk) {
        const int b0 = c0 + tid * 4;
        uint32_t n[4] = {0, 0, 0, 0};
        for (int q = 0; q < cluster; ++q) {
          const uint4 h = ptx::ld_cluster_v4(ptx::mapa(ptx::smem_u32(hist + b0), q));
          n[0] += h.x; n[1] += h.y; n[2] += h.z; n[3] += h.w;
        }
        float m[4];
        int cn[4];
        int sn = 0;
        float sm = 0.0f;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const int line = top_line - (b0 + j);
          const float w = n[j] == 0 ? 0.0f : weight(line == static_cast<int>(kGapLo) ? 0.0f : value_of(key_at(line)));
          sn += static_cast<int>(n[j]);
          sm = fmaf(static_cast<float>(n[j]), w, sm);
          cn[j] = sn;
          m[j] = sm;
        }
        int in = sn;
        float im = sm;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const int pn = __shfl_up_sync(0xffffffffu, in, o);
          const float pm = __shfl_up_sync(0xffffffffu, im, o);
          if (lane >= o) { in += pn; im += pm; }
        }
        if (lane == 31) { sh.warp_i[warp] = in; sh.warp_f[warp] = im; }
        int en = __shfl_up_sync(0xffffffffu, in, 1);
        float em = __shfl_up_sync(0xffffffffu, im, 1);
        if (lane == 0) { en = 0; em = 0.0f; }
        __syncthreads();
        int bn = carry_n;
        float bm = carry_m;
        for (int w = 0; w < warp; ++w) { bn += sh.warp_i[w]; bm += sh.warp_f[w]; }
        bn += en;
        bm += em;
        bool before = mass_search ? bm >= want : bn >= static_cast<int>(want);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const bool now = mass_search ? bm + m[j] >= want : bn + cn[j] >= static_cast<int>(want);
          if (now && !before && n[j] != 0) {
            // rounding may let two neighbours claim the crossing: the smaller bin has it
            atomicMin(reinterpret_cast<unsigned*>(&sh.found), static_cast<unsigned>(b0 + j));
          }
          before = before || now;
        }
        __syncthreads();
        const int hit = sh.found;
        if (hit >= b0 && hit < b0 + 4) sh.found_mass = bm + m[hit - b0];
        for (int w = 0; w < kRowWarps; ++w) { carry_n += sh.warp_i[w]; carry_m += sh.warp_f[w]; }
        __syncthreads();
        if (hit >= 0) {
          mass = sh.found_mass;
          return top_line - hit == static_cast<int>(kGapLo) ? -1 : hit;
        }
      }
      return -1;
    };
    // The same by bisection of the key over the copy, for what the bins do not resolve (values next to zero, or more distinct
    // ones than bins): the largest key that at least `want` of the count or mass lies at or above.
    auto bisect = [&](bool mass_search, float want) {
      uint32_t key = 0;
#pragma unroll 1
      for (uint32_t bit = 0x8000u; bit; bit >>= 1) {
        const uint32_t t = key | bit;
        float s = 0.0f;
        each(max(t, floor_key), [&](uint32_t bits) {
          const uint32_t kk = key16(bits);
          if (kk >= t && kk >= floor_key) s += mass_search ? weight(__uint_as_float(bits << 16)) : 1.0f;
        });
        if (row_cluster_sum(s, sh, rank, cluster, turn) >= want) key = t;
      }
      return key;
    };
    float mass = 0.0f;
    if (by_count) {
      const int b = find(false, static_cast<float>(k), mass);
      floor_key = b >= 0 ? key_at(top_line - b) : bisect(false, static_cast<float>(k));
      z = mass;
      if (by_mass && b < 0) {
        float s = 0.0f;
        each(floor_key, [&](uint32_t bits) {
          if (key16(bits) >= floor_key) s += weight(__uint_as_float(bits << 16));
        });
        z = row_cluster_sum(s, sh, rank, cluster, turn);
      }
    }
    if (by_mass) {
      const float want = pp * z;
      const int b = find(true, want, mass);
      floor_key = max(floor_key, b >= 0 ? key_at(top_line - b) : bisect(true, want));
    }
  }

  // ---- inverse-CDF draw in index order over the kept set ----
  // Round i of a warp covers 256 neighbouring logits; its weight goes to seg[i * warps + warp].
  const int32_t floor_line = static_cast<int32_t>((floor_key ^ 0x8000u) << 16);
  const auto kept = [&](uint32_t high) {      // key16(high >> 16) >= floor_key, as two operations on a logit in the upper half of a word
    const int32_t i = static_cast<int32_t>(high);
    return (i ^ ((i >> 31) & 0x7fff0000)) >= floor_line;
  };
  auto lane_weight = [&](int v) {
    float s = 0.0f;
    if (v < nv) {
      const uint4 q = vals[v];
      if (!reaches(q, floor_key)) return 0.0f;
      const uint32_t w[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        if (kept(w[j] << 16)) s += weight(__uint_as_float(w[j] << 16));
        if (kept(w[j] & 0xffff0000u)) s += weight(__uint_as_float(w[j] & 0xffff0000u));
      }
    }
    return s;
  };
  auto warp_scan = [&](float s) {
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const float p = __shfl_up_sync(0xffffffffu, s, o);
      if (lane >= o) s += p;
    }
    return s;
  };
  const int rounds = (nv + kRowThreads - 1) / kRowThreads, segs = rounds * kRowWarps;
  // four rounds' scans side by side: one after the other each would wait for five shuffles by itself; a warp that keeps nothing has none to do
  for (int i = 0; i < rounds; i += 4) {
    float s[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) s[j] = lane_weight((i + j) * kRowThreads + tid);
    if (__any_sync(0xffffffffu, s[0] != 0.0f || s[1] != 0.0f || s[2] != 0.0f || s[3] != 0.0f)) {
#pragma unroll
      for (int o = 1; o < 32; o <<= 1)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const float p = __shfl_up_sync(0xffffffffu, s[j], o);
          if (lane >= o) s[j] += p;
        }
    }
    if (lane == 31)
#pragma unroll
      for (int j = 0; j < 4; ++j)
        if (i + j < rounds) sh.seg[(i + j) * kRowWarps + warp] = s[j];
  }
  __syncthreads();
  if (warp == 0) {
    // Upper borders of the segments. A scan by halves adds neighbours up in different orders: its sums may rise by a rounding over a
    // segment that keeps nothing, or fall. The border of an empty segment is that of the one before, and no border lies
    // below an earlier one: they rise at segments that hold something and nowhere else.
    float top = 0.0f;
    bool odd = false;      // a NaN among the weights
    for (int s0 = lane; s0 - lane < segs; s0 += 128) {      // 32 segments a scan, four scans side by side
      float border[4], sum[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) sum[j] = border[j] = s0 + 32 * j < segs ? sh.seg[s0 + 32 * j] : 0.0f;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const float p = __shfl_up_sync(0xffffffffu, sum[j], o);
          if (lane >= o) sum[j] += p;
        }
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        odd = odd || border[j] != border[j];
        border[j] = border[j] > 0.0f ? sum[j] : 0.0f;
      }
#pragma unroll
      for (int o = 1; o < 32; o <<= 1)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const float p = __shfl_up_sync(0xffffffffu, border[j], o);
          if (lane >= o) border[j] = fmaxf(border[j], p);
        }
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        if (s0 + 32 * j < segs) sh.seg[s0 + 32 * j] = top + border[j];
        top += __shfl_sync(0xffffffffu, border[j], 31);
      }
    }
    if (__any_sync(0xffffffffu, odd)) top = __int_as_float(0x7fffffff);
    if (lane < cluster) ptx::st_cluster_f32(ptx::mapa(ptx::smem_u32(&sh.slice_mass[rank]), lane), top);
  }
  ptx::cluster_sync();
  float lo = 0.0f, total = 0.0f;
  for (int q = 0; q < cluster; ++q) {
    if (q == rank) lo = total;
    total += sh.slice_mass[q];
  }
  const float u = uniforms != nullptr ? uniforms[row] : philox_uniform(seed, step, static_cast<uint32_t>(row));
  const float target = u * total;
  // rounding fell off the end, a NaN among the weights, a caller's number outside [0, 1): the mode is always in the kept set
  if (!(target >= 0.0f && target < total)) {
    store_mode();
    return;
  }
  const float hi = lo + sh.slice_mass[rank];
  if (!(lo <= target && target < hi)) return;
  // exactly one segment holds the target, and it keeps something: neighbours share a border, adding `lo` leaves them in order
  for (int s = warp; s < segs; s += kRowWarps) {
    const float a = s > 0 ? lo + sh.seg[s - 1] : lo, b = lo + sh.seg[s];
    if (!(a <= target && target < b)) continue;
    const int v = (s / kRowWarps) * kRowThreads + (s % kRowWarps) * 32 + lane;
    const float own = lane_weight(v), incl = warp_scan(own);
    const unsigned reach = __ballot_sync(0xffffffffu, own > 0.0f && target < a + incl), some = __ballot_sync(0xffffffffu, own > 0.0f);
    const int pick_lane = reach ? __ffs(reach) - 1 : 31 - __clz(some);
    if (lane == pick_lane) {
      float acc = a + (incl - own);
      int pick = (v0 + v) * 8;
      for (int j = 0; j < 8; ++j) {
        const uint32_t bits = (reinterpret_cast<const uint32_t*>(&vals[v])[j >> 1] >> (16 * (j & 1))) & 0xffffu;
        if (key16(bits) < floor_key) continue;
        const float w = weight(__uint_as_float(bits << 16));
        if (w > 0.0f) pick = (v0 + v) * 8 + j;
        acc += w;
        if (acc > target) break;
      }
      ids[row] = pick;
    }
  }
}

}  // namespace
}  // namespace b2

using namespace b2;

extern "C" int b2_argmax(const void* logits, int is_bf16, int64_t* ids, float* max_out, int rows, int vocab,
                         int64_t row_stride, cudaStream_t stream) {
  if (rows <= 0) return 0;
  if (vocab <= 0) return -kBadArgument;
  const int c = cluster_for(rows, vocab, kNumSMs + 12);      // 40 rows x 4 still pay: 128256 logits 5.1 us, 5.6 with two CTAs a row
  const dim3 grid(static_cast<unsigned>(rows) * c), block(kRowThreads);
  const cudaError_t e = is_bf16 ? launch_cluster(argmax_kernel<true>, grid, block, c, 0, stream, logits, ids, max_out, vocab, row_stride, c)
                                : launch_cluster(argmax_kernel<false>, grid, block, c, 0, stream, logits, ids, max_out, vocab, row_stride, c);
  return e != cudaSuccess ? cuda_rc(e) : last_launch_rc();
}

extern "C" int b2_sample(const void* logits, int is_bf16, int64_t* ids, const float* temperature, const int32_t* top_k,
                         const float* top_p, const float* uniforms, uint64_t seed, uint64_t step, int rows, int vocab,
                         int64_t row_stride, cudaStream_t stream) {
  if (rows <= 0) return 0;
  if (vocab <= 0) return -kBadArgument;
  // Every CTA of a row clears and walks over all bins, so that clusters are narrower here: eight CTAs only for a few long rows, at least
  // two from 32768 logits on and four from 65536 (slices of at most 64 KB: two CTAs fit an SM, and a long list of rows follows in waves).
  // us with top-k and top-p by 1 / 2 / 4 / 8 CTAs a row (the passes over a copy were 3 to 15 % slower then): 256 x 1000 11.4 / 23 / 53 / 161 (30 with the kernel of one CTA a row above),
  // 64 x 32000 14.1 / 12.9 / 16.0 / 45, 600 x 50257 91 / 82 / 141 / 379, 17 x 128256 - / 18.8 / 15.5 / 23.9.
  int c = cluster_for(rows, vocab, kNumSMs);
  if (c == kMaxCluster && (rows > 8 || vocab <= 16384)) c = 4;
  while (c < 4 && vocab > 32768 * c) c <<= 1;
  while (c < kMaxCluster && vocab / c * 2 + kBins * 4 > 196 * 1024) c <<= 1;
  const int slice = ((vocab + 7) / 8 + c - 1) / c;      // 16-byte vectors of a CTA
  const int smem = slice * 16 + kBins * 4;
  if (is_bf16 && smem <= 200 * 1024 && slice <= kMaxSegs / kRowWarps * kRowThreads) {
    static DeviceOnce attr_once;
    if (const int rc = attr_once.max_smem(sample_row_kernel, 200 * 1024)) return rc;
    const cudaError_t e = launch_cluster(sample_row_kernel, dim3(static_cast<unsigned>(rows) * c), dim3(kRowThreads), c, smem, stream,
                                         static_cast<const __nv_bfloat16*>(logits), ids, temperature, top_k, top_p, uniforms, seed, step, vocab, row_stride, c, slice);
    return e != cudaSuccess ? cuda_rc(e) : last_launch_rc();
  }
  if (is_bf16)
    launch_pdl(sample_kernel<true>, dim3(rows), dim3(kThreads), 0, stream, logits, ids, temperature, top_k, top_p, uniforms, seed, step,
                                                       vocab, row_stride);
  else
    launch_pdl(sample_kernel<false>, dim3(rows), dim3(kThreads), 0, stream, logits, ids, temperature, top_k, top_p, uniforms, seed, step,
                                                        vocab, row_stride);
  return last_launch_rc();
}
