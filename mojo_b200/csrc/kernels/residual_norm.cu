// A plain residual kept in f32: one kernel between any two sublayers adds the finished one (a matrix product's rows, the
// weighted rows of a token's experts, a row with a gate, or several of them, scaled per channel) and RMS- or layer-normalises
// what the next one reads. The first
// call starts the stream from the embedding tables. One CTA per token row; a warp per row where many short ones fold experts' rows in bf16.
#include <cstdint>
#include <type_traits>
#include "b2/elem.cuh"
#include "b2/launch.h"
#include "b2/mixers.h"
#include "b2/ptx.cuh"
#include "b2/short_conv.cuh"
#include "b2/vec.cuh"

namespace b2 {
namespace {

constexpr int kMaxTop = 32, kWarpRows = 4;

// AT: rows of a token's experts that are requested before the first is used. WARP: a warp per row, kWarpRows of them in a CTA; else a CTA
// per row.
template <typename T, int VEC, int AT, bool WARP>
__global__ void residual_norm_kernel(const B2ResidualArgs a, Status* status) {
  ptx::grid_dep_sync();
  constexpr int kRows = WARP ? kWarpRows : 1;
  extern __shared__ float rows_sm[];    // the rows; every thread touches its own columns only
  __shared__ float scratch[33], e_w_all[kRows][kMaxTop];
  __shared__ int e_row_all[kRows][kMaxTop];
  // functions, not values: with the numbers in registers of their own f32 rows of experts take a fifth longer
  const auto tid = [] { return WARP ? threadIdx.x & 31 : threadIdx.x; };
  const auto n_threads = [] { return WARP ? 32 : blockDim.x; };
  const unsigned mine = WARP ? threadIdx.x >> 5 : 0;
  const unsigned out_row = WARP ? blockIdx.x * kRows + mine : blockIdx.x;
  if (WARP && static_cast<int>(out_row) >= a.n_out) return;      // whole warps, and nothing below joins them
  float *x_sm = rows_sm + static_cast<int64_t>(mine) * a.width, *e_w = e_w_all[mine];
  int* e_row = e_row_all[mine];
  const auto sum_all = [&](float v) {
    if constexpr (WARP) return warp_sum(v);
    else return block_sum(v, scratch);
  };
  int64_t row = out_row;
  if (a.rows_index != nullptr) {
    row = a.rows_index[out_row];
    if (!B2_ASSERT(status, row >= 0 && row < a.rows, kSiteKvIndex, row, a.rows)) return;   // uniform per row
  }
  if (a.experts != nullptr) {
    if (tid() < a.top) {
      const int slot = a.expert_slot[row * a.top + tid()];
      const bool ok = B2_ASSERT(status, slot >= (a.own != nullptr ? -1 : 0) && slot < a.expert_rows, kSiteEpCount, slot, a.expert_rows);
      e_row[tid()] = ok ? slot : 0;
      e_w[tid()] = !ok ? 0.0f : a.expert_w != nullptr ? a.expert_w[row * a.top + tid()] : 1.0f;
    }
    if constexpr (WARP) __syncwarp();
    else __syncthreads();
  }
  const int W = a.width;
  float* x = a.x + row * W;
  const T* y = a.y != nullptr ? static_cast<const T*>(a.y) + row * W : nullptr;
  const T *emb = nullptr, *big = nullptr;
  if (a.ids != nullptr) {
    const int64_t id = a.ids[row];
    if (B2_ASSERT(status, id >= 0 && id < a.vocab, kSiteKvIndex, id, a.vocab)) {
      emb = static_cast<const T*>(a.embed) + id * W;
      if (a.bigram != nullptr) {
        const int64_t prev = a.prev[row];
        const int64_t at = prev < 0 ? a.buckets : (prev * a.mul_prev + id * a.mul_cur) % a.buckets;
        if (B2_ASSERT(status, at >= 0 && at <= a.buckets, kSiteKvIndex, at, a.buckets)) big = static_cast<const T*>(a.bigram) + at * W;
      }
    }
  }
  const T* own = a.own != nullptr ? static_cast<const T*>(a.own) + row * W : nullptr;
  const T* gated = a.gated != nullptr ? static_cast<const T*>(a.gated) + row * W : nullptr;
  const float gate = gated != nullptr ? sigmoid_f32(a.gate[row * a.ld_gate]) : 0.0f;
  const bool fold = y != nullptr || a.experts != nullptr || gated != nullptr;
  float ss = 0.0f;
  for (int c = tid() * VEC; c < W; c += n_threads() * VEC) {
    float v[VEC];
    if (a.ids != nullptr) {
      float e[VEC] = {}, b[VEC] = {};
      if (emb != nullptr) load_f32<VEC>(emb + c, e);
      if (big != nullptr) load_f32<VEC>(big + c, b);
#pragma unroll
      for (int i = 0; i < VEC; ++i) v[i] = fmaf(e[i], a.embed_scale, b[i]);
      if (a.x0 != nullptr) store_f32<VEC>(static_cast<T*>(a.x0) + row * a.ld_x0 + c, v);
    } else {
      load_f32<VEC>(x + c, v);
    }
    if (fold) {
      float u[VEC] = {}, s[VEC];
      if (y != nullptr) load_f32<VEC>(y + c, u);
      if (a.experts != nullptr) {
        for (int j0 = 0; j0 < a.top; j0 += AT) {
          std::conditional_t<VEC == 8, RawVec<T, VEC>, float[VEC]> e[AT];
#pragma unroll
          for (int j = 0; j < AT; ++j)
            if (j0 + j < a.top) {
              const T* from = (e_row[j0 + j] < 0 ? own : static_cast<const T*>(a.experts) + static_cast<int64_t>(e_row[j0 + j]) * W) + c;
              if constexpr (VEC == 8) e[j].load(from);
              else load_f32<VEC>(from, e[j]);
            }
#pragma unroll
          for (int j = 0; j < AT; ++j)
            if (j0 + j < a.top)
#pragma unroll
              for (int i = 0; i < VEC; ++i) {
                if constexpr (VEC == 8) u[i] = fmaf(e_w[j0 + j], e[j].get(i), u[i]);
                else u[i] = fmaf(e_w[j0 + j], e[j][i], u[i]);
              }
        }
      }
      if (gated != nullptr) {
        float g[VEC];
        load_f32<VEC>(gated + c, g);
#pragma unroll
        for (int i = 0; i < VEC; ++i) u[i] = fmaf(gate, g[i], u[i]);
      }
      if (a.y_scale != nullptr) {
        load_f32<VEC>(a.y_scale + c, s);
#pragma unroll
        for (int i = 0; i < VEC; ++i) v[i] = fmaf(s[i], u[i], v[i]);
      } else {
#pragma unroll
        for (int i = 0; i < VEC; ++i) v[i] += u[i];
      }
    }
    if (a.store && (fold || a.ids != nullptr)) store_f32<VEC>(x + c, v);
#pragma unroll
    for (int i = 0; i < VEC; ++i) ss = a.bias != nullptr ? ss + v[i] : fmaf(v[i], v[i], ss);
    store_f32<VEC>(x_sm + c, v);
  }
  T* h = static_cast<T*>(a.h) + static_cast<int64_t>(out_row) * a.ld_h;
  float r = 1.0f, mean = 0.0f;
  if (a.bias != nullptr) {      // layer norm: squares of the deviations in a second pass
    mean = sum_all(ss) / static_cast<float>(a.mean_width);
    ss = 0.0f;
    for (int c = tid() * VEC; c < a.mean_width; c += n_threads() * VEC) {
      float v[VEC];
      load_f32<VEC>(x_sm + c, v);
#pragma unroll
      for (int i = 0; i < VEC; ++i)
        if (c + i < a.mean_width) ss = fmaf(v[i] - mean, v[i] - mean, ss);
    }
  }
  if (a.weight != nullptr) r = 1.0f / sqrtf(sum_all(ss) / static_cast<float>(a.mean_width) + a.eps);
  for (int c = tid() * VEC; c < W; c += n_threads() * VEC) {
    float v[VEC], w[VEC];
    load_f32<VEC>(x_sm + c, v);
    if (a.weight != nullptr) {
      load_f32<VEC>(a.weight + c, w);
#pragma unroll
      for (int i = 0; i < VEC; ++i) v[i] = (v[i] - mean) * r * w[i];
      if (a.bias != nullptr) {
        load_f32<VEC>(a.bias + c, w);
#pragma unroll
        for (int i = 0; i < VEC; ++i) v[i] += w[i];
      }
    }
    store_f32<VEC>(h + c, v);
  }
}

template <typename T, int VEC, int AT, bool WARP>
int launch_residual(const B2ResidualArgs& a, Status* status, cudaStream_t stream) {
  const int smem = (WARP ? kWarpRows : 1) * a.width * 4;
  static DeviceOnce attr_once;
  if (smem > 40 * 1024)
    if (const int rc = attr_once.max_smem(residual_norm_kernel<T, VEC, AT, WARP>, 200 * 1024)) return rc;
  const int vecs = (a.width + VEC - 1) / VEC;
  const int threads = WARP ? 32 * kWarpRows : vecs >= 256 ? 256 : (vecs + 31) / 32 * 32;
  launch_small(residual_norm_kernel<T, VEC, AT, WARP>, dim3(WARP ? (a.n_out + kWarpRows - 1) / kWarpRows : a.n_out), dim3(threads), smem, stream, a, status);
  return last_launch_rc();
}

}  // namespace
}  // namespace b2

using namespace b2;

extern "C" int b2_residual_norm(const B2ResidualArgs* a, int f32, Status* status, cudaStream_t stream) {
  if (a->n_out <= 0) return 0;
  if (a->width <= 0 || a->width > 50000 || a->mean_width <= 0 || a->mean_width > a->width || a->x == nullptr || a->h == nullptr ||
      (a->bias != nullptr && a->weight == nullptr) || (a->gated != nullptr && a->gate == nullptr) || (a->experts != nullptr && (a->expert_slot == nullptr || a->top < 1 || a->top > kMaxTop)) ||
      (a->ids != nullptr && a->embed == nullptr) || (a->bigram != nullptr && (a->prev == nullptr || a->buckets < 1)) ||
      (a->rows_index == nullptr && a->n_out != a->rows))
    return -kBadArgument;
  const bool v4 = a->width % 4 == 0 && a->ld_h % 4 == 0 && a->ld_x0 % 4 == 0;
  // Experts' rows in bf16 come in pieces of 16 bytes where every row begins on such a boundary, and many short rows go to warps that never meet, which keep
  // more loads in flight than CTAs with a barrier at either end of a row. With six experts a row, the stream out of L2 (us, four elements at a time / eight,
  // a CTA a row / eight, a warp a row): 5 x 2048 5.2 / 3.4 / 10.8, 1000 x 2048 21.6 / 16.9 / 19.2, 2000 x 2048 40 / 28 / 24, 4096 x 1024 45 / 27 / 25, 2000 x 4096
  // 72 / 47 / 73. All else stays with four: eight cost registers, and with them rows in flight, that nothing but experts' rows gives back (rows y of bf16, 1500 x 4096
  // 18.8 with four, 22.9 with eight; 4096 x 2048 25 / 27 by warps), and so do f32 rows that come eight experts at once (1200 x 2048 25 / 61).
  if (f32) return v4 ? launch_residual<float, 4, 4, false>(*a, status, stream) : launch_residual<float, 1, 4, false>(*a, status, stream);
  uintptr_t all = 0;
  for (const void* q : {static_cast<const void*>(a->x), a->y, a->embed, a->bigram, static_cast<const void*>(a->x0), a->experts, a->own, a->gated,
                        static_cast<const void*>(a->h), static_cast<const void*>(a->y_scale), static_cast<const void*>(a->weight), static_cast<const void*>(a->bias)})
    all |= reinterpret_cast<uintptr_t>(q);
  // Three CTAs of eight elements a thread fit an SM, four of the others: 512 x 2048 7.1 us instead of 6.6.
  const bool one_wave_of_four = a->width >= 2048 && a->n_out > 3 * kNumSMs && a->n_out <= 4 * kNumSMs;
  if (a->experts != nullptr && !one_wave_of_four && a->width % 8 == 0 && a->ld_h % 8 == 0 && a->ld_x0 % 8 == 0 && a->mean_width % 8 == 0 && all % 16 == 0)
    return a->width <= 2048 && a->n_out >= 1024 ? launch_residual<__nv_bfloat16, 8, 8, true>(*a, status, stream) : launch_residual<__nv_bfloat16, 8, 4, false>(*a, status, stream);
  return v4 ? launch_residual<__nv_bfloat16, 4, 4, false>(*a, status, stream) : launch_residual<__nv_bfloat16, 1, 4, false>(*a, status, stream);
}
