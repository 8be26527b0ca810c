// Epilogue of the grouped expert products: weights are the 128-row UMMA M side, the tokens of one expert the N side.
// A unit's q_coord is its first row in the token matrix (input and output rows coincide), nsplit the number of its rows
// that hold tokens.
#pragma once
#include <cuda_bf16.h>
#include "b2/act.cuh"
#include "b2/gemm_tc.cuh"
#include "b2/ptx.cuh"

namespace b2 {

struct GroupedEpiParams {
  __nv_bfloat16* y;
  int64_t ldy;
  int n_rows;      // rows of one expert's weight
  int mode;        // B2_EPI_NONE, B2_EPI_RELU2 or B2_EPI_SWIGLU
  B2EpiAct act;
};

template <int BN>
struct GroupedEpilogue {
  static constexpr int CH = BN >= 32 ? 32 : 16;
  GroupedEpiParams p;
  int first = 0, step = 1;      // the chunks of CH tokens that this warp takes, where several share 32 rows of the weights
  __device__ __forceinline__ void operator()(const gemm::WorkUnit& u, uint32_t taddr, int quarter, int lane, uint32_t*,
                                             Status*) const {
#pragma unroll 1
    for (int c = first; c < BN / CH; c += step) {
      if (c * CH >= u.nsplit) break;
      chunk(u, taddr + c * CH, c * CH, quarter, lane);
    }
  }
  // CH tokens from token m0 of the unit on, at `taddr`.
  __device__ __forceinline__ void chunk(const gemm::WorkUnit& u, uint32_t taddr, int m0, int quarter, int lane) const {
    const int p_local = quarter * 32 + lane;
    const int n = u.pb * 128 + p_local;
    __nv_bfloat16* base = p.y + static_cast<int64_t>(u.q_coord) * p.ldy;
    uint32_t r[CH];
    if constexpr (CH == 32) ptx::tmem_ld_32x32(taddr, r);
    else ptx::tmem_ld_32x16(taddr, r);
    ptx::tc_wait_ld();
    if (p.mode == B2_EPI_SWIGLU) {
      // lanes 0-15 hold gates, 16-31 the values that go with them; of two tokens either half works out one
      const bool lower = lane < 16;
      const int out_col = (u.pb * 128 + (p_local & ~31)) / 2 + (lane & 15);
#pragma unroll
      for (int j = 0; j < CH; j += 2) {
        const float v0 = __uint_as_float(r[j]), v1 = __uint_as_float(r[j + 1]);
        const float other = __shfl_xor_sync(0xffffffffu, lower ? v1 : v0, 16);
        const int m = m0 + j + (lower ? 0 : 1);
        const float o = glu(p.act, lower ? v0 : other, lower ? other : v1);
        if (n < p.n_rows && m < u.nsplit) base[static_cast<int64_t>(m) * p.ldy + out_col] = __float2bfloat16(o);
      }
    } else if (n < p.n_rows) {
#pragma unroll
      for (int j = 0; j < CH; ++j) {
        if (m0 + j >= u.nsplit) break;
        const float v = __uint_as_float(r[j]);
        base[static_cast<int64_t>(m0 + j) * p.ldy + n] = __float2bfloat16(p.mode == B2_EPI_RELU2 ? relu2(v) : v);
      }
    }
  }
};

constexpr int grouped_stages_for(int bn) {
  const int stage = 128 * 64 * 2 + bn * 64 * 2;
  const int s = (200 * 1024) / stage;
  return s > 10 ? 10 : s;
}

}  // namespace b2
