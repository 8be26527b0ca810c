// bf16 product for a handful of rows: Y[M, N] = X[M, K] * W[N, K]^T, M <= 32, f32 accumulate, the epilogues of gemm_bf16.cu.
//
// At these sizes every byte of W is read once and the tensor work is nothing; what counts is how soon the loads start, how many
// are on their way, and how little follows the last one. The tcgen05 kernel of gemm_bf16.cu pays for TMEM, one deep ring per SM
// and a semaphore for split tiles: 7.8 us for 3072 x 2048 (2 us of HBM time), 10.8 us for 4096 x 4096 (5 us) in its best configuration for one
// row; this one takes 6.7 and 8.9 us. At 32 rows the two are about level, above that the tensor cores of the other one win. Here a small CTA
// takes 64 weight rows and one slice of K: a producer warp keeps a ring of TMA boxes full, four warps multiply 16 rows each with
// mma.sync, and four CTAs share an SM (about 190 KB on the way). Where the rows alone give too few CTAs, those of a cluster
// split K and the first one adds up the partial sums, in order of rank, through distributed shared memory.
//
// The tensor cores cut off what does not fit when they add to an accumulator, so that a long run of products drifts towards zero.
// Each block of 64 columns is summed by itself and added in rounded 32-bit arithmetic, which costs no time here: error of an f32 result
// against 64 bits 1.1e-7 at K = 4096 and 2.1e-7 at 28672 (one accumulator all along: 9.8e-7 and 8.0e-6; the tcgen05 kernel 8.0e-7, 3.8e-6).
//
// Under programmatic dependent launch the first boxes of W are requested into L2 before the kernel in front has finished (L2 only:
// whoever writes W in that kernel is still seen): 16384 x 2048 behind a norm 14.4 -> 13.5 us. Not where a product narrows its input and a
// CTA's slice is longer than the ring: such products mostly follow the one that widened it, which is still reading weights of its own, and only
// delay it (gate and up, then down, layer by layer, us with / without: width 2048 35.9 / 35.0, 4096 83.5 / 82.5, 5120 96.2 / 95.9; thirteen steps
// of a chat 5.55 / 5.45 ms). More boxes than the ring holds cost time everywhere (5.64 ms with eight, 5.74 with sixteen), and so do
// norms and rotations that let the next kernel start before they wait themselves (5.48 -> 5.59 ms).
#include <cstdint>
#include <cuda.h>
#include <cuda_bf16.h>
#include "b2/act.cuh"
#include "b2/api.h"
#include "b2/config.h"
#include "b2/launch.h"
#include "b2/ptx.cuh"
#include "b2/status.h"
#include "b2/tma.h"

namespace b2 {
namespace {

constexpr int kRows = 64, kWarps = 4, kThreads = kWarps * 32 + 32, kWBytes = kRows * 128, kMaxSplit = 8;
constexpr int stages_of(int nt) { return nt <= 2 ? 5 : 4; }
constexpr int ring_bytes(int nt) { return stages_of(nt) * (kWBytes + nt * 1024); }

struct StreamParams {
  void* y;
  const __nv_bfloat16* residual;
  int64_t ldy;
  int M, N, num_kb, splits, mode;
  B2EpiAct act;
};

__device__ __forceinline__ void ldsm4(uint32_t addr, uint32_t (&r)[4]) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}
__device__ __forceinline__ void mma16816(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
               : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void prefetch_box(const void* tmap, int x, int y) {
  asm volatile("cp.async.bulk.prefetch.tensor.2d.L2.global.tile [%0, {%1, %2}];" ::"l"(tmap), "r"(x), "r"(y) : "memory");
}

template <int NT>      // groups of eight rows of X
__global__ void __launch_bounds__(kThreads) gemm_stream_kernel(const __grid_constant__ CUtensorMap tmap_w, const __grid_constant__ CUtensorMap tmap_x, StreamParams p,
                                                               Status* status) {
  constexpr int STAGES = stages_of(NT), kStage = kWBytes + NT * 1024;
  extern __shared__ uint8_t smem_raw[];
  __shared__ uint64_t bars[2 * STAGES];
  const uint32_t base = (ptx::smem_u32(smem_raw) + 1023u) & ~1023u;
  float* buf = reinterpret_cast<float*>(smem_raw + (base - ptx::smem_u32(smem_raw)));      // the ring again, once it is done with
  const uint32_t full0 = ptx::smem_u32(bars), empty0 = full0 + 8 * STAGES;
  const int warp = ptx::warp_id(), lane = threadIdx.x & 31;
  const int rank = blockIdx.x % p.splits, n0 = blockIdx.x / p.splits * kRows;
  const int kb0 = p.num_kb * rank / p.splits, kb1 = p.num_kb * (rank + 1) / p.splits;
  if (threadIdx.x == kWarps * 32) {
    if (p.N >= p.num_kb * 64 || kb1 - kb0 <= STAGES)      // see the head of the file
      for (int kb = kb0; kb < min(kb1, kb0 + STAGES); ++kb) prefetch_box(&tmap_w, kb * 64, n0);
    for (int s = 0; s < STAGES; ++s) {
      ptx::mbar_init(full0 + 8 * s, 1);
      ptx::mbar_init(empty0 + 8 * s, kWarps);
    }
    ptx::fence_mbar_init();
  }
  __syncthreads();
  ptx::grid_dep_sync();

  float acc[NT][4];
#pragma unroll
  for (int i = 0; i < NT; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = 0.0f;
  if (warp == kWarps) {
    if (lane == 0) {
      int issued = 0;
      for (int kb = kb0; kb < kb1; ++kb, ++issued) {
        const int s = issued % STAGES;
        if (!ptx::mbar_wait(empty0 + 8 * s, ((issued / STAGES) & 1) ^ 1u)) {
          status_record(status, kTimeout, kSiteGemmEmpty, blockIdx.x, kb);
          break;
        }
        const uint32_t at = base + s * kStage;
        ptx::mbar_arrive_expect_tx(full0 + 8 * s, kStage);
        ptx::tma_load_2d(at, &tmap_w, full0 + 8 * s, kb * 64, n0, ptx::kEvictFirst);
        ptx::tma_load_2d(at + kWBytes, &tmap_x, full0 + 8 * s, kb * 64, 0, ptx::kEvictLast);
      }
      // whoever gave up: copies in flight land before the shared memory is used again or given up
      for (int i = max(0, issued - STAGES); i < issued; ++i) ptx::mbar_wait(full0 + 8 * (i % STAGES), (i / STAGES) & 1, 100000000ull);
    }
    __syncwarp();
  } else {
    for (int kb = kb0; kb < kb1; ++kb) {
      const int it = kb - kb0, s = it % STAGES;
      if (!__all_sync(0xffffffffu, ptx::mbar_wait(full0 + 8 * s, (it / STAGES) & 1))) {
        if (lane == 0) status_record(status, kTimeout, kSiteGemmFull, blockIdx.x, kb);
        break;
      }
      const uint32_t w_at = base + s * kStage, x_at = w_at + kWBytes;
      uint32_t a[4][4];
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const int row = warp * 16 + (lane & 15), chunk = k * 2 + (lane >> 4);
        ldsm4(w_at + row * 128 + ((chunk ^ (row & 7)) << 4), a[k]);
      }
#pragma unroll
      for (int i = 0; i < NT; ++i) {
        float sum[4] = {0.0f, 0.0f, 0.0f, 0.0f};      // of this block: see the head of the file
#pragma unroll
        for (int k2 = 0; k2 < 2; ++k2) {
          uint32_t b[4];
          const int row = i * 8 + (lane & 7), chunk = k2 * 4 + (lane >> 3);
          ldsm4(x_at + row * 128 + ((chunk ^ (row & 7)) << 4), b);
          mma16816(sum, a[2 * k2], b[0], b[1]);
          mma16816(sum, a[2 * k2 + 1], b[2], b[3]);
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] += sum[j];
      }
      __syncwarp();
      if (lane == 0) ptx::mbar_arrive(empty0 + 8 * s);
    }
  }

  // ---- partial sums of the cluster's CTAs ----
  if (p.splits > 1) {
    ptx::cluster_sync();      // every CTA is done with its ring
    if (rank > 0 && warp < kWarps) {
      const uint32_t to = ptx::mapa(ptx::smem_u32(buf + (rank - 1) * NT * 4 * kWarps * 32), 0);
#pragma unroll
      for (int i = 0; i < NT; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) ptx::st_cluster_f32(to + ((i * 4 + j) * kWarps * 32 + threadIdx.x) * 4, acc[i][j]);
    }
    ptx::cluster_sync();
    if (rank > 0 || warp == kWarps) return;
    for (int r = 0; r + 1 < p.splits; ++r)
#pragma unroll
      for (int i = 0; i < NT; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] += buf[(r * NT * 4 + i * 4 + j) * kWarps * 32 + threadIdx.x];
  } else if (warp == kWarps) {
    return;
  }
  const int g = lane >> 2, t = lane & 3;
  if (p.mode == B2_EPI_SWIGLU) {
    // odd warps hold the up rows of the gate rows in the warp before
    ptx::named_barrier_sync(1, kWarps * 32);
    float* mine = buf + (warp >> 1) * NT * 4 * 32 + lane;
    if (warp & 1) {
#pragma unroll
      for (int i = 0; i < NT; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) mine[(i * 4 + j) * 32] = acc[i][j];
    }
    ptx::named_barrier_sync(1, kWarps * 32);
    if (warp & 1) return;
    __nv_bfloat16* y = static_cast<__nv_bfloat16*>(p.y);
#pragma unroll
    for (int i = 0; i < NT; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int n = n0 + warp * 16 + 16, col = n0 / 2 + (warp >> 1) * 16 + g + (j >> 1) * 8, m = i * 8 + 2 * t + (j & 1);      // N is a multiple of 32
        if (n < p.N && m < p.M) y[static_cast<int64_t>(m) * p.ldy + col] = __float2bfloat16(glu(p.act, acc[i][j], mine[(i * 4 + j) * 32]));
      }
    return;
  }
#pragma unroll
  for (int i = 0; i < NT; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int n = n0 + warp * 16 + g + (j >> 1) * 8, m = i * 8 + 2 * t + (j & 1);
      if (n >= p.N || m >= p.M) continue;
      const int64_t at = static_cast<int64_t>(m) * p.ldy + n;
      float v = acc[i][j];
      if (p.mode == B2_EPI_F32) {
        static_cast<float*>(p.y)[at] = v;
        continue;
      }
      if (p.mode == B2_EPI_RELU2) v = relu2(v);
      else if (p.mode == B2_EPI_SOFTCAP) v = softcap(v, p.act.cap);
      else if (p.mode == B2_EPI_ADD_RESIDUAL) v += __bfloat162float(p.residual[at]);
      static_cast<__nv_bfloat16*>(p.y)[at] = __float2bfloat16(v);
    }
}

// Split until about three CTAs per SM have work, with four k-blocks (32 KB of W) each at least; the partial sums of the others have
// to fit where the first CTA's ring was.
template <int NT>
int splits_for(int N, int num_kb) {
  const int tiles = (N + kRows - 1) / kRows;
  int splits = 1;
  while (splits < kMaxSplit && tiles * splits * 2 <= 3 * kNumSMs && num_kb >= 8 * splits && (2 * splits - 1) * NT * 4 * kWarps * 32 * 4 <= ring_bytes(NT)) splits *= 2;
  return splits;
}

template <int NT>
int launch(const void* x, const void* w, int64_t ldx, int64_t ldw, int K, StreamParams p, Status* status, cudaStream_t stream) {
  CUtensorMap tw, tx;
  if (!make_tmap_2d(&tw, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, w, p.N, K, ldw * 2, kRows, 64, CU_TENSOR_MAP_SWIZZLE_128B) ||
      !make_tmap_2d(&tx, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, x, p.M, K, ldx * 2, NT * 8, 64, CU_TENSOR_MAP_SWIZZLE_128B))
    return -kBadArgument;
  const int tiles = (p.N + kRows - 1) / kRows;
  p.splits = splits_for<NT>(p.N, p.num_kb);
  constexpr int kSmem = ring_bytes(NT) + 1024;
  auto kern = gemm_stream_kernel<NT>;
  static DeviceOnce attr_once;
  if (const int rc = attr_once.max_smem(kern, kSmem)) return rc;
  const cudaError_t e = launch_cluster(kern, dim3(static_cast<unsigned>(tiles * p.splits)), dim3(kThreads), p.splits, kSmem, stream, tw, tx, p, status);
  return e != cudaSuccess ? cuda_rc(e) : last_launch_rc();
}

}  // namespace

// Whether M <= 32 rows come here. Up to 16 always; above, a warp's turn on a k-block takes so long that only short slices of K pay. us, this
// / gemm_bf16.cu at 32 rows: 3072 x 2048 (8 k-blocks a CTA) 7.5 / 8.8, 6144 x 4096 (16) 14.9 / 17.2, 1536 x 5120 (20) 10.3 / 9.6,
// 2048 x 8192 (32) 15.5 / 12.7, 7168 x 18432 (144) 58 / 48.
bool gemm_stream_takes(int M, int N, int K) {
  const int num_kb = (K + 63) / 64;
  return M <= 16 || (M <= 32 && num_kb <= 16 * splits_for<4>(N, num_kb));
}

// Called by b2_gemm_bf16 (which has checked the shapes) where `gemm_stream_takes` says so.
int launch_gemm_stream(const void* x, const void* w, void* y, const void* residual, int M, int N, int K, int64_t ldx, int64_t ldw, int64_t ldy, int epilogue,
                       const B2EpiAct* act, Status* status, cudaStream_t stream) {
  const StreamParams p{y, static_cast<const __nv_bfloat16*>(residual), ldy, M, N, (K + 63) / 64, 1, epilogue, act != nullptr ? *act : kPlainAct};
  if (M <= 8) return launch<1>(x, w, ldx, ldw, K, p, status, stream);
  if (M <= 16) return launch<2>(x, w, ldx, ldw, K, p, status, stream);
  return launch<4>(x, w, ldx, ldw, K, p, status, stream);
}

}  // namespace b2
