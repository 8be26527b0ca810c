// Forms of the block-scaled fp8 product that b2_gemm_fp8_block chooses between (csrc/kernels/gemm_fp8.cu holds the rule).
#pragma once
#include <cstdint>
#include <cuda_runtime.h>
#include "b2/status.h"

namespace b2 {

// Bit of an explicit configuration that names the kernel on CTA pairs, tiles of 256 rows x (config & 0xffff) columns.
constexpr int kFp8PairConfig = 1 << 28;

// On CTA pairs; `bn` 256 or 128. y 16-byte aligned with ldy a multiple of 8; K a multiple of 128, N of 8.
int gemm_fp8_pair(const void* xq, const float* xs, const void* wq, const float* ws, void* y, int M, int N, int K, int64_t ldy, int bn, Status* status,
                  cudaStream_t stream);

}  // namespace b2
