// Copies that bring 16-bit matrices whose rows do not start on 16-byte boundaries into a layout the tensor maps can
// describe, and results back: a GEMM of odd sizes then runs on the tensor cores as the next larger one of multiples of 8.
// Both directions are streams of a few bytes per product row and column (HBM / L2 bound); they pay as soon as the FP32-pipe
// kernel, at a hundredth of the tensor cores' rate, would take longer than their launches: 2000 x 3001 x 2501 bf16 1365 us there
// and 62 with the copies, 500 x 1001 x 999 166 / 15, 28 x 3134 x 4883 823 / 26.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "ptx.cuh"

namespace tsm100 {
namespace gemm_pad {

constexpr int kThreads = 256;
constexpr int kUnpadRows = 8;
// Up to how many CTAs the next kernel of the call is placed from the start: 300 x 1301 x 1203 bf16, whole call, 15.5 us with the 256 of other kernels,
// 14.7 this way; 3 of 22 x 1923 x 1267 18.7 with 1024 for the copies in, 17.0 this way.
constexpr uint32_t kFewCtasIn = 8192, kFewCtasOut = 1024;

// src [rows][cols] with row pitch ld (problems src_batch apart) -> dst [drows][dcols] packed, zeros beyond rows and cols.
// dcols is a multiple of 8 and dst 16-byte aligned: one thread per eight values.  blockIdx.y = problem.
__global__ void __launch_bounds__(kThreads)
pad_kernel(const uint16_t* __restrict__ src, int64_t ld, int64_t src_batch, int32_t rows, int32_t cols,
           uint4* __restrict__ dst, int32_t drows, int32_t dcols) {
  ptx::launch_dependents_if_few(kFewCtasIn);
  src = ptx::wait_prior_grid(src);
  const uint16_t* s = src + blockIdx.y * src_batch;
  const int64_t per_row = dcols / 8, total = drows * per_row;
  uint4* d = dst + blockIdx.y * total;
  for (int64_t i = blockIdx.x * static_cast<int64_t>(kThreads) + threadIdx.x; i < total; i += static_cast<int64_t>(gridDim.x) * kThreads) {
    const int64_t r = i / per_row;
    const int32_t c = static_cast<int32_t>(i - r * per_row) * 8;
    uint32_t w[4] = {0u, 0u, 0u, 0u};
    if (r < rows) {
      const uint16_t* q = s + r * ld + c;
#pragma unroll
      for (int j = 0; j < 8; ++j)
        if (c + j < cols) w[j >> 1] |= static_cast<uint32_t>(q[j]) << ((j & 1) * 16);
    }
    d[i] = make_uint4(w[0], w[1], w[2], w[3]);
  }
}

// src [rows][scols] packed -> dst [rows][cols] with row pitch ld (problems dst_batch apart), cols <= scols.
// One thread per column of ROWS rows, a warp's stores are contiguous and the loads of a thread in flight together: eight rows where there are
// CTAs for all SMs (2000 x 3001 x 65 bf16, whole call, 31.5 us row by row, 24 this way), one where there are few.  grid (x, groups of rows in
// strides, problem).
template <int ROWS>
__global__ void __launch_bounds__(kThreads)
unpad_kernel(const uint16_t* __restrict__ src, int32_t scols, uint16_t* __restrict__ dst, int64_t ld, int64_t dst_batch,
             int32_t rows, int32_t cols) {
  ptx::launch_dependents_if_few(kFewCtasOut);
  src = ptx::wait_prior_grid(src);
  const int32_t c = blockIdx.x * kThreads + threadIdx.x;
  if (c >= cols) return;
  const uint16_t* s = src + blockIdx.z * static_cast<int64_t>(rows) * scols + c;
  uint16_t* d = dst + blockIdx.z * dst_batch + c;
  for (int64_t r = static_cast<int64_t>(blockIdx.y) * ROWS; r < rows; r += static_cast<int64_t>(gridDim.y) * ROWS) {
    uint16_t v[ROWS];
#pragma unroll
    for (int k = 0; k < ROWS; ++k)
      if (r + k < rows) v[k] = s[(r + k) * scols];
#pragma unroll
    for (int k = 0; k < ROWS; ++k)
      if (r + k < rows) d[(r + k) * ld] = v[k];
  }
}

}  // namespace gemm_pad
}  // namespace tsm100
