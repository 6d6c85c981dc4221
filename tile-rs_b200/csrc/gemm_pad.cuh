// Copies that bring 16-bit matrices whose rows do not start on 16-byte boundaries into a layout the tensor maps can
// describe: a GEMM of odd sizes then runs on the tensor cores as any other, and writes its result where it belongs.
// A stream of a few bytes per row and column of the operands (HBM / L2 bound); it pays as soon as the FP32-pipe
// kernel, at a hundredth of the tensor cores' rate, would take longer than a launch.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "ptx.cuh"

namespace tsm100 {
namespace gemm_pad {

constexpr int kThreads = 256;
// src [rows][cols] with row pitch ld (problems `batch` elements apart) -> dst [rows][pitch] packed, zeros beyond cols.
// pitch is a multiple of 8 and dst 16-byte aligned.
struct Operand {
  const uint16_t* src;
  uint4* dst;
  int64_t ld, batch;
  int32_t rows, cols, pitch;
  int32_t blocks;   // of the launch that work on it, 0: it is not copied
};

// Eight values from element `at` of a matrix that ends at `size`, as the two 16-byte vectors that hold them; a value at a time
// where those reach past the matrix.
__device__ __forceinline__ uint4 load8(const uint16_t* src, int64_t at, int64_t size, int valid) {
  const uintptr_t address = reinterpret_cast<uintptr_t>(src + at), from = address & ~uintptr_t(15);
  const uint32_t shift = static_cast<uint32_t>(address & 15);
  uint32_t w[8] = {0u, 0u, 0u, 0u, 0u, 0u, 0u, 0u};
  if (valid >= 8 && from >= reinterpret_cast<uintptr_t>(src) && from + 32 <= reinterpret_cast<uintptr_t>(src + size)) {
    const uint4 x = *reinterpret_cast<const uint4*>(from);
    w[0] = x.x, w[1] = x.y, w[2] = x.z, w[3] = x.w;
    if (shift != 0) {
      const uint4 y = *reinterpret_cast<const uint4*>(from + 16);
      w[4] = y.x, w[5] = y.y, w[6] = y.z, w[7] = y.w;
    }
    if (shift & 8) {
#pragma unroll
      for (int i = 0; i < 6; ++i) w[i] = w[i + 2];
    }
    if (shift & 4) {
#pragma unroll
      for (int i = 0; i < 5; ++i) w[i] = w[i + 1];
    }
    const uint32_t bits = (shift & 2) * 8;
    return make_uint4(__funnelshift_r(w[0], w[1], bits), __funnelshift_r(w[1], w[2], bits), __funnelshift_r(w[2], w[3], bits), __funnelshift_r(w[3], w[4], bits));
  }
#pragma unroll
  for (int j = 0; j < 8; ++j)
    if (j < valid) w[j >> 1] |= static_cast<uint32_t>(src[at + j]) << ((j & 1) * 16);
  return make_uint4(w[0], w[1], w[2], w[3]);
}

// One thread per eight values of a row; the operands' blocks side by side in one launch.  blockIdx.y = problem.
__global__ void __launch_bounds__(kThreads)
pad_kernel(const Operand a, const Operand b) {
  ptx::launch_dependents_if_few();  // 289 x 5995 x 2550 in a row of calls 36.4 us, 50.2 with the GEMM placed beside 2368 CTAs of this
  const bool first = static_cast<int32_t>(blockIdx.x) < a.blocks;
  const Operand& p = first ? a : b;
  const int32_t block = first ? blockIdx.x : blockIdx.x - a.blocks;
  const uint16_t* src = ptx::wait_prior_grid(p.src) + blockIdx.y * p.batch;
  const uint32_t per_row = static_cast<uint32_t>(p.pitch) / 8;
  const int64_t total = static_cast<int64_t>(p.rows) * per_row, step = static_cast<int64_t>(p.blocks) * kThreads;
  const int64_t size = static_cast<int64_t>(p.rows - 1) * p.ld + p.cols;
  uint4* dst = p.dst + blockIdx.y * total;
#pragma unroll 2
  for (int64_t i = static_cast<int64_t>(block) * kThreads + threadIdx.x; i < total; i += step) {
    const int64_t r = total <= 0xffffffffll ? static_cast<int64_t>(static_cast<uint32_t>(i) / per_row) : i / per_row;
    const int32_t c = static_cast<int32_t>(i - r * per_row) * 8;
    dst[i] = load8(src, r * p.ld + c, size, p.cols - c);
  }
}

}  // namespace gemm_pad
}  // namespace tsm100
