// Row softmax for sm_100a: y[r, :] = exp(x[r, :] - max) / sum(exp(x[r, :] - max)).
//
// Semantics follow __tile_softmax_f32 / _f16 (crates/tile_std/src/tile.rs:189-190,
// :2162-2163) as the linalg bridge defines them, `linalg.softmax dimension(1)`
// (crates/rustc_codegen_tile/src/mlir_to_linalg.rs:1305-1343).  The reference's
// own CUDA lowering is one thread per element with two block reductions through
// shared memory and requires cols == blockDim <= 1024
// (crates/rustc_codegen_tile/src/mlir_to_gpu.rs:1242-1336); nothing of it is kept.
//
// The operator is bound by HBM: 2 * sizeof(T) algorithmic bytes per element.
// Kernels, picked by the host from the row width:
//   * softmax_rows_warp  : one warp per row, the whole row held in registers,
//     128-bit coalesced streaming loads, shuffle reductions, one global read and
//     one global write per element.  Rows of up to 256 16-byte vectors.
//   * softmax_rows_cta   : 128 or 256 threads per row, 32 values per thread in
//     registers, warp shuffles plus one shared-memory exchange per reduction; a
//     CTA takes one f32 row or two 16-bit rows and goes.  Rows of up to 2048
//     vectors.
//   * softmax_rows_warp_any, softmax_rows_cta_any: a warp or a CTA per row that
//     starts anywhere.
//   * softmax_rows_twice: wider rows of any alignment, one CTA each, read twice, the
//     second time from the L2 up to 450 KB a row.
//   * softmax_rows_cluster: a few such rows, a cluster of CTAs each.
//   * softmax_rows_stream: any width, x and y at different offsets from a 16-byte
//     boundary; online max/sum in a first pass, normalisation in a second (two
//     reads + one write).
// bf16 / f16 rows are widened to f32 on load; all arithmetic is f32; the store
// narrows with round-to-nearest-even.
#pragma once

#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <type_traits>

#include "ptx.cuh"

namespace tsm100 {
namespace softmax {

struct alignas(16) Vec16 {
  uint32_t w[4];
};

template <typename T>
struct Elem;  // conversion between storage type and f32

template <>
struct Elem<float> {
  static constexpr int kPerVec = 4;
  __device__ static __forceinline__ void unpack(const Vec16& v, float* f) {
#pragma unroll
    for (int i = 0; i < 4; ++i) f[i] = __uint_as_float(v.w[i]);
  }
  __device__ static __forceinline__ Vec16 pack(const float* f) {
    Vec16 v;
#pragma unroll
    for (int i = 0; i < 4; ++i) v.w[i] = __float_as_uint(f[i]);
    return v;
  }
  __device__ static __forceinline__ float load1(const float* p) { return *p; }
  __device__ static __forceinline__ void store1(float* p, float f) { *p = f; }
};

template <>
struct Elem<__nv_bfloat16> {
  static constexpr int kPerVec = 8;
  __device__ static __forceinline__ void unpack(const Vec16& v, float* f) {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      f[2 * i] = __uint_as_float(v.w[i] << 16);
      f[2 * i + 1] = __uint_as_float(v.w[i] & 0xffff0000u);
    }
  }
  __device__ static __forceinline__ Vec16 pack(const float* f) {
    Vec16 v;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      __nv_bfloat162 h = __floats2bfloat162_rn(f[2 * i], f[2 * i + 1]);
      v.w[i] = *reinterpret_cast<uint32_t*>(&h);
    }
    return v;
  }
  __device__ static __forceinline__ __nv_bfloat16 zero() { return __float2bfloat16_rn(0.f); }
  __device__ static __forceinline__ float load1(const __nv_bfloat16* p) { return __bfloat162float(*p); }
  __device__ static __forceinline__ void store1(__nv_bfloat16* p, float f) { *p = __float2bfloat16_rn(f); }
};

template <>
struct Elem<__half> {
  static constexpr int kPerVec = 8;
  __device__ static __forceinline__ void unpack(const Vec16& v, float* f) {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      __half2 h = *reinterpret_cast<const __half2*>(&v.w[i]);
      float2 t = __half22float2(h);
      f[2 * i] = t.x;
      f[2 * i + 1] = t.y;
    }
  }
  __device__ static __forceinline__ Vec16 pack(const float* f) {
    Vec16 v;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      __half2 h = __floats2half2_rn(f[2 * i], f[2 * i + 1]);
      v.w[i] = *reinterpret_cast<uint32_t*>(&h);
    }
    return v;
  }
  __device__ static __forceinline__ __half zero() { return __float2half_rn(0.f); }
  __device__ static __forceinline__ float load1(const __half* p) { return __half2float(*p); }
  __device__ static __forceinline__ void store1(__half* p, float f) { *p = __float2half_rn(f); }
};

// 128-bit streaming accesses: rows are touched exactly once, so they are
// marked evict-first and kept out of L1.
__device__ __forceinline__ Vec16 ld_stream(const Vec16* p) {
  Vec16 v;
  asm volatile("ld.global.cs.v4.u32 {%0, %1, %2, %3}, [%4];"
               : "=r"(v.w[0]), "=r"(v.w[1]), "=r"(v.w[2]), "=r"(v.w[3])
               : "l"(p));
  return v;
}
__device__ __forceinline__ Vec16 ld_keep(const Vec16* p) {  // for data that is read again soon
  Vec16 v;
  asm volatile("ld.global.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.w[0]), "=r"(v.w[1]), "=r"(v.w[2]), "=r"(v.w[3]) : "l"(p));
  return v;
}
__device__ __forceinline__ void st_stream(Vec16* p, const Vec16& v) {
  asm volatile("st.global.cs.v4.u32 [%0], {%1, %2, %3, %4};" ::"l"(p), "r"(v.w[0]), "r"(v.w[1]),
               "r"(v.w[2]), "r"(v.w[3])
               : "memory");
}

__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}
__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// ---------------------------------------------------------------------------
// One warp per row; lane l owns 16-byte vectors l, l+32, l+64, ... (CHUNKS of
// them).  cols must be a multiple of Elem<T>::kPerVec and x, y 16-byte aligned
// with a 16-byte-multiple row pitch (the host checks).
// ---------------------------------------------------------------------------
template <typename T, int CHUNKS, int WARPS>
__global__ void __launch_bounds__(WARPS * 32)
softmax_rows_warp(const T* __restrict__ x, T* __restrict__ y, int64_t rows, int32_t cols) {
  ptx::launch_dependents_if_few();
  ptx::wait_prior_grid();
  constexpr int PV = Elem<T>::kPerVec;
  const int lane = threadIdx.x & 31;
  const int64_t row = static_cast<int64_t>(blockIdx.x) * WARPS + (threadIdx.x >> 5);
  if (row >= rows) return;
  const int nvec = cols / PV;
  const Vec16* xr = reinterpret_cast<const Vec16*>(x + row * cols);
  Vec16* yr = reinterpret_cast<Vec16*>(y + row * cols);

  float v[CHUNKS][PV];
  Vec16 raw[CHUNKS];
#pragma unroll
  for (int c = 0; c < CHUNKS; ++c) {
    const int i = c * 32 + lane;
    if (i < nvec) raw[c] = ld_stream(xr + i);
  }
  float m = -INFINITY;
#pragma unroll
  for (int c = 0; c < CHUNKS; ++c) {
    const int i = c * 32 + lane;
    if (i < nvec) {
      Elem<T>::unpack(raw[c], v[c]);
#pragma unroll
      for (int e = 0; e < PV; ++e) m = fmaxf(m, v[c][e]);
    } else {
#pragma unroll
      for (int e = 0; e < PV; ++e) v[c][e] = -INFINITY;
    }
  }
  m = warp_max(m);
  float s = 0.f;
#pragma unroll
  for (int c = 0; c < CHUNKS; ++c) {
#pragma unroll
    for (int e = 0; e < PV; ++e) {
      // exp(-inf - m) = 0 for the padding; a row of all -inf yields NaN like the oracle.
      const float t = expf(v[c][e] - m);
      v[c][e] = t;
      s += t;
    }
  }
  s = warp_sum(s);
  const float inv = 1.0f / s;
#pragma unroll
  for (int c = 0; c < CHUNKS; ++c) {
    const int i = c * 32 + lane;
    if (i < nvec) {
#pragma unroll
      for (int e = 0; e < PV; ++e) v[c][e] *= inv;
      st_stream(yr + i, Elem<T>::pack(v[c]));
    }
  }
}

// exp(x - m) as 2^(x*log2e - m*log2e): one FMA and one MUFU op.  For |x - m| up to
// ~100 the rounding of the FMA argument costs less than 4e-6 relative, inside the
// 1e-5 bound of the f32 configuration; results below 2^-126 flush to zero.
constexpr float kLog2e = 1.4426950408889634f;
__device__ __forceinline__ float exp_shifted(float x, float m_log2e) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(fmaf(x, kLog2e, -m_log2e)));
  return y;
}

// ---------------------------------------------------------------------------
// THREADS threads per row, VPT 16-byte vectors per thread (vector k*THREADS + tid).
// Same alignment contract as the warp kernel; cols <= THREADS * VPT * kPerVec.
// A CTA takes a row or two and goes (ops.cuh: softmax_typed).  With CTAs that stay for many rows the SMs drift apart, and what they read and write lies
// ever further apart in HBM: 65536 rows of 4096, f32 355 us in CTAs that stay, 307 here (7.0 TB/s), bf16 171 / 158; a plain copy of 1 GiB 357 and 315.
// 16-bit rows, whose arithmetic takes as long as their traffic, come in twos, the loads of the second in flight while the first is worked on: 100000 of 2600
// bf16 204 us in CTAs that stay, 197 a row each, 174 two rows; f32 rows need the registers instead: 20000 of 6000 184, 152 a row each, 191 with room for two.
// ---------------------------------------------------------------------------
template <typename T, int VPT, int THREADS>
__global__ void __launch_bounds__(THREADS)
softmax_rows_cta(const T* __restrict__ x, T* __restrict__ y, int64_t rows, int32_t cols) {
  ptx::launch_dependents_if_few();
  ptx::wait_prior_grid();
  constexpr int PV = Elem<T>::kPerVec;
  constexpr int NW = THREADS / 32;
  __shared__ float red_max[NW];
  __shared__ float red_sum[NW];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int nvec = cols / PV;
  constexpr bool kAhead = sizeof(T) == 2;
  Vec16 raw[VPT], nxt[kAhead ? VPT : 1];
  auto load = [&](Vec16* to, int64_t row) {
    const Vec16* xr = reinterpret_cast<const Vec16*>(x + row * cols);
#pragma unroll
    for (int k = 0; k < VPT; ++k) {
      const int i = k * THREADS + tid;
      if (i < nvec) to[k] = ld_stream(xr + i);
    }
  };
  if (kAhead && static_cast<int64_t>(blockIdx.x) < rows) load(raw, blockIdx.x);
  for (int64_t row = blockIdx.x; row < rows; row += gridDim.x) {
    Vec16* yr = reinterpret_cast<Vec16*>(y + row * cols);
    if constexpr (!kAhead) load(raw, row);
    else if (row + gridDim.x < rows) load(nxt, row + gridDim.x);
    float v[VPT][PV];
    float m = -INFINITY;
#pragma unroll
    for (int k = 0; k < VPT; ++k) {
      const int i = k * THREADS + tid;
      if (i < nvec) {
        Elem<T>::unpack(raw[k], v[k]);
#pragma unroll
        for (int e = 0; e < PV; ++e) m = fmaxf(m, v[k][e]);
      } else {
#pragma unroll
        for (int e = 0; e < PV; ++e) v[k][e] = -INFINITY;
      }
    }
    m = warp_max(m);
    if (lane == 0) red_max[warp] = m;
    __syncthreads();
#pragma unroll
    for (int w = 0; w < NW; ++w) m = fmaxf(m, red_max[w]);
    const float ml = m * kLog2e;
    float s = 0.f;
#pragma unroll
    for (int k = 0; k < VPT; ++k) {
#pragma unroll
      for (int e = 0; e < PV; ++e) {
        const float t = exp_shifted(v[k][e], ml);  // padding: 2^(-inf) = 0
        v[k][e] = t;
        s += t;
      }
    }
    s = warp_sum(s);
    if (lane == 0) red_sum[warp] = s;
    __syncthreads();
    s = 0.f;
#pragma unroll
    for (int w = 0; w < NW; ++w) s += red_sum[w];
    const float inv = 1.0f / s;
#pragma unroll
    for (int k = 0; k < VPT; ++k) {
      const int i = k * THREADS + tid;
      if (i < nvec) {
#pragma unroll
        for (int e = 0; e < PV; ++e) v[k][e] *= inv;
        st_stream(yr + i, Elem<T>::pack(v[k]));
      }
    }
    if constexpr (kAhead) {
#pragma unroll
      for (int k = 0; k < VPT; ++k) raw[k] = nxt[k];
    }
    // red_max is rewritten only after this row's second barrier and red_sum only
    // after the next row's first one, so neither is overwritten while still read.
  }
}

// ---------------------------------------------------------------------------
// Rows of any alignment, and rows too wide for one CTA's registers.
// ---------------------------------------------------------------------------
// A row that starts anywhere is covered by the 16-byte vectors of memory it touches: `head` elements of the first one
// belong to the row before, and the last one may end in the next row.  All vectors but those two are whole and are
// moved with 128-bit accesses; of those two only the row's own elements are loaded and stored, one by one.
template <typename T>
__device__ __forceinline__ T minus_infinity() {
  if constexpr (sizeof(T) == 4) return -INFINITY;
  else if constexpr (std::is_same<T, __half>::value) return __ushort_as_half(0xfc00);
  else return __ushort_as_bfloat16(0xff80);
}
template <typename T>
struct RowSpan {
  const T* base;  // address of the first vector (16-byte aligned)
  int32_t head;   // elements of it before the row
  int32_t end;    // head + cols
  __device__ __forceinline__ RowSpan(const T* row, int32_t cols) {
    head = static_cast<int32_t>((reinterpret_cast<uintptr_t>(row) & 15u) / sizeof(T));
    base = row - head;
    end = head + cols;
  }
  __device__ __forceinline__ bool whole(int32_t e0) const { return e0 >= head && e0 + Elem<T>::kPerVec <= end; }
  // vector i; elements outside the row, and every element when the row has no vector i, are -inf
  template <bool kKeep = false>
  __device__ __forceinline__ Vec16 load(int32_t i) const {
    constexpr int PV = Elem<T>::kPerVec;
    const int32_t e0 = i * PV;
    if (whole(e0)) return kKeep ? ld_keep(reinterpret_cast<const Vec16*>(base + e0)) : ld_stream(reinterpret_cast<const Vec16*>(base + e0));
    T e[PV];
#pragma unroll
    for (int j = 0; j < PV; ++j) e[j] = (e0 + j >= head && e0 + j < end) ? base[e0 + j] : minus_infinity<T>();
    Vec16 v;
#pragma unroll
    for (int w = 0; w < 4; ++w) {
      if constexpr (sizeof(T) == 4) {
        v.w[w] = __float_as_uint(e[w]);
      } else {
        v.w[w] = *reinterpret_cast<const unsigned short*>(&e[2 * w]) |
                 (static_cast<uint32_t>(*reinterpret_cast<const unsigned short*>(&e[2 * w + 1])) << 16);
      }
    }
    return v;
  }
  // to the same place of a row of y that lies at the same offset from a 16-byte boundary
  __device__ __forceinline__ void store(T* y_base, int32_t i, const float* f) const {
    constexpr int PV = Elem<T>::kPerVec;
    const int32_t e0 = i * PV;
    if (whole(e0)) {
      st_stream(reinterpret_cast<Vec16*>(y_base + e0), Elem<T>::pack(f));
    } else {
#pragma unroll
      for (int j = 0; j < PV; ++j)
        if (e0 + j >= head && e0 + j < end) Elem<T>::store1(y_base + e0 + j, f[j]);
    }
  }
};
// exp(x - m), the difference taken first: exact where x is close to m, and a row whose every element is the type's
// lowest value (a mask) keeps its uniform answer.  f32 results by expf; 16-bit ones are rounded to 8 or 11 bits.
template <typename T>
__device__ __forceinline__ float exp_diff(float x, float m) {
  if (sizeof(T) == 4) return expf(x - m);
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"((x - m) * kLog2e));
  return y;
}

// One warp per row, as softmax_rows_warp, for rows that do not start on 16-byte boundaries (up to 32 * CHUNKS vectors).
// 18552 rows of 151 f32: 48 us on the scalar kernel, 6.3 here.
template <typename T, int CHUNKS, int WARPS>
__global__ void __launch_bounds__(WARPS * 32)
softmax_rows_warp_any(const T* __restrict__ x, T* __restrict__ y, int64_t rows, int32_t cols) {
  ptx::launch_dependents_if_few();
  x = ptx::wait_prior_grid(x);
  constexpr int PV = Elem<T>::kPerVec;
  const int lane = threadIdx.x & 31;
  const int64_t row = static_cast<int64_t>(blockIdx.x) * WARPS + (threadIdx.x >> 5);
  if (row >= rows) return;
  const RowSpan<T> span(x + row * cols, cols);
  T* y_base = y + row * cols - span.head;
  float v[CHUNKS][PV];
  float m = -INFINITY;
#pragma unroll
  for (int c = 0; c < CHUNKS; ++c) {
    Elem<T>::unpack(span.load(c * 32 + lane), v[c]);
#pragma unroll
    for (int e = 0; e < PV; ++e) m = fmaxf(m, v[c][e]);
  }
  m = warp_max(m);
  float s = 0.f;
#pragma unroll
  for (int c = 0; c < CHUNKS; ++c)
#pragma unroll
    for (int e = 0; e < PV; ++e) {
      v[c][e] = expf(v[c][e] - m);
      s += v[c][e];
    }
  const float inv = 1.0f / warp_sum(s);
#pragma unroll
  for (int c = 0; c < CHUNKS; ++c) {
#pragma unroll
    for (int e = 0; e < PV; ++e) v[c][e] *= inv;
    span.store(y_base, c * 32 + lane, v[c]);
  }
}

// One CTA per row, as softmax_rows_cta, for rows that do not start on 16-byte boundaries (up to THREADS * VPT vectors), in
// registers.  One barrier per row: every warp takes the exponentials against its own maximum and leaves (maximum, sum);
// after the barrier each folds all pairs into its factor.  The loads of the next row are in flight meanwhile.
template <typename T, int VPT, int THREADS>
__global__ void __launch_bounds__(THREADS)
softmax_rows_cta_any(const T* __restrict__ x, T* __restrict__ y, int64_t rows, int32_t cols) {
  ptx::launch_dependents_if_few();
  x = ptx::wait_prior_grid(x);
  constexpr int PV = Elem<T>::kPerVec;
  constexpr int NW = THREADS / 32;
  __shared__ float2 slots[2][NW];  // alternating: a slot is rewritten after the next row's barrier at the earliest
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  Vec16 raw[VPT];
  int64_t row = blockIdx.x;
  if (row < rows) {
    const RowSpan<T> span(x + row * cols, cols);
#pragma unroll
    for (int k = 0; k < VPT; ++k) raw[k] = span.load(k * THREADS + tid);
  }
  for (int parity = 0; row < rows; row += gridDim.x, parity ^= 1) {
    const RowSpan<T> span(x + row * cols, cols);
    float v[VPT][PV];
    float m = -INFINITY;
#pragma unroll
    for (int k = 0; k < VPT; ++k) {
      Elem<T>::unpack(raw[k], v[k]);
#pragma unroll
      for (int e = 0; e < PV; ++e) m = fmaxf(m, v[k][e]);
    }
    if (row + gridDim.x < rows) {
      const RowSpan<T> next(x + (row + gridDim.x) * cols, cols);
#pragma unroll
      for (int k = 0; k < VPT; ++k) raw[k] = next.load(k * THREADS + tid);
    }
    m = warp_max(m);
    const float m_safe = m == -INFINITY ? 0.f : m;  // nothing but -inf in this warp: its exponentials are 0, not NaN
    float s = 0.f;
#pragma unroll
    for (int k = 0; k < VPT; ++k)
#pragma unroll
      for (int e = 0; e < PV; ++e) {
        v[k][e] = exp_diff<T>(v[k][e], m_safe);
        s += v[k][e];
      }
    s = warp_sum(s);
    if (lane == 0) slots[parity][warp] = make_float2(m, s);
    __syncthreads();
    float gm = -INFINITY, gs = 0.f;
#pragma unroll
    for (int w = 0; w < NW; ++w) gm = fmaxf(gm, slots[parity][w].x);
#pragma unroll
    for (int w = 0; w < NW; ++w) {
      const float2 p = slots[parity][w];
      gs += p.x == -INFINITY ? p.y : p.y * expf(p.x - gm);  // a warp of -inf adds its 0 (or the NaN it met)
    }
    // a row of nothing but -inf: 0 * (1 / 0) = NaN, as exp(-inf + inf) is
    const float factor = m == -INFINITY ? 1.0f / gs : expf(m - gm) / gs;
    T* y_base = y + row * cols - span.head;
#pragma unroll
    for (int k = 0; k < VPT; ++k) {
#pragma unroll
      for (int e = 0; e < PV; ++e) v[k][e] *= factor;
      span.store(y_base, k * THREADS + tid, v[k]);
    }
  }
}

// One CTA per row of any width and alignment, the row read twice, the second time from the L2 as long as the rows in flight fit
// half of it (one row per SM: 450 KB; wider rows come from HBM twice): online maximum and sum per thread, then the exponentials
// again.  No copy of the row in shared memory or registers: several CTAs per SM are in different phases, and HBM reads,
// exponentials and writes overlap (2000 rows of 16392 bf16: 44.8 us with the row in shared memory, 30.9 here).
// kSkip: a thread's steps of four vectors end with the row (with 1024 threads a row of 1100 vectors would otherwise be four times
// as much work); for rows that fill their steps the test costs 7 % and is left out.
constexpr int kTwiceUnroll = 4;
template <typename T, int THREADS, bool kSkip>
__global__ void __launch_bounds__(THREADS, 1024 / THREADS)
softmax_rows_twice(const T* __restrict__ x, T* __restrict__ y, int64_t rows, int32_t cols) {
  // no launch_dependents: the CTAs of a next call would take the places that become free while others still have a row to go (2000 x
  // 16392 bf16 in a row of calls 33.3 us with it, 31.4 without)
  x = ptx::wait_prior_grid(x);
  constexpr int PV = Elem<T>::kPerVec;
  constexpr int NW = THREADS / 32;
  constexpr int UNROLL = kTwiceUnroll;
  __shared__ float2 slots[2][NW];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  int parity = 0;
  for (int64_t row = blockIdx.x; row < rows; row += gridDim.x, parity ^= 1) {
    const RowSpan<T> span(x + row * cols, cols);
    const int32_t nvec = (span.end + PV - 1) / PV;
    float m = -INFINITY, s = 0.f;
    for (int32_t i0 = tid; i0 < nvec; i0 += UNROLL * THREADS) {
      Vec16 raw[UNROLL];
#pragma unroll
      for (int u = 0; u < UNROLL; ++u)
        if (!kSkip || i0 + u * THREADS < nvec) raw[u] = span.template load<true>(i0 + u * THREADS);
#pragma unroll
      for (int u = 0; u < UNROLL; ++u) {
        if (kSkip && i0 + u * THREADS >= nvec) break;
        float f[PV];
        Elem<T>::unpack(raw[u], f);
        float mv = f[0];
#pragma unroll
        for (int e = 1; e < PV; ++e) mv = fmaxf(mv, f[e]);
        if (mv > m) {
          s *= exp_diff<T>(m, mv);  // 0 while m = -inf
          m = mv;
        }
        const float m_safe = m == -INFINITY ? 0.f : m;
#pragma unroll
        for (int e = 0; e < PV; ++e) s += exp_diff<T>(f[e], m_safe);
      }
    }
    const float wm = warp_max(m);
    s = warp_sum(m == -INFINITY ? s : s * expf(m - wm));  // a thread of -inf adds its 0 (or the NaN it met)
    if (lane == 0) slots[parity][warp] = make_float2(wm, s);
    __syncthreads();  // slots[parity] is rewritten after the next row's barrier at the earliest
    const float2 mine = lane < NW ? slots[parity][lane] : make_float2(-INFINITY, 0.f);
    const float gm = warp_max(mine.x);
    const float gs = warp_sum(mine.x == -INFINITY ? mine.y : mine.y * expf(mine.x - gm));
    const float inv = 1.0f / gs;  // a row of nothing but -inf: exp(-inf + inf) = NaN below
    T* y_base = y + row * cols - span.head;
    for (int32_t i0 = tid; i0 < nvec; i0 += UNROLL * THREADS) {
      Vec16 raw[UNROLL];
#pragma unroll
      for (int u = 0; u < UNROLL; ++u)
        if (!kSkip || i0 + u * THREADS < nvec) raw[u] = span.load(i0 + u * THREADS);
#pragma unroll
      for (int u = 0; u < UNROLL; ++u) {
        if (kSkip && i0 + u * THREADS >= nvec) break;
        float f[PV];
        Elem<T>::unpack(raw[u], f);
#pragma unroll
        for (int e = 0; e < PV; ++e) f[e] = exp_diff<T>(f[e], gm) * inv;
        span.store(y_base, i0 + u * THREADS, f);
      }
    }
  }
}

// A cluster of 2 .. 8 CTAs per row, VPT 16-byte vectors per thread in registers (vector (k * ctas + rank) * THREADS +
// tid), any alignment: the form for a few wide rows (8 rows of 128000 16-bit values: 42 us with a CTA per row, 6.4 with
// eight).  With rows enough for all SMs the exchange between CTAs costs more than it gives (1000 rows of 50001: 132 us).
// Every warp takes the exponentials against its OWN maximum and leaves (maximum, sum); after one barrier each warp of the
// cluster reads all pairs through distributed shared memory and folds them into its factor exp(m_warp - m_row) / sum_row.
template <typename T, int VPT, int THREADS>
__global__ void __launch_bounds__(THREADS)
softmax_rows_cluster(const T* __restrict__ x, T* __restrict__ y, int64_t rows, int32_t cols) {
  ptx::launch_dependents_if_few();
  x = ptx::wait_prior_grid(x);
  constexpr int PV = Elem<T>::kPerVec;
  constexpr int NW = THREADS / 32;
  __shared__ float2 slots[NW];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const uint32_t ctas = ptx::cluster_nctarank(), rank = ptx::cluster_ctarank();
  const int64_t row = blockIdx.x / ctas;  // grid = rows * ctas
  const RowSpan<T> span(x + row * cols, cols);
  Vec16 raw[VPT];
#pragma unroll
  for (int k = 0; k < VPT; ++k) raw[k] = span.load((k * ctas + rank) * THREADS + tid);
  float v[VPT][PV];
  float m = -INFINITY;
#pragma unroll
  for (int k = 0; k < VPT; ++k) {
    Elem<T>::unpack(raw[k], v[k]);
#pragma unroll
    for (int e = 0; e < PV; ++e) m = fmaxf(m, v[k][e]);
  }
  m = warp_max(m);
  const float m_safe = m == -INFINITY ? 0.f : m;  // nothing but -inf in this warp: its exponentials are 0, not NaN
  float s = 0.f;
#pragma unroll
  for (int k = 0; k < VPT; ++k)
#pragma unroll
    for (int e = 0; e < PV; ++e) {
      v[k][e] = exp_diff<T>(v[k][e], m_safe);
      s += v[k][e];
    }
  s = warp_sum(s);
  if (lane == 0) slots[warp] = make_float2(m, s);
  ptx::cluster_sync_all();
  float gm = -INFINITY, gs = 0.f;
  float2 pair[(8 * NW + 31) / 32];
#pragma unroll
  for (int j = 0; j < (8 * NW + 31) / 32; ++j) {
    const int i = j * 32 + lane;
    pair[j] = make_float2(-INFINITY, 0.f);
    if (i < static_cast<int>(ctas) * NW) pair[j] = ptx::ld_shared_cluster_f32x2(ptx::mapa_shared(ptx::smem_u32(&slots[i % NW]), i / NW));
    gm = fmaxf(gm, pair[j].x);
  }
  gm = warp_max(gm);
#pragma unroll
  for (int j = 0; j < (8 * NW + 31) / 32; ++j)
    gs += pair[j].x == -INFINITY ? pair[j].y : pair[j].y * expf(pair[j].x - gm);  // a warp of -inf adds its 0 (or the NaN it met)
  gs = warp_sum(gs);
  // a row of nothing but -inf: 0 * (1 / 0) = NaN, as exp(-inf + inf) is
  const float factor = m == -INFINITY ? 1.0f / gs : expf(m - gm) / gs;
  T* y_base = y + row * cols - span.head;
#pragma unroll
  for (int k = 0; k < VPT; ++k) {
#pragma unroll
    for (int e = 0; e < PV; ++e) v[k][e] *= factor;
    span.store(y_base, (k * ctas + rank) * THREADS + tid, v[k]);
  }
  ptx::cluster_sync_all();  // nobody leaves while its pairs may still be read
}

// max or sum over a CTA
template <int THREADS>
__device__ __forceinline__ float block_reduce(float v, float* red, bool is_max) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  v = is_max ? warp_max(v) : warp_sum(v);
  __syncthreads();  // red[] may still be read from a previous reduction
  if (lane == 0) red[warp] = v;
  __syncthreads();
  float r = (lane < THREADS / 32) ? red[lane] : (is_max ? -INFINITY : 0.f);
  r = is_max ? warp_max(r) : warp_sum(r);
  return r;
}

// ---------------------------------------------------------------------------
// Any width, any alignment: scalar accesses, online (max, sum) in pass one.
// ---------------------------------------------------------------------------
template <typename T, int THREADS>
__global__ void __launch_bounds__(THREADS)
softmax_rows_stream(const T* __restrict__ x, T* __restrict__ y, int64_t rows, int64_t cols) {
  x = ptx::wait_prior_grid(x);
  __shared__ float red[32];
  for (int64_t row = blockIdx.x; row < rows; row += gridDim.x) {
    const T* xr = x + row * cols;
    T* yr = y + row * cols;
    float m = -INFINITY, s = 0.f;
    for (int64_t i = threadIdx.x; i < cols; i += THREADS) {
      const float f = Elem<T>::load1(xr + i);
      if (f > m) {
        s = s * expf(m - f);  // m = -inf on the first element: s is 0, expf(-inf) = 0
        m = f;
      }
      s += expf(f - m);
    }
    const float gm = block_reduce<THREADS>(m, red, true);
    // a thread that saw no element has m = -inf and s = 0: contributes 0
    s = (m == -INFINITY) ? 0.f : s * expf(m - gm);
    s = block_reduce<THREADS>(s, red, false);
    const float inv = 1.0f / s;
    for (int64_t i = threadIdx.x; i < cols; i += THREADS)
      Elem<T>::store1(yr + i, expf(Elem<T>::load1(xr + i) - gm) * inv);
  }
}

}  // namespace softmax
}  // namespace tsm100
