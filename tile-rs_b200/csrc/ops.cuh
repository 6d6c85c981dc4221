// Host-side launch logic for the three operators: argument validation, kernel
// selection, tensor-map construction, launch.  Header-only so that both the
// library (capi_ops.cu) and the translation units the cuda_sm100 target emits
// instantiate the same kernels with the same dispatch.
//
// Every function returns a TSM100_* status and, on failure, writes a message
// to *err.  Nothing here synchronises; the operators that need device scratch (operand
// planes of the tcgen05 f32 kernels, padded copies, partial results) take it from, and
// return it to, the library's own memory pool on the caller's stream (scratch.hpp).
#pragma once

#include <cuda.h>
#include <cuda_runtime.h>

#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstring>
#include <map>
#include <mutex>
#include <string>
#include <tuple>
#include <type_traits>
#include <utility>

#include "../../include/tile_sm100.h"
#include "attention_decode.cuh"
#include "attention_decode_stream.cuh"
#include "attention_f32_tc.cuh"
#include "attention_narrow.cuh"
#include "attention_simt.cuh"
#include "attention_tc.cuh"
#include "attention_tf32x3.cuh"
#include "ewise.cuh"
#include "gemm_f32_fused.cuh"
#include "gemm_pad.cuh"
#include "gemm_simt.cuh"
#include "gemm_skinny.cuh"
#include "gemm_tc.cuh"
#include "gemm_tc2.cuh"
#include "gemm_tf32_tc.cuh"
#include "gemm_tf32x3.cuh"
#include "route.hpp"
#include "rowops.cuh"
#include "scratch.hpp"
#include "softmax.cuh"

namespace tsm100 {
namespace ops {

inline int32_t op_fail(std::string* err, int32_t code, const std::string& msg) {
  if (err) *err = msg;
  return code;
}

inline int32_t cuda_ok(std::string* err, cudaError_t e, const char* what) {
  if (e == cudaSuccess) return TSM100_OK;
  const int32_t code = (e == cudaErrorNoDevice || e == cudaErrorInsufficientDriver) ? TSM100_ERR_NO_DEVICE
                                                                                      : TSM100_ERR_LAUNCH;
  return op_fail(err, code, std::string(what) + " failed: " + cudaGetErrorString(e));
}

// What an operator's launch function answers, without a message, when the pool cannot give it the scratch it would like
// and a form without scratch exists: the dispatch then takes that one.
constexpr int32_t kNoScratch = -1;
inline int32_t take_scratch(std::string* err, void** ws, size_t bytes, cudaStream_t s) {
  const cudaError_t e = scratch::take(ws, bytes, s);
  if (e == cudaErrorMemoryAllocation || e == cudaErrorNotSupported) {
    (void)cudaGetLastError();
    return kNoScratch;
  }
  return cuda_ok(err, e, "scratch from the library's memory pool");
}

inline size_t dtype_size(int32_t dtype) { return dtype == TSM100_F32 ? 4 : 2; }
inline bool dtype_valid(int32_t dtype) { return dtype == TSM100_F32 || dtype == TSM100_F16 || dtype == TSM100_BF16; }
inline bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }

// ---------------------------------------------------------------------------
// per-(kernel, device) facts: asked of the CUDA runtime once, then remembered
// ---------------------------------------------------------------------------
// cudaFuncSetAttribute and the occupancy queries cost a few microseconds each, which is as long as
// a small launch itself; their answers depend on the kernel and the device only.
struct KernelFacts {
  std::mutex mu;
  std::map<std::tuple<const void*, int, int>, int> value;  // (kernel, device, what) -> answer
};
inline KernelFacts& kernel_facts() {
  static KernelFacts f;
  return f;
}
enum { kFactSmemSet = 1, kFactNonPortableSet = 2, kFactBlocksPerSm = 3, kFactClusters = 4 };

// `compute` returns (ok, answer); an answer is remembered only when ok.
template <typename F>
inline bool kernel_fact(const void* kern, int what, int* answer, F compute) {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) dev = -1;
  KernelFacts& f = kernel_facts();
  const auto key = std::make_tuple(kern, dev, what);
  {
    std::lock_guard<std::mutex> lock(f.mu);
    auto it = f.value.find(key);
    if (it != f.value.end()) {
      *answer = it->second;
      return true;
    }
  }
  if (!compute(answer)) return false;
  std::lock_guard<std::mutex> lock(f.mu);
  f.value[key] = *answer;
  return true;
}

// cudaFuncAttributeMaxDynamicSharedMemorySize, set once per kernel and device.
template <typename K>
inline cudaError_t set_dyn_smem_once(K kern, int bytes) {
  cudaError_t e = cudaSuccess;
  int unused = 0;
  kernel_fact(reinterpret_cast<const void*>(kern), kFactSmemSet, &unused, [&](int* out) {
    e = cudaFuncSetAttribute(reinterpret_cast<const void*>(kern), cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    *out = bytes;
    return e == cudaSuccess;
  });
  return e;
}
template <typename K>
inline cudaError_t allow_wide_clusters_once(K kern) {
  cudaError_t e = cudaSuccess;
  int unused = 0;
  kernel_fact(reinterpret_cast<const void*>(kern), kFactNonPortableSet, &unused, [&](int* out) {
    e = cudaFuncSetAttribute(reinterpret_cast<const void*>(kern), cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    *out = 1;
    return e == cudaSuccess;
  });
  return e;
}
// Launches a kernel in clusters of `cluster` CTAs where that is not 0; chained: as a programmatic dependent of the one before it in
// the stream (the rules that such kernels keep are in ptx.cuh).  What that saves is the time between two kernels of a chain of calls:
// the end of one grid, the launch of the next and its set-up run side by side.  bf16 MLP of 16 tokens, 4096 x 16384: 84.1 us, 78.1
// chained and with the weights' first tiles fetched meanwhile; one token of one sequence of 32768, with rotation and appends: 38.1 / 36.3, of
// 1000 18.8 / 14.1; 16 x 4096 x 4096 in a row of calls 8.9 / 8.4 (all as graph replays).
template <typename... P, typename... A>
inline cudaError_t launch_kernel(bool chained, void (*kern)(P...), dim3 grid, unsigned threads, size_t smem, cudaStream_t s, unsigned cluster, A&&... args) {
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute attr[2];
  unsigned n = 0;
  if (cluster) {
    attr[n].id = cudaLaunchAttributeClusterDimension;
    attr[n].val.clusterDim.x = cluster;
    attr[n].val.clusterDim.y = 1;
    attr[n].val.clusterDim.z = 1;
    ++n;
  }
  if (chained) {
    attr[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[n].val.programmaticStreamSerializationAllowed = 1;
    ++n;
  }
  cfg.attrs = attr;
  cfg.numAttrs = n;
  cfg.gridDim = grid;
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  return cudaLaunchKernelEx(&cfg, kern, std::forward<A>(args)...);
}
template <typename... P, typename... A>
inline cudaError_t launch_chained(void (*kern)(P...), dim3 grid, unsigned threads, size_t smem, cudaStream_t s, unsigned cluster, A&&... args) {
  return launch_kernel(true, kern, grid, threads, smem, s, cluster, std::forward<A>(args)...);
}
// How many clusters of `cluster` CTAs of a kernel the GPU holds at once, asked once per kernel and device; `fallback` if it cannot tell.
template <typename K>
inline int resident_clusters(K kern, unsigned threads, size_t smem, unsigned cluster, unsigned grid, int fallback) {
  int answer = fallback;
  kernel_fact(reinterpret_cast<const void*>(kern), kFactClusters, &answer, [&](int* out) {
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = cluster;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    int n = 0;
    if (cudaOccupancyMaxActiveClusters(&n, kern, &cfg) != cudaSuccess || n < 1) {
      (void)cudaGetLastError();
      return false;
    }
    *out = n;
    return true;
  });
  return answer;
}
// Resident CTAs per SM of a kernel launched with `threads` threads and no dynamic shared memory (at least 1).
template <typename K>
inline int blocks_per_sm(K kern, int threads) {
  int per_sm = 1;
  kernel_fact(reinterpret_cast<const void*>(kern), kFactBlocksPerSm + (threads << 8), &per_sm, [&](int* out) {
    int n = 1;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, kern, threads, 0) != cudaSuccess || n < 1) {
      (void)cudaGetLastError();
      return false;
    }
    *out = n;
    return true;
  });
  return per_sm < 1 ? 1 : per_sm;
}

// ---------------------------------------------------------------------------
// tensor maps
// ---------------------------------------------------------------------------
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

inline int32_t encode_fn(std::string* err, EncodeTiledFn* out) {
  static EncodeTiledFn cached = nullptr;
  if (!cached) {
    void* fn = nullptr;
    cudaDriverEntryPointQueryResult qres;
    cudaError_t e = cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &qres);
    if (e != cudaSuccess || qres != cudaDriverEntryPointSuccess || !fn)
      return op_fail(err, TSM100_ERR_NO_DEVICE, "cuTensorMapEncodeTiled is not available from the CUDA driver");
    cached = reinterpret_cast<EncodeTiledFn>(fn);
  }
  *out = cached;
  return TSM100_OK;
}

// A map is a pure function of its arguments, and a repeated launch (same pointers, same shape) asks for the same
// ones again: each thread keeps the last few it encoded.
struct TmapKey {
  const void* base;
  uint64_t dim[4], stride[3];  // stride: bytes; dimension 0 is contiguous
  uint32_t box[4];
  int32_t dtype, rank;
};
struct TmapSlot {
  TmapKey key;
  CUtensorMap map;
  bool used = false;
};

// `key` all zeros beyond its rank.  128-byte swizzle (64-byte where a row of the box has 64 bytes), out-of-range elements read as zero.
inline int32_t make_tmap(std::string* err, CUtensorMap* out, const TmapKey& key, uint32_t elem_bytes) {
  constexpr int kSlots = 16;
  static thread_local TmapSlot cache[kSlots];
  static thread_local int next = 0;
  for (int i = 0; i < kSlots; ++i)
    if (cache[i].used && std::memcmp(&cache[i].key, &key, sizeof key) == 0) {
      *out = cache[i].map;
      return TSM100_OK;
    }
  EncodeTiledFn fn;
  int32_t st = encode_fn(err, &fn);
  if (st != TSM100_OK) return st;
  cuuint64_t dims[4], strides[3];
  cuuint32_t box[4], estr[4] = {1, 1, 1, 1};
  for (int i = 0; i < key.rank; ++i) dims[i] = key.dim[i], box[i] = key.box[i];
  for (int i = 0; i + 1 < key.rank; ++i) {
    strides[i] = key.stride[i];
    if (strides[i] & 15u) return op_fail(err, TSM100_ERR_INVALID, "tensor map needs a 16-byte aligned base and 16-byte-multiple strides");
  }
  if (!aligned16(key.base)) return op_fail(err, TSM100_ERR_INVALID, "tensor map needs a 16-byte aligned base and 16-byte-multiple strides");
  CUresult r = fn(out, static_cast<CUtensorMapDataType>(key.dtype), static_cast<cuuint32_t>(key.rank), const_cast<void*>(key.base), dims, strides, box, estr,
                  CU_TENSOR_MAP_INTERLEAVE_NONE, box[0] * elem_bytes == 64 ? CU_TENSOR_MAP_SWIZZLE_64B : CU_TENSOR_MAP_SWIZZLE_128B,
                  CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) {
    char buf[96];
    snprintf(buf, sizeof buf, "cuTensorMapEncodeTiled failed: CUresult %d", static_cast<int>(r));
    return op_fail(err, TSM100_ERR_LAUNCH, buf);
  }
  TmapSlot& slot = cache[next];
  next = (next + 1) % kSlots;
  slot.key = key;
  slot.map = *out;
  slot.used = true;
  return TSM100_OK;
}
// dims (x contiguous, y, z), strides in elements of `elem_bytes`, box (box_x, box_y, 1).
inline int32_t make_tmap_3d(std::string* err, CUtensorMap* out, const void* base, uint64_t dim_x, uint64_t dim_y,
                            uint64_t dim_z, uint64_t stride_y, uint64_t stride_z, uint32_t box_x, uint32_t box_y,
                            CUtensorMapDataType dtype, uint32_t elem_bytes) {
  TmapKey key;
  std::memset(&key, 0, sizeof key);
  key.base = base;
  key.dim[0] = dim_x, key.dim[1] = dim_y, key.dim[2] = dim_z;
  key.stride[0] = stride_y * elem_bytes, key.stride[1] = stride_z * elem_bytes;
  key.box[0] = box_x, key.box[1] = box_y, key.box[2] = 1;
  key.dtype = static_cast<int32_t>(dtype), key.rank = 3;
  return make_tmap(err, out, key, elem_bytes);
}

// 16-bit elements (bf16 or f16).
inline int32_t make_tmap_16bit_3d(std::string* err, CUtensorMap* out, const void* base, uint64_t dim_x,
                                  uint64_t dim_y, uint64_t dim_z, uint64_t stride_y, uint64_t stride_z,
                                  uint32_t box_x, uint32_t box_y, bool is_bf16) {
  return make_tmap_3d(err, out, base, dim_x, dim_y, dim_z, stride_y, stride_z, box_x, box_y,
                      is_bf16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2);
}

inline int32_t sm_count(std::string* err, int* sms) {
  static int cached[64] = {0};
  int dev = 0;
  int32_t st = cuda_ok(err, cudaGetDevice(&dev), "cudaGetDevice");
  if (st != TSM100_OK) return st;
  if (dev < 64 && cached[dev]) {
    *sms = cached[dev];
    return TSM100_OK;
  }
  int n = 0;
  st = cuda_ok(err, cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev), "cudaDeviceGetAttribute");
  if (st != TSM100_OK) return st;
  if (dev < 64) cached[dev] = n;
  *sms = n;
  return TSM100_OK;
}

// ---------------------------------------------------------------------------
// softmax
// ---------------------------------------------------------------------------
template <typename T, int CHUNKS>
inline cudaError_t launch_softmax_warp(const T* x, T* y, int64_t rows, int32_t cols, cudaStream_t s) {
  constexpr int WARPS = 4;
  const int64_t grid = (rows + WARPS - 1) / WARPS;
  return launch_chained(softmax::softmax_rows_warp<T, CHUNKS, WARPS>, static_cast<unsigned>(grid), WARPS * 32, 0, s, 0, x, y, rows, cols);
}

// As many CTAs per row as its vectors need, one cluster per row.
template <typename T, int VPT, int THREADS>
inline int32_t softmax_cluster_launch(std::string* err, const T* x, T* y, int64_t rows, int64_t cols, int64_t ctas, cudaStream_t s) {
  return cuda_ok(err, launch_chained(softmax::softmax_rows_cluster<T, VPT, THREADS>, static_cast<unsigned>(rows * ctas), THREADS, 0, s,
                                     static_cast<unsigned>(ctas), x, y, rows, static_cast<int32_t>(cols)),
                 "softmax_rows_cluster launch");
}

template <typename T>
inline int32_t softmax_typed(std::string* err, const T* x, T* y, int64_t rows, int64_t cols, cudaStream_t s) {
  constexpr int PV = softmax::Elem<T>::kPerVec;
  const bool vec_ok = (cols % PV == 0) && aligned16(x) && aligned16(y);
  const int64_t nvec = cols / PV;
  cudaError_t e;
  if (vec_ok && nvec <= 32 * 8 && rows <= 4ll * 0x7fffffff) {  // one warp per row
    const int32_t c = static_cast<int32_t>(cols);
    if (nvec <= 32 * 1) e = launch_softmax_warp<T, 1>(x, y, rows, c, s);
    else if (nvec <= 32 * 2) e = launch_softmax_warp<T, 2>(x, y, rows, c, s);
    else if (nvec <= 32 * 4) e = launch_softmax_warp<T, 4>(x, y, rows, c, s);
    else e = launch_softmax_warp<T, 8>(x, y, rows, c, s);
    return cuda_ok(err, e, "softmax_rows_warp launch");
  }
  if (vec_ok && nvec <= 256 * 8) {  // 128 or 256 threads per row, 32 values each
    int sms_cta = 0;
    int32_t st_cta = sm_count(err, &sms_cta);
    if (st_cta != TSM100_OK) return st_cta;
    const int32_t c = static_cast<int32_t>(cols);
    // f32: a row to a CTA; 16-bit: two, as soon as there are more rows than CTAs at once (softmax.cuh)
    auto launch = [&](auto kern, int threads) {
      int64_t ctas = rows;
      if (sizeof(T) == 2) {
        const int64_t resident = static_cast<int64_t>(sms_cta) * blocks_per_sm(kern, threads);
        if (rows > resident) ctas = std::max(resident, (rows + 1) / 2);
      }
      const unsigned grid = static_cast<unsigned>(std::min<int64_t>(ctas, 0x7fffffff));
      e = launch_chained(kern, grid, threads, 0, s, 0, x, y, rows, c);
    };
    if (nvec <= 128 * 4) launch(softmax::softmax_rows_cta<T, 4, 128>, 128);
    else if (nvec <= 128 * 8) launch(softmax::softmax_rows_cta<T, 8, 128>, 128);
    else launch(softmax::softmax_rows_cta<T, 8, 256>, 256);
    return cuda_ok(err, e, "softmax_rows_cta launch");
  }
  int sms = 0;
  int32_t st = sm_count(err, &sms);
  if (st != TSM100_OK) return st;
  // Rows that start anywhere, or too wide for one CTA's registers.  x and y must lie at the same offset from a 16-byte
  // boundary, in every row alike (their row pitch is the same), a whole number of elements away from it.
  const uintptr_t xa = reinterpret_cast<uintptr_t>(x), ya = reinterpret_cast<uintptr_t>(y);
  const int64_t span = (cols + 2 * PV - 2) / PV;  // the most 16-byte vectors a row can touch
  if (((xa ^ ya) & 15u) == 0 && xa % sizeof(T) == 0 && cols <= 1 << 30) {
    const int32_t c = static_cast<int32_t>(cols);
    if (route::softmax_row_per_warp(span, rows, sms) && rows <= 4ll * 0x7fffffff) {
      constexpr int WARPS = 4;
      const unsigned grid = static_cast<unsigned>((rows + WARPS - 1) / WARPS);
      if (span <= 32 * 2) e = launch_chained(softmax::softmax_rows_warp_any<T, 2, WARPS>, grid, WARPS * 32, 0, s, 0, x, y, rows, c);
      else if (span <= 32 * 4) e = launch_chained(softmax::softmax_rows_warp_any<T, 4, WARPS>, grid, WARPS * 32, 0, s, 0, x, y, rows, c);
      else e = launch_chained(softmax::softmax_rows_warp_any<T, 8, WARPS>, grid, WARPS * 32, 0, s, 0, x, y, rows, c);
      return cuda_ok(err, e, "softmax_rows_warp_any launch");
    }
    // up to 1024 vectors a row stays in registers: 8000 rows of 3501 bf16 78 us scalar, 66 read twice, 27 here; 3000 of 1111
    // f32 17 / 23 / 8.5; 4000 of 8001 bf16 70 / 32 / 29
    if (span <= 256 * 4) {
      auto launch = [&](auto kern, int threads) {
        const unsigned grid = static_cast<unsigned>(std::min<int64_t>(rows, static_cast<int64_t>(sms) * blocks_per_sm(kern, threads)));
        e = launch_chained(kern, grid, threads, 0, s, 0, x, y, rows, c);
      };
      if (span <= 128 * 4) launch(softmax::softmax_rows_cta_any<T, 4, 128>, 128);
      else launch(softmax::softmax_rows_cta_any<T, 4, 256>, 256);
      return cuda_ok(err, e, "softmax_rows_cta_any launch");
    }
    if (const int ctas = route::softmax_cluster(span, rows, sms)) {
      if (span <= 8 * 1024) return softmax_cluster_launch<T, 4, 256>(err, x, y, rows, cols, ctas, s);
      return softmax_cluster_launch<T, 8, 512>(err, x, y, rows, cols, ctas, s);
    }
    // one CTA per row.  1000 rows of 50001 bf16: 97 us scalar, 49 here; 1212 of 97648 f32 286 / 214; 2000 of 16392 bf16 (in shared
    // memory) 45 / 31
    const int64_t row_bytes = cols * static_cast<int64_t>(sizeof(T));
    const int threads = route::softmax_twice_threads(row_bytes, rows, sms);
    const unsigned grid = static_cast<unsigned>(std::min<int64_t>(rows, route::softmax_twice_stays(row_bytes, rows, threads, sms) ? sms * (1024ll / threads) : 0x7fffffff));
    auto launch = [&](auto kern) { e = launch_chained(kern, grid, threads, 0, s, 0, x, y, rows, c); };
    if (route::softmax_twice_skip((cols + PV - 1) / PV, threads, softmax::kTwiceUnroll)) {
      if (threads == 256) launch(softmax::softmax_rows_twice<T, 256, true>);
      else if (threads == 512) launch(softmax::softmax_rows_twice<T, 512, true>);
      else launch(softmax::softmax_rows_twice<T, 1024, true>);
    } else {
      if (threads == 256) launch(softmax::softmax_rows_twice<T, 256, false>);
      else if (threads == 512) launch(softmax::softmax_rows_twice<T, 512, false>);
      else launch(softmax::softmax_rows_twice<T, 1024, false>);
    }
    return cuda_ok(err, e, "softmax_rows_twice launch");
  }
  constexpr int THREADS = 512;
  const unsigned grid = static_cast<unsigned>(std::min<int64_t>(rows, static_cast<int64_t>(sms) * 4));
  e = launch_chained(softmax::softmax_rows_stream<T, THREADS>, grid, THREADS, 0, s, 0, x, y, rows, cols);
  return cuda_ok(err, e, "softmax_rows_stream launch");
}

inline int32_t softmax(std::string* err, const tsm100_softmax_desc* d, const void* x, void* y, void* stream) {
  if (!d || !x || !y) return op_fail(err, TSM100_ERR_INVALID, "softmax: null argument");
  if (!dtype_valid(d->dtype)) return op_fail(err, TSM100_ERR_INVALID, "softmax: unknown dtype");
  if (d->rows < 0 || d->cols < 0) return op_fail(err, TSM100_ERR_INVALID, "softmax: negative shape");
  if (d->rows == 0 || d->cols == 0) return TSM100_OK;  // empty tile: nothing to do
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  switch (d->dtype) {
    case TSM100_F32:
      return softmax_typed<float>(err, static_cast<const float*>(x), static_cast<float*>(y), d->rows, d->cols, s);
    case TSM100_BF16:
      return softmax_typed<__nv_bfloat16>(err, static_cast<const __nv_bfloat16*>(x),
                                          static_cast<__nv_bfloat16*>(y), d->rows, d->cols, s);
    default:
      return softmax_typed<__half>(err, static_cast<const __half*>(x), static_cast<__half*>(y), d->rows, d->cols, s);
  }
}

// ---------------------------------------------------------------------------
// rms_norm / row reductions / SiLU * Mul
// ---------------------------------------------------------------------------
template <typename T, int OP>
inline int32_t row_op_typed(std::string* err, const T* x, T* y, int64_t rows, int64_t cols, float eps, cudaStream_t s) {
  namespace ro = rowops;
  constexpr int PV = softmax::Elem<T>::kPerVec;
  const bool vec_ok = (cols % PV == 0) && aligned16(x) && (OP != ro::kRmsNorm || aligned16(y));
  const int64_t nvec = cols / PV;
  int sms = 0;
  int32_t st = sm_count(err, &sms);
  if (st != TSM100_OK) return st;
  cudaError_t e = cudaSuccess;
  // A CTA to a row: two rows, the loads of the second in flight while the first is worked on, as soon as there are more rows than CTAs at once; CTAs
  // that stay for the whole launch drift apart (softmax.cuh).  rms_norm of 65536 x 4096 f32 335 us that way, 312 here, bf16 170 / 158, 100000 x 2600
  // 201 / 165.  A warp to a row: CTAs that stay, 60000 x 256 f32 17.2 us, 17.8 with two rounds each.
  auto launch = [&](auto kern, int threads, int rows_per_cta) {
    const int64_t resident = static_cast<int64_t>(sms) * blocks_per_sm(kern, threads);
    const int64_t want = (rows + rows_per_cta - 1) / rows_per_cta;
    const int64_t most = rows_per_cta == 1 ? std::max(resident, (want + 1) / 2) : resident;
    const unsigned grid = static_cast<unsigned>(std::min<int64_t>({want, most, 0x7fffffff}));
    e = launch_chained(kern, grid, threads, 0, s, 0, x, y, rows, static_cast<int32_t>(cols), eps);
  };
  if (vec_ok && nvec <= 32 * 8) {  // one warp per row, four rows per CTA
    if (nvec <= 32 * 1) launch(ro::row_op_kernel<T, OP, 1, 32, 128>, 128, 4);
    else if (nvec <= 32 * 2) launch(ro::row_op_kernel<T, OP, 2, 32, 128>, 128, 4);
    else if (nvec <= 32 * 4) launch(ro::row_op_kernel<T, OP, 4, 32, 128>, 128, 4);
    else launch(ro::row_op_kernel<T, OP, 8, 32, 128>, 128, 4);
    return cuda_ok(err, e, "row_op_kernel (warp per row) launch");
  }
  if (vec_ok && nvec <= 256 * 8) {  // 128 or 256 threads per row, 32 values each
    if (nvec <= 128 * 4) launch(ro::row_op_kernel<T, OP, 4, 128, 128>, 128, 1);
    else if (nvec <= 128 * 8) launch(ro::row_op_kernel<T, OP, 8, 128, 128>, 128, 1);
    else launch(ro::row_op_kernel<T, OP, 8, 256, 256>, 256, 1);
    return cuda_ok(err, e, "row_op_kernel (CTA per row) launch");
  }
  constexpr int THREADS = 512;
  const unsigned grid = static_cast<unsigned>(std::min<int64_t>(rows, static_cast<int64_t>(sms) * 4));
  e = launch_chained(ro::row_op_stream_kernel<T, OP, THREADS>, grid, THREADS, 0, s, 0, x, y, rows, cols, eps);
  return cuda_ok(err, e, "row_op_stream_kernel launch");
}

template <int OP>
inline int32_t row_op(std::string* err, int32_t dtype, int64_t rows, int64_t cols, float eps, const void* x, void* y,
                      void* stream, const char* what) {
  if (!dtype_valid(dtype)) return op_fail(err, TSM100_ERR_INVALID, std::string(what) + ": unknown dtype");
  if (rows < 0 || cols < 0) return op_fail(err, TSM100_ERR_INVALID, std::string(what) + ": negative shape");
  // an empty tile has no input bytes: its pointer may be anything, a reduction still writes its fill value
  if (!y || (!x && rows > 0 && cols > 0)) return op_fail(err, TSM100_ERR_INVALID, std::string(what) + ": null argument");
  if (rows == 0) return TSM100_OK;
  if (cols == 0 && OP == rowops::kRmsNorm) return TSM100_OK;  // empty tile: nothing to write
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  switch (dtype) {
    case TSM100_F32:
      return row_op_typed<float, OP>(err, static_cast<const float*>(x), static_cast<float*>(y), rows, cols, eps, s);
    case TSM100_BF16:
      return row_op_typed<__nv_bfloat16, OP>(err, static_cast<const __nv_bfloat16*>(x), static_cast<__nv_bfloat16*>(y),
                                              rows, cols, eps, s);
    default:
      return row_op_typed<__half, OP>(err, static_cast<const __half*>(x), static_cast<__half*>(y), rows, cols, eps, s);
  }
}

inline int32_t rms_norm(std::string* err, const tsm100_rms_norm_desc* d, const void* x, void* y, void* stream) {
  if (!d) return op_fail(err, TSM100_ERR_INVALID, "rms_norm: null descriptor");
  return row_op<rowops::kRmsNorm>(err, d->dtype, d->rows, d->cols, d->eps, x, y, stream, "rms_norm");
}

inline int32_t reduce(std::string* err, const tsm100_reduce_desc* d, const void* x, void* y, void* stream) {
  if (!d) return op_fail(err, TSM100_ERR_INVALID, "reduce: null descriptor");
  if (d->kind == TSM100_REDUCE_SUM)
    return row_op<rowops::kReduceSum>(err, d->dtype, d->rows, d->cols, 0.f, x, y, stream, "reduce");
  if (d->kind == TSM100_REDUCE_MAX)
    return row_op<rowops::kReduceMax>(err, d->dtype, d->rows, d->cols, 0.f, x, y, stream, "reduce");
  return op_fail(err, TSM100_ERR_INVALID, "reduce: unknown kind");
}

template <typename T>
inline int32_t silu_mul_typed(std::string* err, const T* gate, const T* up, T* y, int64_t n, cudaStream_t s) {
  namespace ro = rowops;
  constexpr int PV = softmax::Elem<T>::kPerVec;
  // 16-bit data: twice the elements per byte, so twice the threads keep the same bytes in flight (measured: 5.87 -> 6.16 TB/s)
  constexpr int THREADS = sizeof(T) == 2 ? 512 : 256, UNROLL = 4;
  int sms = 0;
  int32_t st = sm_count(err, &sms);
  if (st != TSM100_OK) return st;
  const bool vec_ok = (n % PV == 0) && aligned16(gate) && aligned16(y) && (!up || aligned16(up));
  if (vec_ok) {
    const int64_t nvec = n / PV;
    // Four vectors to a thread, fewer where that leaves SMs without a CTA (MLP of 45 tokens, 1024 x 2048, 19.5 -> 18.8 us), and CTAs that go after
    // one round: 65536 x 4096 f32 534 us in eight to an SM that stay, 456 here, bf16 265 / 238.
    const int64_t want = (nvec + THREADS * UNROLL - 1) / (THREADS * UNROLL), most = (nvec + THREADS - 1) / THREADS;
    const unsigned grid = static_cast<unsigned>(std::max<int64_t>(std::min<int64_t>(most, sms), std::min<int64_t>(want, 0x7fffffff)));
    auto kern = up ? ro::silu_mul_kernel<T, true, UNROLL, THREADS> : ro::silu_mul_kernel<T, false, UNROLL, THREADS>;
    return cuda_ok(err, launch_chained(kern, grid, THREADS, 0, s, 0, gate, up, y, nvec), "silu_mul_kernel launch");
  }
  const int64_t want = (n + THREADS - 1) / THREADS;
  const unsigned grid = static_cast<unsigned>(std::max<int64_t>(1, std::min<int64_t>(want, static_cast<int64_t>(sms) * 8)));
  auto kern = up ? ro::silu_mul_scalar_kernel<T, true, THREADS> : ro::silu_mul_scalar_kernel<T, false, THREADS>;
  return cuda_ok(err, launch_chained(kern, grid, THREADS, 0, s, 0, gate, up, y, n), "silu_mul_scalar_kernel launch");
}

inline int32_t silu_mul(std::string* err, const tsm100_silu_mul_desc* d, const void* gate, const void* up, void* y,
                        void* stream) {
  if (!d || !gate || !y) return op_fail(err, TSM100_ERR_INVALID, "silu_mul: null argument");
  if (!dtype_valid(d->dtype)) return op_fail(err, TSM100_ERR_INVALID, "silu_mul: unknown dtype");
  if (d->rows < 0 || d->cols < 0) return op_fail(err, TSM100_ERR_INVALID, "silu_mul: negative shape");
  if (d->rows == 0 || d->cols == 0) return TSM100_OK;
  const int64_t n = d->rows * d->cols;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  switch (d->dtype) {
    case TSM100_F32:
      return silu_mul_typed<float>(err, static_cast<const float*>(gate), static_cast<const float*>(up), static_cast<float*>(y), n, s);
    case TSM100_BF16:
      return silu_mul_typed<__nv_bfloat16>(err, static_cast<const __nv_bfloat16*>(gate), static_cast<const __nv_bfloat16*>(up),
                                           static_cast<__nv_bfloat16*>(y), n, s);
    default:
      return silu_mul_typed<__half>(err, static_cast<const __half*>(gate), static_cast<const __half*>(up),
                                    static_cast<__half*>(y), n, s);
  }
}

// ---------------------------------------------------------------------------
// RoPE and KV-cache update
// ---------------------------------------------------------------------------
inline int32_t rope(std::string* err, const tsm100_rope_desc* d, void* x, void* stream) {
  if (!d) return op_fail(err, TSM100_ERR_INVALID, "rope: null descriptor");
  if (!dtype_valid(d->dtype)) return op_fail(err, TSM100_ERR_INVALID, "rope: unknown dtype");
  if (d->batch < 0 || d->seq_len < 0 || d->heads < 0 || d->head_dim < 0 || d->start_pos < 0 || d->head_dim % 2 != 0)
    return op_fail(err, TSM100_ERR_INVALID, "rope: bad shape (head_dim must be even, nothing negative)");
  if (!(d->theta > 0.f)) return op_fail(err, TSM100_ERR_INVALID, "rope: theta must be positive");
  const int64_t tokens = static_cast<int64_t>(d->batch) * d->seq_len;
  if (tokens == 0 || d->heads == 0 || d->head_dim == 0) return TSM100_OK;
  if (!x) return op_fail(err, TSM100_ERR_INVALID, "rope: null buffer");
  int sms = 0;
  int32_t st = sm_count(err, &sms);
  if (st != TSM100_OK) return st;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const int pv = d->dtype == TSM100_F32 ? 4 : 8;  // elements per 16 bytes
  const bool vec = d->head_dim % pv == 0 && aligned16(x);
  const int64_t n = tokens * (vec ? d->head_dim / pv : d->head_dim / 2);
  // CTAs that go after one round, as in softmax.cuh: [8][8192][32][128] f32 342 us in eight to an SM that stay, 327 here
  const unsigned grid = static_cast<unsigned>(std::max<int64_t>(1, std::min<int64_t>((n + 255) / 256, 0x7fffffff)));
  auto launch = [&](auto* xt) -> cudaError_t {
    using T = std::remove_pointer_t<decltype(xt)>;
    if (vec) {
      const int32_t heads_per = route::rope_heads_per_thread(grid, d->heads, sms);
      const dim3 grid2(grid, static_cast<unsigned>((d->heads + heads_per - 1) / heads_per));
      auto kern = route::rope_few(static_cast<int64_t>(grid2.x) * grid2.y, heads_per, sms) ? rowops::rope_vec_kernel<T, true> : rowops::rope_vec_kernel<T, false>;
      return launch_chained(kern, grid2, 256, 0, s, 0, xt, tokens, d->seq_len, d->heads, heads_per, d->head_dim, d->start_pos, d->theta);
    }
    return launch_chained(rowops::rope_kernel<T>, grid, 256, 0, s, 0, xt, tokens, d->seq_len, d->heads, d->head_dim, d->start_pos, d->theta);
  };
  const cudaError_t e = d->dtype == TSM100_F32    ? launch(static_cast<float*>(x))
                        : d->dtype == TSM100_BF16 ? launch(static_cast<__nv_bfloat16*>(x))
                                                  : launch(static_cast<__half*>(x));
  return cuda_ok(err, e, "rope_kernel launch");
}

template <typename T>
inline cudaError_t kv_cache_update_typed(const tsm100_kv_cache_update_desc* d, const void* src, void* cache, int sms, cudaStream_t s) {
  constexpr int PV = softmax::Elem<T>::kPerVec;
  const bool vec = d->head_dim % PV == 0 && aligned16(src) && aligned16(cache);
  const int64_t n = static_cast<int64_t>(d->batch) * d->seq_len * d->heads * (vec ? d->head_dim / PV : d->head_dim);
  const unsigned grid = static_cast<unsigned>(std::max<int64_t>(1, std::min<int64_t>((n + 255) / 256, static_cast<int64_t>(sms) * 8)));
  const bool small = n + static_cast<int64_t>(grid) * 256 < 0xffffffffll;  // the loop index cannot wrap
  auto launch = [&](auto vec_tag, auto index_tag) {
    constexpr int V = decltype(vec_tag)::value;
    using I = decltype(index_tag);
    return launch_chained(rowops::kv_cache_update_kernel<T, V, I>, grid, 256, 0, s, 0, static_cast<const T*>(src), static_cast<T*>(cache),
                          static_cast<int64_t>(d->batch), d->seq_len, d->heads, d->head_dim, d->start_pos, d->max_seq);
  };
  if (vec && small) return launch(std::integral_constant<int, PV>{}, uint32_t{});
  if (vec) return launch(std::integral_constant<int, PV>{}, int64_t{});
  if (small) return launch(std::integral_constant<int, 1>{}, uint32_t{});
  return launch(std::integral_constant<int, 1>{}, int64_t{});
}

inline int32_t kv_cache_update(std::string* err, const tsm100_kv_cache_update_desc* d, const void* src, void* cache, void* stream) {
  if (!d) return op_fail(err, TSM100_ERR_INVALID, "kv_cache_update: null descriptor");
  if (!dtype_valid(d->dtype)) return op_fail(err, TSM100_ERR_INVALID, "kv_cache_update: unknown dtype");
  if (d->batch < 0 || d->seq_len < 0 || d->heads < 0 || d->head_dim < 0 || d->start_pos < 0 ||
      static_cast<int64_t>(d->start_pos) + d->seq_len > d->max_seq)
    return op_fail(err, TSM100_ERR_INVALID, "kv_cache_update: bad shape (need start_pos + seq_len <= max_seq, nothing negative)");
  if (static_cast<int64_t>(d->batch) * d->seq_len * d->heads * d->head_dim == 0) return TSM100_OK;
  if (!src || !cache) return op_fail(err, TSM100_ERR_INVALID, "kv_cache_update: null buffer");
  int sms = 0;
  int32_t st = sm_count(err, &sms);
  if (st != TSM100_OK) return st;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  cudaError_t e = d->dtype == TSM100_F32    ? kv_cache_update_typed<float>(d, src, cache, sms, s)
                  : d->dtype == TSM100_BF16 ? kv_cache_update_typed<__nv_bfloat16>(d, src, cache, sms, s)
                                            : kv_cache_update_typed<__half>(d, src, cache, sms, s);
  return cuda_ok(err, e, "kv_cache_update_kernel launch");
}

// ---------------------------------------------------------------------------
// GEMM
// ---------------------------------------------------------------------------
// Row pitches of A, B and C in elements: the descriptor's value, or the row length when it is 0.
struct GemmPitch {
  int64_t lda, ldb, ldc;
};
inline GemmPitch gemm_pitch(const tsm100_gemm_desc* d) {
  return {d->lda ? d->lda : d->k, d->ldb ? d->ldb : (d->b_transposed ? d->k : d->n), d->ldc ? d->ldc : d->n};
}
template <typename InT, typename OutT>
inline int32_t gemm_simt_launch(std::string* err, const tsm100_gemm_desc* d, const void* a, const void* b, void* c,
                                cudaStream_t s) {
  const GemmPitch ld = gemm_pitch(d);
  gemm_simt::Params p{static_cast<int32_t>(d->m), static_cast<int32_t>(d->n), static_cast<int32_t>(d->k), d->batch,
                      d->b_transposed, ld.lda, ld.ldb, ld.ldc};
  int sms = 0;
  int32_t st = sm_count(err, &sms);
  if (st != TSM100_OK) return st;
  const int64_t big_tiles = ((d->m + 63) / 64) * ((d->n + 63) / 64) * d->batch;
  if (big_tiles >= 2ll * sms) {
    dim3 grid(static_cast<unsigned>((d->n + 63) / 64), static_cast<unsigned>((d->m + 63) / 64),
              static_cast<unsigned>(d->batch));
    gemm_simt::gemm_simt_kernel<InT, OutT, 64, 64, 16, 4, 4><<<grid, 256, 0, s>>>(
        static_cast<const InT*>(a), static_cast<const InT*>(b), static_cast<OutT*>(c), p);
  } else {
    dim3 grid(static_cast<unsigned>((d->n + 31) / 32), static_cast<unsigned>((d->m + 31) / 32),
              static_cast<unsigned>(d->batch));
    gemm_simt::gemm_simt_kernel<InT, OutT, 32, 32, 16, 4, 4><<<grid, 64, 0, s>>>(
        static_cast<const InT*>(a), static_cast<const InT*>(b), static_cast<OutT*>(c), p);
  }
  return cuda_ok(err, cudaGetLastError(), "gemm_simt launch");
}

// f32 inputs on tensor cores (three TF32 products per product, see gemm_tf32x3.cuh)
inline int32_t gemm_tf32x3_launch(std::string* err, const tsm100_gemm_desc* d, const void* a, const void* b, void* c,
                                  cudaStream_t s) {
  namespace g = gemm_tf32x3;
  int sms = 0;
  int32_t st = sm_count(err, &sms);
  if (st != TSM100_OK) return st;
  const int64_t tiles = ((d->m + g::kBM - 1) / g::kBM) * ((d->n + g::kBN - 1) / g::kBN) * d->batch;
  if (tiles * g::kMaxSplit > 0x7fffffff) return op_fail(err, TSM100_ERR_INVALID, "gemm: too many tiles for one launch");
  static_assert(g::kBM == 64 && g::kBN == 64 && g::kBK == 32 && g::kMaxSplit == route::kMaxWarpF32Split, "route.hpp plans in these units");
  const int splits = route::gemm_f32_warp_splits(tiles, d->k, sms);
  g::Params p;
  p.m = static_cast<int32_t>(d->m);
  p.n = static_cast<int32_t>(d->n);
  p.k = static_cast<int32_t>(d->k);
  p.batch = d->batch;
  p.k_per_cta = static_cast<int32_t>(((d->k + splits - 1) / splits + g::kBK - 1) / g::kBK * g::kBK);
  const GemmPitch ld = gemm_pitch(d);
  p.lda = ld.lda, p.ldb = ld.ldb, p.ldc = ld.ldc;
  const int stages = splits > 1 ? g::kStagesSplit : g::kStages;
  auto launch = [&](auto kern) -> cudaError_t {
    cudaError_t e = set_dyn_smem_once(kern, g::kSmemBytes);
    if (e != cudaSuccess) return e;
    return launch_chained(kern, static_cast<unsigned>(tiles * splits), g::kThreads, static_cast<size_t>(stages) * g::kStageBytes, s,
                          static_cast<unsigned>(splits), static_cast<const float*>(a), static_cast<const float*>(b), static_cast<float*>(c), p);
  };
  cudaError_t e;
  if (d->b_transposed)
    e = splits > 1 ? launch(g::gemm_tf32x3_kernel<true, g::kStagesSplit>) : launch(g::gemm_tf32x3_kernel<true, g::kStages>);
  else
    e = splits > 1 ? launch(g::gemm_tf32x3_kernel<false, g::kStagesSplit>) : launch(g::gemm_tf32x3_kernel<false, g::kStages>);
  return cuda_ok(err, e, "gemm_tf32x3_kernel launch");
}

// The hi / lo planes of two operands (gemm_tf32_tc.cuh), `batch` of them; `transpose_b`: b comes as [cols][rows].  The same
// launch clears zero[0 .. n_zero).
inline int32_t split_operands_launch(std::string* err, gemm_tf32_tc::SplitOperand a, gemm_tf32_tc::SplitOperand b, bool transpose_b,
                                     int32_t batch, int sms, cudaStream_t s, uint32_t* zero = nullptr, int64_t n_zero = 0) {
  namespace g = gemm_tf32_tc;
  auto row_blocks = [&](const g::SplitOperand& p) {
    const int64_t items = p.rows * (p.kp / 4);
    return static_cast<int32_t>(std::max<int64_t>(1, std::min<int64_t>((items + 255) / 256, 16ll * sms)));
  };
  auto vec = [](const g::SplitOperand& p) { return p.kp == p.cols && p.ld % 4 == 0 && p.batch_stride % 4 == 0 && aligned16(p.src); };
  const int64_t tiles = (b.rows + 31) / 32 * ((b.cols + 31) / 32);
  a.blocks = row_blocks(a);
  if (transpose_b && tiles > 0x7fffffff - a.blocks) return op_fail(err, TSM100_ERR_INVALID, "operand split: too many tiles for one launch");
  b.blocks = transpose_b ? static_cast<int32_t>(tiles) : row_blocks(b);
  const dim3 grid(static_cast<unsigned>(a.blocks) + static_cast<unsigned>(b.blocks), static_cast<unsigned>(batch));
  auto kern = transpose_b ? (vec(a) ? g::split_operands_kernel<true, true> : g::split_operands_kernel<false, true>)
                          : (vec(a) && vec(b) ? g::split_operands_kernel<true, false> : g::split_operands_kernel<false, false>);
  return cuda_ok(err, launch_chained(kern, grid, 256, 0, s, 0, a, b, zero, n_zero), "split_operands_kernel launch");
}

// f32 inputs on the tcgen05 tensor cores: split pass (hi / lo planes, B's planes K-major), then the
// contraction with chunked accumulation (gemm_tf32_tc.cuh).  The planes live in stream-ordered scratch.
inline int32_t gemm_tf32_tc_launch(std::string* err, const tsm100_gemm_desc* d, const void* a, const void* b, void* c,
                                   uint32_t* status, bool rows_aligned, cudaStream_t s) {
  namespace g = gemm_tf32_tc;
  const uint64_t M = d->m, N = d->n, K = d->k, B = d->batch;
  const GemmPitch ld = gemm_pitch(d);
  int sms = 0;
  int32_t st = sm_count(err, &sms);
  if (st != TSM100_OK) return st;
  cudaError_t e = cudaSuccess;
  // Problems with more than one 128-row and 128-column block run on CTA pairs (256 x 256 or 256 x 128 tiles); the rest
  // on single CTAs (128 x 256 tiles).
  const bool pairs = M > 128 && N > 128;
  const route::PairTiles plan = pairs ? route::gemm_f32_pair_tiles(d->m, d->n, d->k, d->batch, sms) : route::PairTiles{g::kBN, 0, 1};
  const int bn = plan.bn;
  const uint64_t kp = (K + 3) / 4 * 4;  // row pitch of the planes: every row starts on a 16-byte boundary
  const size_t a_plane = static_cast<size_t>(B) * M * kp, b_plane = static_cast<size_t>(B) * N * kp;  // elements
  // rows that start anywhere: a flag per 128 x 128 block of C, behind the planes
  const int64_t flags = rows_aligned ? 0 : static_cast<int64_t>(B * ((M + 127) / 128) * ((N + 127) / 128));
  // tiles that several pairs share: partial sums of each of them, in front, and two counters per tile behind the flags
  const int64_t shared_tiles = plan.splits > 1 ? static_cast<int64_t>((M + 255) / 256) * ((N + bn - 1) / bn) * B - plan.whole_tiles : 0;
  const size_t part = static_cast<size_t>(shared_tiles) * plan.splits * 256 * bn;  // elements
  float* ws = nullptr;
  {
    const int32_t got = take_scratch(err, reinterpret_cast<void**>(&ws), (part + 2 * (a_plane + b_plane) + flags + 2 * shared_tiles) * sizeof(float), s);
    if (got != TSM100_OK) return got;
  }
  float *a_hi = ws + part, *a_lo = a_hi + a_plane, *b_hi = a_lo + a_plane, *b_lo = b_hi + b_plane;
  uint32_t* flag_words = reinterpret_cast<uint32_t*>(b_lo + b_plane);
  const float* af = static_cast<const float*>(a);
  const float* bf = static_cast<const float*>(b);
  st = split_operands_launch(err, {af, a_hi, a_lo, ld.lda, static_cast<int64_t>(M) * ld.lda, static_cast<int64_t>(M), static_cast<int32_t>(K), static_cast<int32_t>(kp), 0},
                             {bf, b_hi, b_lo, ld.ldb, static_cast<int64_t>(d->b_transposed ? N : K) * ld.ldb, static_cast<int64_t>(N), static_cast<int32_t>(K), static_cast<int32_t>(kp), 0},
                             !d->b_transposed, d->batch, sms, s, flag_words, flags + 2 * shared_tiles);
  CUtensorMap ta_hi, ta_lo, tb_hi, tb_lo;
  const CUtensorMapDataType f32 = CU_TENSOR_MAP_DATA_TYPE_FLOAT32;
  const uint32_t box_b = pairs ? bn / 2 : g::kBN;
  if (st == TSM100_OK) st = make_tmap_3d(err, &ta_hi, a_hi, K, M, B, kp, M * kp, g::kBK, g::kBM, f32, 4);
  if (st == TSM100_OK) st = make_tmap_3d(err, &ta_lo, a_lo, K, M, B, kp, M * kp, g::kBK, g::kBM, f32, 4);
  if (st == TSM100_OK) st = make_tmap_3d(err, &tb_hi, b_hi, K, N, B, kp, N * kp, g::kBK, box_b, f32, 4);
  if (st == TSM100_OK) st = make_tmap_3d(err, &tb_lo, b_lo, K, N, B, kp, N * kp, g::kBK, box_b, f32, 4);
  if (st == TSM100_OK) {
    g::Params p;
    p.m = static_cast<int32_t>(M);
    p.n = static_cast<int32_t>(N);
    p.k = static_cast<int32_t>(K);
    p.batch = d->batch;
    const uint64_t bm = pairs ? g::pair::kPairM : g::kBM;
    p.m_blocks = static_cast<int32_t>((M + bm - 1) / bm);
    p.n_blocks = static_cast<int32_t>((N + bn - 1) / bn);
    p.c_batch_stride = static_cast<int64_t>(M) * ld.ldc;
    p.ldc = ld.ldc;
    p.status = status;
    p.vec_store = aligned16(c) && ld.ldc % 4 == 0 ? 1 : 0;
    // Accumulation chunk: 128 of K, or shorter for the problems that the FP32 pipe took before, whose error was smaller at
    // short K (relative to the 64-bit result: FP32 pipe 2.9e-7 at K = 257, 6.9e-7 at 1501; here 9e-7 with chunks of 128,
    // 3.8e-7 with 64, 1.4e-7 .. 1.8e-7 with 32)
    p.chunk_kb = rows_aligned ? 4 : K >= 512 ? 2 : 1;
    p.flags = flag_words;
    p.b_transposed = d->b_transposed;
    p.a = af, p.b = bf;
    p.lda = ld.lda, p.ldb = ld.ldb;
    p.a_batch_stride = static_cast<int64_t>(M) * ld.lda;
    p.b_batch_stride = static_cast<int64_t>(d->b_transposed ? N : K) * ld.ldb;
    const int64_t tiles = static_cast<int64_t>(p.m_blocks) * p.n_blocks * p.batch;
    p.whole_tiles = static_cast<int32_t>(tiles - shared_tiles);
    p.splits = plan.splits;
    p.part = reinterpret_cast<float4*>(ws);
    p.arrivals = flag_words + flags;
    auto launch_pairs = [&](auto kern, int smem) -> cudaError_t {
      cudaError_t pe = set_dyn_smem_once(kern, smem);
      if (pe != cudaSuccess) return pe;
      const int max_clusters = resident_clusters(kern, g::kThreads, static_cast<size_t>(smem), 2, static_cast<unsigned>(sms & ~1), sms / 2);
      // as many pairs as the GPU holds at once, but one for every share (nobody waits for another pair)
      const int64_t npairs = std::max<int64_t>(shared_tiles * plan.splits, std::min<int64_t>(tiles, std::min<int64_t>(max_clusters, sms / 2)));
      return launch_chained(kern, static_cast<unsigned>(2 * npairs), g::kThreads, static_cast<size_t>(smem), s, 2, ta_hi, ta_lo, tb_hi, tb_lo,
                            static_cast<float*>(c), p);
    };
    if (pairs) {
      if (rows_aligned)
        e = bn == 256 ? launch_pairs(g::pair::gemm_tf32_tc2_kernel<256, false>, g::pair::smem_bytes<256>())
                      : launch_pairs(g::pair::gemm_tf32_tc2_kernel<128, false>, g::pair::smem_bytes<128>());
      else
        e = bn == 256 ? launch_pairs(g::pair::gemm_tf32_tc2_kernel<256, true>, g::pair::smem_bytes<256>())
                      : launch_pairs(g::pair::gemm_tf32_tc2_kernel<128, true>, g::pair::smem_bytes<128>());
      st = cuda_ok(err, e, "gemm_tf32_tc2_kernel launch");
    } else {
      auto kern = rows_aligned ? g::gemm_tf32_tc_kernel<false> : g::gemm_tf32_tc_kernel<true>;
      e = set_dyn_smem_once(kern, g::kSmemBytes);
      if (e == cudaSuccess) {
        const unsigned grid = static_cast<unsigned>(std::min<int64_t>(tiles, sms));
        e = launch_chained(kern, grid, g::kThreads, g::kSmemBytes, s, 0, ta_hi, ta_lo, tb_hi, tb_lo, static_cast<float*>(c), p);
      }
      st = cuda_ok(err, e, "gemm_tf32_tc_kernel launch");
    }
  }
  e = cudaFreeAsync(ws, s);  // stream-ordered: after the kernel that reads the planes
  if (st == TSM100_OK && e != cudaSuccess) st = cuda_ok(err, e, "cudaFreeAsync");
  return st;
}

// f32 inputs on the tcgen05 tensor cores, split on the way in (gemm_f32_fused.cuh).
inline int32_t gemm_f32_fused_launch(std::string* err, const tsm100_gemm_desc* d, const void* a, const void* b, void* c,
                                      const route::GemmF32& plan, uint32_t* status, bool rows_aligned, cudaStream_t s) {
  namespace g = gemm_f32_fused;
  const int bn = plan.bn;
  const GemmPitch ld = gemm_pitch(d);
  int sms = 0;
  int32_t st = sm_count(err, &sms);
  if (st != TSM100_OK) return st;
  g::Params p = {};
  p.g.m = static_cast<int32_t>(d->m);
  p.g.n = static_cast<int32_t>(d->n);
  p.g.k = static_cast<int32_t>(d->k);
  p.g.batch = d->batch;
  p.g.m_blocks = static_cast<int32_t>((d->m + g::kBM - 1) / g::kBM);
  p.g.n_blocks = static_cast<int32_t>((d->n + bn - 1) / bn);
  p.g.c_batch_stride = d->m * ld.ldc;
  p.g.ldc = ld.ldc;
  p.g.status = status;
  p.g.vec_store = aligned16(c) && ld.ldc % 4 == 0 ? 1 : 0;
  p.g.chunk_kb = rows_aligned ? g::kChunkKbAligned : g::kChunkKb;
  p.g.b_transposed = d->b_transposed;
  p.g.a = static_cast<const float*>(a);
  p.g.b = static_cast<const float*>(b);
  p.g.lda = ld.lda, p.g.ldb = ld.ldb;
  p.g.a_batch_stride = d->m * ld.lda;
  p.g.b_batch_stride = (d->b_transposed ? d->n : d->k) * ld.ldb;
  p.vec_a = aligned16(a) && d->k % 4 == 0 && ld.lda % 4 == 0;
  p.vec_b = aligned16(b) && d->k % 4 == 0 && ld.ldb % 4 == 0;
  const int64_t kb = (d->k + g::kBK - 1) / g::kBK;
  p.kb_per_cta = static_cast<int32_t>((kb + plan.splits - 1) / plan.splits);
  const int splits = static_cast<int>((kb + p.kb_per_cta - 1) / p.kb_per_cta);  // a last CTA without work is dropped
  const int64_t tiles = static_cast<int64_t>(p.g.m_blocks) * p.g.n_blocks * p.g.batch;
  const unsigned grid = static_cast<unsigned>(splits > 1 ? tiles * splits : std::min<int64_t>(tiles, sms));
  auto launch = [&](auto kern, int smem) -> cudaError_t {
    cudaError_t e = set_dyn_smem_once(kern, smem);
    if (e != cudaSuccess) return e;
    return launch_chained(kern, grid, g::kThreads, static_cast<size_t>(smem), s, static_cast<unsigned>(splits > 1 ? splits : 0), static_cast<float*>(c), p);
  };
  auto pick = [&](auto bn_tag) -> cudaError_t {
    constexpr int BN = decltype(bn_tag)::value;
    auto kern = p.kb_per_cta <= g::kStages ? (d->b_transposed ? g::gemm_f32_fused_kernel<BN, true, true> : g::gemm_f32_fused_kernel<BN, false, true>)
                                           : (d->b_transposed ? g::gemm_f32_fused_kernel<BN, true, false> : g::gemm_f32_fused_kernel<BN, false, false>);
    return launch(kern, g::smem_bytes<BN>());
  };
  return cuda_ok(err, bn == 64 ? pick(std::integral_constant<int, 64>{}) : pick(std::integral_constant<int, 128>{}), "gemm_f32_fused_kernel launch");
}

// C for TMA stores of 32 rows x 128 bytes (gemm_tc.cuh: store_rows).
template <typename OutT>
inline int32_t make_tmap_c(std::string* err, CUtensorMap* out, void* c, uint64_t m, uint64_t n, uint64_t batch, uint64_t ldc) {
  const CUtensorMapDataType type = sizeof(OutT) == 4 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32
                                   : std::is_same<OutT, __half>::value ? CU_TENSOR_MAP_DATA_TYPE_FLOAT16 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16;
  return make_tmap_3d(err, out, c, n, m, batch, ldc, m * ldc, gemm_tc::kBoxCols<OutT>, 32, type, sizeof(OutT));
}

// c_cols: 0, or N where rows of C may start anywhere.
template <typename OutT, bool kBT, bool kBf16>
inline int32_t gemm_tc_launch(std::string* err, const tsm100_gemm_desc* d, const void* a, const void* b, void* c,
                              uint32_t* status, cudaStream_t s, int64_t c_cols = 0) {
  namespace g = gemm_tc;
  CUtensorMap ta, tb, tc = {};
  const uint64_t M = d->m, N = d->n, K = d->k, B = d->batch;
  const GemmPitch ld = gemm_pitch(d);
  const uint64_t lda = ld.lda, ldb = ld.ldb;
  int32_t st = make_tmap_16bit_3d(err, &ta, a, K, M, B, lda, M * lda, g::kBK, g::kBM, kBf16);
  if (st != TSM100_OK) return st;
  if (kBT)
    st = make_tmap_16bit_3d(err, &tb, b, K, N, B, ldb, N * ldb, g::kBK, g::kBN, kBf16);
  else
    st = make_tmap_16bit_3d(err, &tb, b, N, K, B, ldb, K * ldb, 64, g::kBK, kBf16);
  if (st == TSM100_OK && c_cols == 0) st = make_tmap_c<OutT>(err, &tc, c, M, N, B, ld.ldc);
  if (st != TSM100_OK) return st;
  g::Params p;
  p.m = static_cast<int32_t>(M);
  p.n = static_cast<int32_t>(N);
  p.k = static_cast<int32_t>(K);
  p.batch = d->batch;
  p.m_blocks = static_cast<int32_t>((M + g::kBM - 1) / g::kBM);
  p.n_blocks = static_cast<int32_t>((N + g::kBN - 1) / g::kBN);
  p.c_batch_stride = static_cast<int64_t>(M) * ld.ldc;
  p.ldc = ld.ldc;
  p.status = status;
  int sms = 0;
  st = sm_count(err, &sms);
  if (st != TSM100_OK) return st;
  const int64_t tiles = static_cast<int64_t>(p.m_blocks) * p.n_blocks * p.batch;
  auto kern = c_cols ? g::gemm_tc_kernel<OutT, kBT, kBf16, true> : g::gemm_tc_kernel<OutT, kBT, kBf16>;
  cudaError_t e = set_dyn_smem_once(kern, g::kSmemBytes);
  if (e != cudaSuccess) return cuda_ok(err, e, "cudaFuncSetAttribute(gemm_tc_kernel)");
  const unsigned grid = static_cast<unsigned>(std::min<int64_t>(tiles, sms));
  return cuda_ok(err, launch_chained(kern, grid, g::kThreads, g::kSmemBytes, s, 0, ta, tb, tc, static_cast<OutT*>(c), p), "gemm_tc_kernel launch");
}

// Few output tiles: 128 columns x NT rows of C per CTA, K split over clusters (gemm_skinny.cuh).
static_assert(gemm_skinny::kMaxSplit == route::kMaxGemmSplit && gemm_skinny::kBK == 64 && gemm_skinny::kBN == 128, "route.hpp plans in these units");
template <typename OutT, bool kBT, bool kBf16, int NT>
inline int32_t gemm_skinny_launch_nt(std::string* err, const tsm100_gemm_desc* d, const void* a, const void* b, void* c,
                                     const route::Gemm16& plan, uint32_t* status, cudaStream_t s, int64_t c_cols = 0) {
  namespace g = gemm_skinny;
  CUtensorMap ta, tb;
  const uint64_t M = d->m, N = d->n, K = d->k, B = d->batch;
  const GemmPitch ld = gemm_pitch(d);
  const uint64_t lda = ld.lda, ldb = ld.ldb;
  int32_t st = make_tmap_16bit_3d(err, &ta, a, K, M, B, lda, M * lda, g::kBK, NT, kBf16);
  if (st != TSM100_OK) return st;
  if (kBT)
    st = make_tmap_16bit_3d(err, &tb, b, K, N, B, ldb, N * ldb, g::kBK, g::kBN, kBf16);
  else
    st = make_tmap_16bit_3d(err, &tb, b, N, K, B, ldb, K * ldb, 64, g::kBK, kBf16);
  if (st != TSM100_OK) return st;
  g::Params p;
  p.m = static_cast<int32_t>(M);
  p.n = static_cast<int32_t>(N);
  p.k = static_cast<int32_t>(K);
  p.batch = d->batch;
  p.m_blocks = static_cast<int32_t>((M + NT - 1) / NT);
  p.n_blocks = static_cast<int32_t>((N + g::kBN - 1) / g::kBN);
  p.c_batch_stride = static_cast<int64_t>(M) * ld.ldc;
  p.ldc = ld.ldc;
  p.status = status;
  const int64_t tiles = static_cast<int64_t>(p.m_blocks) * p.n_blocks * p.batch;
  p.kb_per_cta = static_cast<int32_t>(plan.k_blocks_per_cta);
  const int64_t kb = (K + g::kBK - 1) / g::kBK, splits = (kb + p.kb_per_cta - 1) / p.kb_per_cta;  // a last CTA without work is dropped
  int sms = 0;
  if (const int32_t got = sm_count(err, &sms); got != TSM100_OK) return got;
  p.early = route::skinny_places_early(B * N * K * 2, tiles * splits, sms) ? 1 : 0;
  auto kern = g::gemm_skinny_kernel<OutT, kBT, kBf16, NT, false>;
  if constexpr (sizeof(OutT) == 2)
    if (c_cols) kern = g::gemm_skinny_kernel<OutT, kBT, kBf16, NT, true>;
  constexpr int smem = g::smem_bytes<NT>();
  cudaError_t e = set_dyn_smem_once(kern, smem);
  if (e != cudaSuccess) return cuda_ok(err, e, "cudaFuncSetAttribute(gemm_skinny_kernel)");
  e = launch_chained(kern, static_cast<unsigned>(tiles * splits), g::kThreads, smem, s, static_cast<unsigned>(splits), ta, tb,
                     static_cast<OutT*>(c), p);
  return cuda_ok(err, e, "gemm_skinny_kernel launch");
}
template <typename OutT, bool kBT, bool kBf16>
inline int32_t gemm_skinny_launch(std::string* err, const tsm100_gemm_desc* d, const void* a, const void* b, void* c,
                                  const route::Gemm16& plan, uint32_t* status, cudaStream_t s, int64_t c_cols = 0) {
  switch (plan.rows) {
    case 16: return gemm_skinny_launch_nt<OutT, kBT, kBf16, 16>(err, d, a, b, c, plan, status, s, c_cols);
    case 32: return gemm_skinny_launch_nt<OutT, kBT, kBf16, 32>(err, d, a, b, c, plan, status, s, c_cols);
    case 64: return gemm_skinny_launch_nt<OutT, kBT, kBf16, 64>(err, d, a, b, c, plan, status, s, c_cols);
    default: return gemm_skinny_launch_nt<OutT, kBT, kBf16, 128>(err, d, a, b, c, plan, status, s, c_cols);
  }
}

// CTA-pair kernel (256 x 256 tile per two SMs), launched as clusters of two.
template <typename OutT, bool kBT, bool kBf16>
inline int32_t gemm_tc2_launch(std::string* err, const tsm100_gemm_desc* d, const void* a, const void* b, void* c,
                               uint32_t* status, cudaStream_t s, int64_t c_cols = 0) {
  namespace g = gemm_tc2;
  CUtensorMap ta, tb, tc = {};
  const uint64_t M = d->m, N = d->n, K = d->k, B = d->batch;
  const GemmPitch ld = gemm_pitch(d);
  const uint64_t lda = ld.lda, ldb = ld.ldb;
  int32_t st = make_tmap_16bit_3d(err, &ta, a, K, M, B, lda, M * lda, g::kBK, g::kCtaM, kBf16);
  if (st != TSM100_OK) return st;
  if (kBT)
    st = make_tmap_16bit_3d(err, &tb, b, K, N, B, ldb, N * ldb, g::kBK, g::kCtaN, kBf16);
  else
    st = make_tmap_16bit_3d(err, &tb, b, N, K, B, ldb, K * ldb, 64, g::kBK, kBf16);
  if (st == TSM100_OK && c_cols == 0) st = make_tmap_c<OutT>(err, &tc, c, M, N, B, ld.ldc);
  if (st != TSM100_OK) return st;
  gemm_tc::Params p;
  p.m = static_cast<int32_t>(M);
  p.n = static_cast<int32_t>(N);
  p.k = static_cast<int32_t>(K);
  p.batch = d->batch;
  p.m_blocks = static_cast<int32_t>((M + g::kPairM - 1) / g::kPairM);
  p.n_blocks = static_cast<int32_t>((N + g::kBN - 1) / g::kBN);
  p.status = status;
  p.c_batch_stride = static_cast<int64_t>(M) * ld.ldc;
  p.ldc = ld.ldc;
  int sms = 0;
  st = sm_count(err, &sms);
  if (st != TSM100_OK) return st;
  const int64_t tiles = static_cast<int64_t>(p.m_blocks) * p.n_blocks * p.batch;
  auto kern = c_cols ? g::gemm_tc2_kernel<OutT, kBT, kBf16, g::kLoose>
              : route::gemm16_pairs_store_boxes(d->k, tiles, sms) ? g::gemm_tc2_kernel<OutT, kBT, kBf16, g::kBoxes> : g::gemm_tc2_kernel<OutT, kBT, kBf16, g::kLanes>;
  cudaError_t e = set_dyn_smem_once(kern, g::kSmemBytes);
  if (e != cudaSuccess) return cuda_ok(err, e, "cudaFuncSetAttribute(gemm_tc2_kernel)");
  const int max_clusters = resident_clusters(kern, g::kThreads, g::kSmemBytes, 2, static_cast<unsigned>(sms & ~1), sms / 2);
  const int64_t pairs = std::min<int64_t>(tiles, std::min<int64_t>(max_clusters, sms / 2));
  e = launch_chained(kern, static_cast<unsigned>(2 * pairs), g::kThreads, g::kSmemBytes, s, 2, ta, tb, tc, static_cast<OutT*>(c), p);
  return cuda_ok(err, e, "gemm_tc2_kernel launch");
}

template <typename OutT, bool kBT, bool kBf16>
inline int32_t gemm_16bit_launch(std::string* err, const tsm100_gemm_desc* d, const void* a, const void* b, void* c, int sms, uint32_t* status,
                                 cudaStream_t s, int64_t c_cols = 0) {
  const route::Gemm16 plan = route::gemm16(d->m, d->n, d->k, d->batch, sms);
  switch (plan.kind) {
    case route::Gemm16::kPairs: return gemm_tc2_launch<OutT, kBT, kBf16>(err, d, a, b, c, status, s, c_cols);
    case route::Gemm16::kSingles: return gemm_tc_launch<OutT, kBT, kBf16>(err, d, a, b, c, status, s, c_cols);
    default: return gemm_skinny_launch<OutT, kBT, kBf16>(err, d, a, b, c, plan, status, s, c_cols);
  }
}

// A 16-bit problem whose rows start anywhere, on the tensor cores: operands whose rows do not start on 16-byte boundaries are copied to scratch where
// they do; the tensor maps end at N and K, and columns of C are written one by one.
inline int32_t gemm_padded(std::string* err, const tsm100_gemm_desc* d, const void* a, const void* b, void* c,
                           uint32_t* status, cudaStream_t s) {
  namespace g = gemm_pad;
  int sms = 0;
  int32_t st = sm_count(err, &sms);
  if (st != TSM100_OK) return st;
  cudaError_t e = cudaSuccess;
  const GemmPitch ld = gemm_pitch(d);
  const int64_t batch = d->batch, b_rows = d->b_transposed ? d->n : d->k, b_cols = d->b_transposed ? d->k : d->n;
  const int64_t a_pitch = (d->k + 7) / 8 * 8, b_pitch = (b_cols + 7) / 8 * 8;
  const bool pad_a = ld.lda % 8 != 0 || !aligned16(a), pad_b = ld.ldb % 8 != 0 || !aligned16(b);
  const int64_t a_elems = pad_a ? batch * d->m * a_pitch : 0, b_elems = pad_b ? batch * b_rows * b_pitch : 0;  // multiples of 8
  const int64_t c_cols = d->n % 8 != 0 || ld.ldc % 8 != 0 || !aligned16(c) ? d->n : 0;
  tsm100_gemm_desc t = *d;
  t.ldc = ld.ldc;
  const void *ta = a, *tb = b;
  uint16_t* ws = nullptr;
  if (pad_a || pad_b) {
    const int32_t got = take_scratch(err, reinterpret_cast<void**>(&ws), static_cast<size_t>(a_elems + b_elems) * 2, s);
    if (got != TSM100_OK) return got;
    auto operand = [&](bool copied, const void* src, int64_t pitch, int64_t rows, int64_t cols, uint16_t* dst, int64_t dst_pitch) {
      const int64_t items = copied ? rows * (dst_pitch / 8) : 0;
      return g::Operand{static_cast<const uint16_t*>(src), reinterpret_cast<uint4*>(dst), pitch, rows * pitch, static_cast<int32_t>(rows), static_cast<int32_t>(cols),
                        static_cast<int32_t>(dst_pitch), static_cast<int32_t>(std::min<int64_t>((items + g::kThreads - 1) / g::kThreads, 16ll * sms))};
    };
    const g::Operand oa = operand(pad_a, a, ld.lda, d->m, d->k, ws, a_pitch), ob = operand(pad_b, b, ld.ldb, b_rows, b_cols, ws + a_elems, b_pitch);
    if (pad_a) ta = ws, t.lda = a_pitch;
    if (pad_b) tb = ws + a_elems, t.ldb = b_pitch;
    e = launch_chained(g::pad_kernel, dim3(static_cast<unsigned>(oa.blocks + ob.blocks), static_cast<unsigned>(batch)), g::kThreads, 0, s, 0, oa, ob);
    st = cuda_ok(err, e, "gemm operand padding launch");
  }
  if (st == TSM100_OK) {
    if (d->dtype == TSM100_BF16)
      st = d->b_transposed ? gemm_16bit_launch<__nv_bfloat16, true, true>(err, &t, ta, tb, c, sms, status, s, c_cols) : gemm_16bit_launch<__nv_bfloat16, false, true>(err, &t, ta, tb, c, sms, status, s, c_cols);
    else
      st = d->b_transposed ? gemm_16bit_launch<__half, true, false>(err, &t, ta, tb, c, sms, status, s, c_cols) : gemm_16bit_launch<__half, false, false>(err, &t, ta, tb, c, sms, status, s, c_cols);
  }
  if (ws) {
    e = cudaFreeAsync(ws, s);
    if (st == TSM100_OK && e != cudaSuccess) st = cuda_ok(err, e, "cudaFreeAsync");
  }
  return st;
}

// `status` is a device word the tensor-core kernel writes if one of its bounded
// waits runs out; it must be zero when the launch starts.
inline int32_t gemm(std::string* err, const tsm100_gemm_desc* d, const void* a, const void* b, void* c,
                    uint32_t* status, void* stream) {
  if (!d || !a || !b || !c) return op_fail(err, TSM100_ERR_INVALID, "gemm: null argument");
  if (!dtype_valid(d->dtype) || !dtype_valid(d->out_dtype)) return op_fail(err, TSM100_ERR_INVALID, "gemm: unknown dtype");
  if (d->m < 0 || d->n < 0 || d->k < 0 || d->batch < 0) return op_fail(err, TSM100_ERR_INVALID, "gemm: negative shape");
  if (d->m > 0x7fffffff || d->n > 0x7fffffff || d->k > 0x7fffffff)
    return op_fail(err, TSM100_ERR_INVALID, "gemm: dimension exceeds 2^31-1");
  if (d->dtype == TSM100_F32 && d->out_dtype != TSM100_F32)
    return op_fail(err, TSM100_ERR_INVALID, "gemm: f32 inputs produce f32 output");
  if (d->dtype != TSM100_F32 && d->out_dtype != TSM100_F32 && d->out_dtype != d->dtype)
    return op_fail(err, TSM100_ERR_INVALID, "gemm: 16-bit inputs produce the same 16-bit type or f32");
  const GemmPitch ld = gemm_pitch(d);
  if (ld.lda < d->k || ld.ldb < (d->b_transposed ? d->k : d->n) || ld.ldc < d->n)
    return op_fail(err, TSM100_ERR_INVALID, "gemm: a row pitch (lda, ldb, ldc) is shorter than its row");
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  if (d->m == 0 || d->n == 0 || d->batch == 0) return TSM100_OK;
  if (d->k == 0) {  // empty contraction: C = 0 (linalg.fill)
    const size_t os = dtype_size(d->out_dtype);
    return cuda_ok(err, cudaMemset2DAsync(c, static_cast<size_t>(ld.ldc) * os, 0, static_cast<size_t>(d->n) * os,
                                          static_cast<size_t>(d->batch) * d->m, s), "cudaMemset2DAsync");
  }
  if (d->dtype == TSM100_F32) {
    const bool vec_ok = aligned16(a) && aligned16(b) && aligned16(c) && d->k % 4 == 0 && (d->b_transposed || d->n % 4 == 0) &&
                        d->n % 2 == 0 && ld.lda % 4 == 0 && ld.ldb % 4 == 0 && ld.ldc % 2 == 0;
    if (status != nullptr) {
      int sms = 0;
      int32_t st = sm_count(err, &sms);
      if (st != TSM100_OK) return st;
      const route::GemmF32 plan = route::gemm_f32(d->m, d->n, d->k, d->batch, vec_ok, sms, d->b_transposed != 0);
      const int64_t tiles = ((d->m + 127) / 128) * ((d->n + 255) / 256) * d->batch;
      if (plan.kind == route::GemmF32::kPlanes && tiles < 0x7fffffff) {
        st = gemm_tf32_tc_launch(err, d, a, b, c, status, vec_ok, s);
        if (st != kNoScratch) return st;
      }
      if (plan.kind == route::GemmF32::kFused) return gemm_f32_fused_launch(err, d, a, b, c, plan, status, vec_ok, s);
    }
    if (vec_ok) return gemm_tf32x3_launch(err, d, a, b, c, s);
    return gemm_simt_launch<float, float>(err, d, a, b, c, s);
  }

  const bool bf16 = d->dtype == TSM100_BF16;
  const bool out_f32 = d->out_dtype == TSM100_F32;
  // TMA needs 16-byte-multiple row pitches; the epilogue stores 16-byte vectors.
  const bool tma_ok = status != nullptr && aligned16(a) && aligned16(b) && aligned16(c) && (d->k % 8 == 0) &&
                      (d->b_transposed || d->n % 8 == 0) && (d->n * dtype_size(d->out_dtype)) % 16 == 0 &&
                      ld.lda % 8 == 0 && ld.ldb % 8 == 0 && (ld.ldc * dtype_size(d->out_dtype)) % 16 == 0 &&
                      (static_cast<int64_t>((d->m + 127) / 128) * ((d->n + 255) / 256) * d->batch < 0x7fffffff);
  if (tma_ok) {
    int sms = 0;
    int32_t st = sm_count(err, &sms);
    if (st != TSM100_OK) return st;
    if (bf16) {
      if (out_f32) return d->b_transposed ? gemm_16bit_launch<float, true, true>(err, d, a, b, c, sms, status, s) : gemm_16bit_launch<float, false, true>(err, d, a, b, c, sms, status, s);
      return d->b_transposed ? gemm_16bit_launch<__nv_bfloat16, true, true>(err, d, a, b, c, sms, status, s) : gemm_16bit_launch<__nv_bfloat16, false, true>(err, d, a, b, c, sms, status, s);
    }
    if (out_f32) return d->b_transposed ? gemm_16bit_launch<float, true, false>(err, d, a, b, c, sms, status, s) : gemm_16bit_launch<float, false, false>(err, d, a, b, c, sms, status, s);
    return d->b_transposed ? gemm_16bit_launch<__half, true, false>(err, d, a, b, c, sms, status, s) : gemm_16bit_launch<__half, false, false>(err, d, a, b, c, sms, status, s);
  }
  // Rows that start anywhere: copied into padded scratch where that pays.  Only for 16-bit results, whose last place hides the
  // order of the f32 sums; an f32 result keeps the FP32 pipe's rounding to nearest.
  const int64_t n8 = (d->n + 7) / 8 * 8, k8 = (d->k + 7) / 8 * 8;
  if (status != nullptr && !out_f32 && d->batch <= 65535 && n8 <= 0x7fffffff && k8 <= 0x7fffffff &&
      route::gemm16_copies_pay(d->m, d->n, d->k, d->batch, bf16) && (d->m + 127) / 128 * ((n8 + 255) / 256) * d->batch < 0x7fffffff) {
    const int32_t st = gemm_padded(err, d, a, b, c, status, s);
    if (st != kNoScratch) return st;
  }
  if (bf16) {
    if (out_f32) return gemm_simt_launch<__nv_bfloat16, float>(err, d, a, b, c, s);
    return gemm_simt_launch<__nv_bfloat16, __nv_bfloat16>(err, d, a, b, c, s);
  }
  if (out_f32) return gemm_simt_launch<__half, float>(err, d, a, b, c, s);
  return gemm_simt_launch<__half, __half>(err, d, a, b, c, s);
}

// ---------------------------------------------------------------------------
// attention
// ---------------------------------------------------------------------------
// Head dims 32, 64, 96 (and 128 for f32) with 16-byte aligned rows: the warp-level tensor-core kernel (f32: three
// TF32 products per product; 16-bit data, whose values are TF32 numbers already: one for Q K^T, two for P V).
template <typename T>
inline bool attention_tf32x3_ok(const attn_simt::Params& p, const void* q, const void* k, const void* v, const void* o) {
  constexpr int64_t vec = 16 / static_cast<int64_t>(sizeof(T));
  const bool dim_ok = p.head_dim == 32 || p.head_dim == 64 || p.head_dim == 96 || (sizeof(T) == 4 && p.head_dim == 128);
  return dim_ok && aligned16(q) && aligned16(k) && aligned16(v) && aligned16(o) && p.q_row_stride % vec == 0 &&
         p.q_head_stride % vec == 0 && p.kv_head_stride % vec == 0 && p.o_row_stride % vec == 0 && p.o_head_stride % vec == 0;
}
template <typename T, int D>
inline int32_t attention_tf32x3_launch_d(std::string* err, const attn_simt::Params& p, const T* q, const T* k,
                                         const T* v, T* o, cudaStream_t s) {
  namespace at = attn_tf32;
  const int64_t grid = static_cast<int64_t>((p.seq + at::kBM - 1) / at::kBM) * p.batch * p.heads_q;
  if (grid > 0x7fffffff) return op_fail(err, TSM100_ERR_INVALID, "attention: too many query blocks for one launch");
  auto kern = at::attention_tf32x3_kernel<T, D>;
  constexpr int smem = at::smem_bytes<T, D>();
  cudaError_t e = set_dyn_smem_once(kern, smem);
  if (e != cudaSuccess) return cuda_ok(err, e, "cudaFuncSetAttribute(attention_tf32x3_kernel)");
  return cuda_ok(err, launch_chained(kern, static_cast<unsigned>(grid), at::kThreads, smem, s, 0, q, k, v, o, p), "attention_tf32x3_kernel launch");
}
template <typename T>
inline int32_t attention_tf32x3_launch(std::string* err, const attn_simt::Params& p, const void* q, const void* k,
                                       const void* v, void* o, cudaStream_t s) {
  const T* qf = static_cast<const T*>(q);
  const T* kf = static_cast<const T*>(k);
  const T* vf = static_cast<const T*>(v);
  T* of = static_cast<T*>(o);
  if constexpr (sizeof(T) == 4)
    if (p.head_dim == 128) return attention_tf32x3_launch_d<T, 128>(err, p, qf, kf, vf, of, s);
  switch (p.head_dim) {
    case 96: return attention_tf32x3_launch_d<T, 96>(err, p, qf, kf, vf, of, s);
    case 64: return attention_tf32x3_launch_d<T, 64>(err, p, qf, kf, vf, of, s);
    default: return attention_tf32x3_launch_d<T, 32>(err, p, qf, kf, vf, of, s);
  }
}

// f32 on the tcgen05 kernel: one launch writes the parts of K and of V into stream-ordered scratch.  Row 0 of every (batch, KV head) is
// kv_head_stride elements after the one before.
template <int D>
inline int32_t attention_f32_tc_launch_d(std::string* err, const attn_simt::Params& p, const float* q, const float* k,
                                         const float* v, float* o, uint32_t* status, cudaStream_t s) {
  namespace at = attn_f32_tc;
  using Sh = at::Shape<D>;
  int sms = 0;
  int32_t st = sm_count(err, &sms);
  if (st != TSM100_OK) return st;
  const uint64_t n_kv = static_cast<uint64_t>(p.batch) * p.heads_kv, len = p.seq_kv;
  const size_t plane = n_kv * len * D;
  uint16_t* ws = nullptr;
  {
    const int32_t got = take_scratch(err, reinterpret_cast<void**>(&ws), 6 * plane * sizeof(uint16_t), s);
    if (got != TSM100_OK) return got;
  }
  at::SplitParams sp = {{k, v}, {ws, ws + 3 * plane}, p.kv_head_stride, static_cast<int64_t>(len * D / 8)};
  const int64_t per_head = std::max<int64_t>(1, std::min<int64_t>((sp.head_vecs + 255) / 256, 4ll * sms / static_cast<int64_t>(n_kv)));
  cudaError_t e = launch_chained(at::split_kv_kernel, dim3(static_cast<unsigned>(per_head), static_cast<unsigned>(n_kv), 2), 256, 0, s, 0, sp);
  st = cuda_ok(err, e, "split_kv_kernel launch");
  CUtensorMap tk, tv;
  if (st == TSM100_OK) st = make_tmap_16bit_3d(err, &tk, ws, D, len, 3 * n_kv, D, len * D, Sh::kGroup, at::kBKV, true);
  if (st == TSM100_OK) st = make_tmap_16bit_3d(err, &tv, ws + 3 * plane, D, len, 3 * n_kv, D, len * D, Sh::kGroup, at::kBKV, true);
  if (st == TSM100_OK) {
    auto kern = at::attention_f32_tc_kernel<D>;
    e = set_dyn_smem_once(kern, at::smem_bytes<D>());
    if (e == cudaSuccess) {
      at::Params pp;
      pp.a = p;
      pp.status = status;
      const int64_t grid = static_cast<int64_t>((p.seq + at::kBQ - 1) / at::kBQ) * p.batch * p.heads_q;
      e = launch_chained(kern, static_cast<unsigned>(grid), at::kThreads, at::smem_bytes<D>(), s, 0, tk, tv, q, o, pp);
    }
    st = cuda_ok(err, e, "attention_f32_tc_kernel launch");
  }
  e = cudaFreeAsync(ws, s);  // stream-ordered: after the kernel that reads the planes
  if (st == TSM100_OK && e != cudaSuccess) st = cuda_ok(err, e, "cudaFreeAsync");
  return st;
}
inline int32_t attention_f32_tc_launch(std::string* err, const attn_simt::Params& p, const void* q, const void* k, const void* v,
                                       void* o, uint32_t* status, cudaStream_t s) {
  const float *qf = static_cast<const float*>(q), *kf = static_cast<const float*>(k), *vf = static_cast<const float*>(v);
  float* of = static_cast<float*>(o);
  switch (p.head_dim) {
    case 128: return attention_f32_tc_launch_d<128>(err, p, qf, kf, vf, of, status, s);
    case 96: return attention_f32_tc_launch_d<96>(err, p, qf, kf, vf, of, status, s);
    case 64: return attention_f32_tc_launch_d<64>(err, p, qf, kf, vf, of, status, s);
    default: return attention_f32_tc_launch_d<32>(err, p, qf, kf, vf, of, status, s);
  }
}
// Of the problems that attention_tf32x3_ok takes, those for the tcgen05 kernel.
inline bool attention_f32_tc_ok(const attn_simt::Params& p, const uint32_t* status) {
  const int64_t blocks = static_cast<int64_t>((p.seq + 127) / 128) * p.batch * p.heads_q;
  const int64_t n_kv = static_cast<int64_t>(p.batch) * p.heads_kv;
  return status != nullptr && route::attention_f32_on_tcgen05(p.head_dim, p.seq_kv) && blocks <= 0x7fffffff && n_kv <= 65535 && p.seq_kv <= 1 << 20;
}

template <typename T>
inline int32_t attention_simt_launch(std::string* err, const tsm100_attention_desc* d, const void* q, const void* k,
                                     const void* v, void* o, uint32_t* status, cudaStream_t s) {
  const int64_t sd = static_cast<int64_t>(d->seq) * d->head_dim;
  attn_simt::Params p{d->seq, d->head_dim, d->heads_q, d->heads_kv, d->batch, d->causal,
                      static_cast<float>(1.0 / std::sqrt(static_cast<double>(d->head_dim))),
                      d->seq, 0, d->head_dim, sd, sd, d->head_dim, sd};
  if (attention_tf32x3_ok<T>(p, q, k, v, o)) {
    if (sizeof(T) == 4 && attention_f32_tc_ok(p, status)) {
      const int32_t st = attention_f32_tc_launch(err, p, q, k, v, o, status, s);
      if (st != kNoScratch) return st;
    }
    return attention_tf32x3_launch<T>(err, p, q, k, v, o, s);
  }
  const int64_t rows = static_cast<int64_t>(d->batch) * d->heads_q * d->seq;
  const int64_t grid = (rows + attn_simt::kWarps - 1) / attn_simt::kWarps;
  if (grid > 0x7fffffff) return op_fail(err, TSM100_ERR_INVALID, "attention: too many query rows for one launch");
  attn_simt::attention_simt_kernel<T><<<static_cast<unsigned>(grid), attn_simt::kWarps * 32, 0, s>>>(
      static_cast<const T*>(q), static_cast<const T*>(k), static_cast<const T*>(v), static_cast<T*>(o), p);
  return cuda_ok(err, cudaGetLastError(), "attention_simt launch");
}

// ---------------------------------------------------------------------------
// prefill attention: seq_len new tokens against a KV cache that already holds them and start_pos earlier ones
// ---------------------------------------------------------------------------
template <typename T>
inline int32_t attention_prefill_simt_launch(std::string* err, const tsm100_attention_prefill_desc* d, const void* q,
                                             const void* k, const void* v, void* o, uint32_t* status, cudaStream_t s) {
  const int64_t hd = static_cast<int64_t>(d->heads_q) * d->head_dim;
  attn_simt::Params p{d->seq_len, d->head_dim, d->heads_q, d->heads_kv, 1, 1,
                      static_cast<float>(1.0 / std::sqrt(static_cast<double>(d->head_dim))),
                      d->start_pos + d->seq_len, d->start_pos, hd, d->head_dim,
                      static_cast<int64_t>(d->max_seq) * d->head_dim, hd, d->head_dim};
  if (attention_tf32x3_ok<T>(p, q, k, v, o)) {
    if (sizeof(T) == 4 && attention_f32_tc_ok(p, status)) {
      const int32_t st = attention_f32_tc_launch(err, p, q, k, v, o, status, s);
      if (st != kNoScratch) return st;
    }
    return attention_tf32x3_launch<T>(err, p, q, k, v, o, s);
  }
  const int64_t rows = static_cast<int64_t>(d->heads_q) * d->seq_len;
  const int64_t grid = (rows + attn_simt::kWarps - 1) / attn_simt::kWarps;
  if (grid > 0x7fffffff) return op_fail(err, TSM100_ERR_INVALID, "attention_prefill: too many query rows for one launch");
  attn_simt::attention_simt_kernel<T><<<static_cast<unsigned>(grid), attn_simt::kWarps * 32, 0, s>>>(
      static_cast<const T*>(q), static_cast<const T*>(k), static_cast<const T*>(v), static_cast<T*>(o), p);
  return cuda_ok(err, cudaGetLastError(), "attention_simt (prefill) launch");
}

// KV heads per band of the causal launch order: as many as keep K and V of the band (16-bit) within
// 32 MiB, a quarter of the L2, so that the blocks in flight - a few weight levels of one band, at a band's end
// together with the start of the next - read K and V from DRAM once.
inline int32_t attention_kv_band(uint64_t kv_len, int64_t kv_heads, uint64_t head_dim) {
  const uint64_t per_head = std::max<uint64_t>(1, kv_len * head_dim * 2 * 2);
  const int64_t band = static_cast<int64_t>((32ull << 20) / per_head);
  return static_cast<int32_t>(std::max<int64_t>(1, std::min<int64_t>(band, std::max<int64_t>(kv_heads, 1))));
}

// The tcgen05 attention kernels: heads of 128, and of 64 and less.
template <bool kBf16, bool kCache, int D, bool kSplit, bool kLone = kSplit>
struct AttentionFwd {
  static auto kernel() {
    if constexpr (D == 64) return attn_narrow::attention_narrow_kernel<kBf16, kCache, kSplit, kLone>;
    else return attn::attention_fwd_kernel<kBf16, kCache, kSplit, kLone>;
  }
  static constexpr int smem() {
    if constexpr (D == 64) return attn_narrow::kSmemBytes;
    else return attn::kSmemBytes;
  }
};

// Launches the tcgen05 attention kernel over the rows of `heads` heads that see at most `keys` keys, the KV steps of a block dealt to
// several CTAs and merged by a second kernel where route.hpp says so.
template <bool kBf16, bool kCache, int D>
inline int32_t attention_fwd_launch(std::string* err, const CUtensorMap& tq, const CUtensorMap& tk, const CUtensorMap& tv, void* o,
                                    attn::Params p, int64_t heads, int64_t keys, cudaStream_t s) {
  namespace at = attn;
  constexpr int smem = AttentionFwd<kBf16, kCache, D, false>::smem();
  static_assert(attn_narrow::kThreads == at::kThreads, "one launch for both");
  int sms = 0;
  int32_t st = sm_count(err, &sms);
  if (st != TSM100_OK) return st;
  uint16_t* out = static_cast<uint16_t*>(o);
  p.block_rows = 2 * at::kBQ;
  p.splits = route::attention_split_ctas(route::div_up(p.seq, 2 * at::kBQ) * heads, keys, sms);
  if (p.splits == 1) p.block_rows = route::attention_block_rows(p.seq, heads, keys, p.q_offset, p.causal != 0, sms);
  p.q_blocks = static_cast<int32_t>(route::div_up(p.seq, p.block_rows));
  const int64_t blocks = p.q_blocks * heads;
  if (blocks > 0x7fffffff) return op_fail(err, TSM100_ERR_INVALID, "attention: too many tiles for one launch");
  p.blocks = static_cast<int32_t>(blocks);
  p.part = nullptr;
  p.part_ml = nullptr;
  const size_t rows = static_cast<size_t>(blocks) * p.splits * (2 * at::kBQ);
  float* ws = nullptr;
  if (p.splits > 1) {
    st = take_scratch(err, reinterpret_cast<void**>(&ws), rows * (D + 2) * sizeof(float), s);
    if (st == kNoScratch) p.splits = 1;
    else if (st != TSM100_OK) return st;
  }
  cudaError_t e = cudaSuccess;
  if (p.splits == 1) {
    const bool lone = p.block_rows == at::kBQ || p.seq - (p.q_blocks - 1) * (2 * at::kBQ) <= at::kBQ;  // some block has one tile
    auto kern = lone ? AttentionFwd<kBf16, kCache, D, false, true>::kernel() : AttentionFwd<kBf16, kCache, D, false>::kernel();
    e = set_dyn_smem_once(kern, smem);
    if (e != cudaSuccess) return cuda_ok(err, e, "cudaFuncSetAttribute(attention_fwd_kernel)");
    return cuda_ok(err, launch_chained(kern, static_cast<unsigned>(blocks), at::kThreads, smem, s, 0, tq, tk, tv, out, p), "attention_fwd_kernel launch");
  }
  p.part = reinterpret_cast<float4*>(ws);
  p.part_ml = reinterpret_cast<float2*>(ws + rows * D);
  auto kern = AttentionFwd<kBf16, kCache, D, true>::kernel();
  e = set_dyn_smem_once(kern, smem);
  if (e == cudaSuccess) e = launch_chained(kern, static_cast<unsigned>(blocks * p.splits), at::kThreads, smem, s, 0, tq, tk, tv, out, p);
  if (e == cudaSuccess)
    e = launch_chained(at::attention_merge_kernel<kBf16, kCache, D>, static_cast<unsigned>(blocks * (D / 16)), 2 * at::kBQ, 0, s, 0, out, p);
  st = cuda_ok(err, e, "attention_fwd_kernel (split) launch");
  e = cudaFreeAsync(ws, s);
  if (st == TSM100_OK && e != cudaSuccess) st = cuda_ok(err, e, "cudaFreeAsync");
  return st;
}

// Which 16-bit problems run on the tcgen05 kernels: head_dim 128 (attention_tc.cuh), 32 and 64 (attention_narrow.cuh).  96 stays on the TF32
// kernel: in tensor memory three score buffers of 128 columns leave room for two O of 64, not of 96.  b4, 32 / 8 heads of
// 64, 2000 tokens, causal: 724 us on the TF32 kernel, 132 here (graph replays); both 1.6e-3 from the 64-bit result, the rounding of bf16.  Short
// sequences of 32 and 64 stay there too (route.hpp).  rows: query rows per head, heads: of all problems.
inline bool attention_tc_ok(int32_t dtype, int32_t head_dim, int64_t rows, int64_t heads, int64_t seq_kv, const uint32_t* status,
                            const void* q, const void* k, const void* v, const void* o) {
  if (dtype == TSM100_F32 || status == nullptr || !aligned16(q) || !aligned16(k) || !aligned16(v) || !aligned16(o)) return false;
  if (head_dim == attn::kD) return true;
  if (head_dim != 32 && head_dim != 64) return false;
  int sms = 0;
  std::string unused;
  if (sm_count(&unused, &sms) != TSM100_OK) return false;
  return route::attention_narrow_on_tcgen05(head_dim, seq_kv, route::div_up(rows, 2 * attn::kBQ) * heads, sms);
}

template <bool kBf16, int D>
inline int32_t attention_prefill_tc_launch(std::string* err, const tsm100_attention_prefill_desc* d, const void* q, const void* k,
                                           const void* v, void* o, uint32_t* status, cudaStream_t s) {
  namespace at = attn;
  CUtensorMap tq, tk, tv;
  const uint64_t d_row = d->head_dim, hq = d->heads_q, hkv = d->heads_kv, kv_len = static_cast<uint64_t>(d->start_pos) + d->seq_len;
  // token-major Q: row pitch heads_q * D, head pitch D; caches: row pitch D, head pitch max_seq * D, kv_len rows visible
  int32_t st = make_tmap_16bit_3d(err, &tq, q, d_row, d->seq_len, hq, hq * d_row, d_row, 64, at::kBQ, kBf16);
  if (st == TSM100_OK) st = make_tmap_16bit_3d(err, &tk, k, d_row, kv_len, hkv, d_row, static_cast<uint64_t>(d->max_seq) * d_row, 64, at::kBKV, kBf16);
  if (st == TSM100_OK) st = make_tmap_16bit_3d(err, &tv, v, d_row, kv_len, hkv, d_row, static_cast<uint64_t>(d->max_seq) * d_row, 64, at::kBKV, kBf16);
  if (st != TSM100_OK) return st;
  at::Params p;
  p.seq = d->seq_len;
  p.heads_q = d->heads_q;
  p.heads_kv = d->heads_kv;
  p.batch = 1;
  p.causal = 1;
  p.kv_band = attention_kv_band(kv_len, d->heads_kv, d_row);
  p.scale_log2 = static_cast<float>((1.0 / std::sqrt(static_cast<double>(d->head_dim))) * 1.4426950408889634);
  p.status = status;
  p.seq_kv = static_cast<int32_t>(kv_len);
  p.q_offset = d->start_pos;
  p.o_row_stride = static_cast<int64_t>(hq * d_row);
  p.o_head_stride = static_cast<int64_t>(d_row);
  p.head_dim = d->head_dim;
  return attention_fwd_launch<kBf16, true, D>(err, tq, tk, tv, o, p, d->heads_q, static_cast<int64_t>(kv_len), s);
}

inline int32_t attention_prefill(std::string* err, const tsm100_attention_prefill_desc* d, const void* q, const void* k,
                                 const void* v, void* o, uint32_t* status, void* stream) {
  if (!d || !q || !k || !v || !o) return op_fail(err, TSM100_ERR_INVALID, "attention_prefill: null argument");
  if (!dtype_valid(d->dtype)) return op_fail(err, TSM100_ERR_INVALID, "attention_prefill: unknown dtype");
  if (d->heads_q <= 0 || d->heads_kv <= 0 || d->seq_len < 0 || d->start_pos < 0 || d->head_dim <= 0 ||
      static_cast<int64_t>(d->start_pos) + d->seq_len > d->max_seq)
    return op_fail(err, TSM100_ERR_INVALID, "attention_prefill: bad shape (need heads > 0 and start_pos + seq_len <= max_seq)");
  if (d->heads_q % d->heads_kv != 0)
    return op_fail(err, TSM100_ERR_INVALID, "attention_prefill: heads_q must be a multiple of heads_kv");
  if (d->head_dim > attn_simt::kMaxD) return op_fail(err, TSM100_ERR_INVALID, "attention_prefill: head_dim > 256 unsupported");
  if (d->seq_len == 0) return TSM100_OK;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  if (attention_tc_ok(d->dtype, d->head_dim, d->seq_len, d->heads_q, static_cast<int64_t>(d->start_pos) + d->seq_len, status, q, k, v, o)) {
    const bool wide = d->head_dim == attn::kD;
    if (d->dtype == TSM100_BF16)
      return wide ? attention_prefill_tc_launch<true, 128>(err, d, q, k, v, o, status, s)
                  : attention_prefill_tc_launch<true, 64>(err, d, q, k, v, o, status, s);
    return wide ? attention_prefill_tc_launch<false, 128>(err, d, q, k, v, o, status, s)
                : attention_prefill_tc_launch<false, 64>(err, d, q, k, v, o, status, s);
  }
  if (d->dtype == TSM100_F32) return attention_prefill_simt_launch<float>(err, d, q, k, v, o, status, s);
  if (d->dtype == TSM100_BF16) return attention_prefill_simt_launch<__nv_bfloat16>(err, d, q, k, v, o, status, s);
  return attention_prefill_simt_launch<__half>(err, d, q, k, v, o, status, s);
}

// ---------------------------------------------------------------------------
// decode attention (one query token against a KV cache)
// ---------------------------------------------------------------------------
template <typename T, int G, int D>
inline int32_t attention_decode_launch(std::string* err, const tsm100_attention_decode_desc* d, const T* q, const T* k,
                                       const T* v, T* o, int head_base, int heads_here, int splits, cudaStream_t s) {
  namespace ad = attn_decode;
  ad::Params p;
  p.batch = d->batch;
  p.heads_q = d->heads_q;
  p.heads_kv = d->heads_kv;
  p.seq_len = d->seq_len;
  p.max_seq = d->max_seq;
  p.group = d->heads_q / d->heads_kv;
  p.head_base = head_base;
  p.heads_here = heads_here;
  p.scale_log2 = static_cast<float>((1.0 / std::sqrt(static_cast<double>(D))) * 1.4426950408889634);
  auto kern = ad::attention_decode_kernel<T, G, D>;
  constexpr int smem = ad::smem_floats<T, G, D>() * static_cast<int>(sizeof(float));
  cudaError_t e = set_dyn_smem_once(kern, smem);
  if (e != cudaSuccess) return cuda_ok(err, e, "cudaFuncSetAttribute(attention_decode_kernel)");
  int sms = 0;
  const int32_t st = sm_count(err, &sms);
  if (st != TSM100_OK) return st;
  const unsigned grid = static_cast<unsigned>(static_cast<int64_t>(d->batch) * d->heads_kv * splits);
  e = launch_kernel(route::decode_is_chained(grid, static_cast<int64_t>(d->seq_len) * D * 2 * static_cast<int64_t>(sizeof(T)) / splits, sms), kern, grid, ad::kThreads, smem, s, static_cast<unsigned>(splits), q, k, v, o, p);
  return cuda_ok(err, e, "attention_decode_kernel launch");
}

// The tensor-core decode kernel for an element type: mma.sync on 16-bit caches, three TF32 products on f32 caches.
template <typename T, int D, int STAGES, int WARPS>
struct DecodeTc {
  static auto kernel() {
    if constexpr (sizeof(T) == 4) return attn_decode::tf32::attention_decode_tf32_kernel<D, STAGES, WARPS>;
    else return attn_decode::mma::attention_decode_mma_kernel<T, D, STAGES, WARPS>;
  }
  static constexpr int smem() {
    if constexpr (sizeof(T) == 4) return attn_decode::tf32::smem_bytes<D, STAGES, WARPS>();
    else return attn_decode::mma::smem_bytes<D, STAGES, WARPS>();
  }
};

template <typename T, int D, int STAGES, int WARPS>
inline int32_t attention_decode_mma_launch(std::string* err, const tsm100_attention_decode_desc* d, const T* q, const T* k,
                                           const T* v, T* o, int head_base, int heads_here, int splits, cudaStream_t s) {
  namespace ad = attn_decode;
  ad::Params p;
  p.batch = d->batch;
  p.heads_q = d->heads_q;
  p.heads_kv = d->heads_kv;
  p.seq_len = d->seq_len;
  p.max_seq = d->max_seq;
  p.group = d->heads_q / d->heads_kv;
  p.head_base = head_base;
  p.heads_here = heads_here;
  p.scale_log2 = static_cast<float>((1.0 / std::sqrt(static_cast<double>(D))) * 1.4426950408889634);
  auto kern = DecodeTc<T, D, STAGES, WARPS>::kernel();
  constexpr int smem = DecodeTc<T, D, STAGES, WARPS>::smem();
  cudaError_t e = set_dyn_smem_once(kern, smem);
  if (e != cudaSuccess) return cuda_ok(err, e, "cudaFuncSetAttribute(attention_decode_mma_kernel)");
  if (splits > ad::kMaxSplits) {
    e = allow_wide_clusters_once(kern);
    if (e != cudaSuccess) return cuda_ok(err, e, "cudaFuncSetAttribute(attention_decode_mma_kernel, wide clusters)");
  }
  int sms = 0;
  const int32_t st = sm_count(err, &sms);
  if (st != TSM100_OK) return st;
  const unsigned grid = static_cast<unsigned>(static_cast<int64_t>(d->batch) * d->heads_kv * splits);
  // the kernel for f32 caches does not wait for the one before it: bound by the arithmetic, it took longer beside its last CTAs (24 caches
  // of 10449 x 64, 8 heads each, 52.3 us, 53.5 chained)
  e = launch_kernel(sizeof(T) == 2 && route::decode_is_chained(grid, static_cast<int64_t>(d->seq_len) * D * 2 * static_cast<int64_t>(sizeof(T)) / splits, sms), kern, grid, WARPS * 32, smem, s, static_cast<unsigned>(splits), q, k, v, o, p);
  return cuda_ok(err, e, "attention_decode_mma_kernel launch");
}

// 16-bit caches, a few units: `splits` independent CTAs per unit and a merge kernel (programmatic dependent launch).
template <typename T, int D>
inline int32_t attention_decode_global_launch(std::string* err, const tsm100_attention_decode_desc* d, const T* q, const T* k,
                                              const T* v, T* o, int splits, cudaStream_t s) {
  namespace ad = attn_decode;
  constexpr int WARPS = 8, STAGES = 3;
  const int64_t units = static_cast<int64_t>(d->batch) * d->heads_kv;
  cudaError_t e = cudaSuccess;
  float* ws = nullptr;
  {
    const int32_t got = take_scratch(err, reinterpret_cast<void**>(&ws), static_cast<size_t>(units) * splits * ad::mma::kRows * (D + 2) * sizeof(float), s);
    if (got != TSM100_OK) return got;
  }
  ad::Params p;
  p.batch = d->batch;
  p.heads_q = d->heads_q;
  p.heads_kv = d->heads_kv;
  p.seq_len = d->seq_len;
  p.max_seq = d->max_seq;
  p.group = d->heads_q / d->heads_kv;
  p.scale_log2 = static_cast<float>((1.0 / std::sqrt(static_cast<double>(D))) * 1.4426950408889634);
  p.splits = splits;
  p.part = ws;
  auto kern = ad::mma::attention_decode_mma_kernel<T, D, STAGES, WARPS, true>;
  constexpr int smem = ad::mma::smem_bytes<D, STAGES, WARPS>();
  e = set_dyn_smem_once(kern, smem);
  for (int base = 0; base < p.group && e == cudaSuccess; base += ad::mma::kRows) {
    p.head_base = base;
    p.heads_here = std::min(ad::mma::kRows, p.group - base);
    e = launch_chained(kern, static_cast<unsigned>(units * splits), WARPS * 32, smem, s, 0, q, k, v, o, p);
    if (e != cudaSuccess) break;
    e = launch_chained(ad::mma::attention_decode_merge_kernel<T, D>, static_cast<unsigned>(units * p.heads_here), D, 0, s, 0, o, p);
  }
  int32_t st = cuda_ok(err, e, "attention_decode_mma_kernel (partial results) launch");
  e = cudaFreeAsync(ws, s);
  if (st == TSM100_OK && e != cudaSuccess) st = cuda_ok(err, e, "cudaFreeAsync");
  return st;
}

// 16-bit caches, up to eight query heads each: the tiles of all caches dealt out evenly (attention_decode_stream.cuh).
static_assert(attn_decode::stream::kTileBytes == route::kDecodeTileBytes, "route.hpp plans in these units");
template <typename T, int D>
inline int32_t attention_decode_stream_launch(std::string* err, const tsm100_attention_decode_desc* d, const T* q, const T* k, const T* v, T* o,
                                              const route::DecodeStream& plan, uint32_t* status, cudaStream_t s) {
  namespace ad = attn_decode::stream;
  const uint64_t units = static_cast<uint64_t>(d->batch) * d->heads_kv;
  CUtensorMap tk, tv;
  TmapKey key;
  std::memset(&key, 0, sizeof key);
  key.base = k;
  key.dim[0] = 64, key.dim[1] = d->max_seq, key.dim[2] = D / 64, key.dim[3] = units;
  key.stride[0] = D * 2, key.stride[1] = 128, key.stride[2] = static_cast<uint64_t>(d->max_seq) * D * 2;
  key.box[0] = 64, key.box[1] = ad::tile_rows<D>(), key.box[2] = D / 64, key.box[3] = 1;
  key.dtype = static_cast<int32_t>(std::is_same<T, __half>::value ? CU_TENSOR_MAP_DATA_TYPE_FLOAT16 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16), key.rank = 4;
  int32_t st = make_tmap(err, &tk, key, 2);
  key.base = v;
  if (st == TSM100_OK) st = make_tmap(err, &tv, key, 2);
  if (st != TSM100_OK) return st;
  ad::Params p;
  p.heads_q = d->heads_q;
  p.heads_kv = d->heads_kv;
  p.group = d->heads_q / d->heads_kv;
  p.head_base = 0;
  p.heads_here = p.group;
  p.seq_len = d->seq_len;
  p.max_seq = d->max_seq;
  p.tiles = plan.tiles;
  p.grain = plan.grain;
  p.grains = plan.grains;
  p.scale_log2 = static_cast<float>((1.0 / std::sqrt(static_cast<double>(D))) * 1.4426950408889634);
  p.part = nullptr;
  p.status = status;
  const bool merged = plan.grain != plan.tiles;
  if (merged) {
    st = take_scratch(err, reinterpret_cast<void**>(&p.part), static_cast<size_t>(plan.ctas) * 2 * ad::record_floats<D>() * sizeof(float), s);
    if (st != TSM100_OK) return st;
  }
  auto kern = ad::attention_decode_stream_kernel<T, D>;
  constexpr int smem = ad::smem_bytes<D>();
  cudaError_t e = set_dyn_smem_once(kern, smem);
  if (e == cudaSuccess)
    e = launch_chained(kern, static_cast<unsigned>(plan.ctas), ad::kThreads, smem, s, 0, tk, tv, q, reinterpret_cast<const uint8_t*>(k), reinterpret_cast<const uint8_t*>(v), o, p);
  if (e == cudaSuccess && merged)
    e = launch_chained(ad::attention_decode_stream_merge_kernel<T, D>, static_cast<unsigned>(units * p.heads_here), D, 0, s, 0, o, p, static_cast<int32_t>(plan.ctas));
  st = cuda_ok(err, e, "attention_decode_stream_kernel launch");
  if (merged) {
    e = cudaFreeAsync(p.part, s);
    if (st == TSM100_OK && e != cudaSuccess) st = cuda_ok(err, e, "cudaFreeAsync");
  }
  return st;
}

// How many clusters of `size` CTAs of the eight-warp decode kernel the GPU holds at once (asked once per
// kernel, size and device; 0 if such clusters cannot be placed at all).
template <typename T, int D>
inline int decode_lone_clusters(int size) {
  namespace ad = attn_decode;
  static int cached[64][2] = {};  // [device][size == 16]: 0 unknown, else count + 1
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 0;
  int& slot = cached[dev][size > ad::kMaxSplits ? 1 : 0];
  if (size != ad::kMaxSplits && size != ad::kMaxSplitsWide) return 0;
  if (slot == 0) {
    auto kern = DecodeTc<T, D, 3, 8>::kernel();
    constexpr int smem = DecodeTc<T, D, 3, 8>::smem();
    int clusters = 0;
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = static_cast<unsigned>(size);
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    cfg.blockDim = dim3(8 * 32);
    cfg.dynamicSmemBytes = smem;
    cfg.gridDim = dim3(static_cast<unsigned>(size));
    const bool ok = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) == cudaSuccess &&
                    cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess &&
                    cudaOccupancyMaxActiveClusters(&clusters, kern, &cfg) == cudaSuccess;
    if (!ok) (void)cudaGetLastError();  // the answer is "none", not an error of the caller's launch
    slot = (ok ? clusters : 0) + 1;
  }
  return slot - 1;
}

// f32 caches: from this many query heads per cache on, the tensor-core kernel (three TF32 products) is faster than
// the FP32-pipe kernel, whose instruction count grows with the heads while the cache row is read once either way
constexpr int kDecodeF32TensorCoreGroup = 5;

template <typename T, int D>
inline int32_t attention_decode_typed(std::string* err, const tsm100_attention_decode_desc* d, const void* q, const void* k,
                                      const void* v, void* o, uint32_t* status, cudaStream_t s) {
  int sms = 0;
  int32_t st = sm_count(err, &sms);
  if (st != TSM100_OK) return st;
  const int64_t units = static_cast<int64_t>(d->batch) * d->heads_kv;
  // split the positions of one (batch, KV head) over a cluster until the GPU is covered about twice, keeping
  // at least 256 positions per CTA
  int splits = 1;
  while (splits < attn_decode::kMaxSplits && units * splits < 2ll * sms && d->seq_len / (2 * splits) >= 256) splits *= 2;
  const int group = d->heads_q / d->heads_kv;
  const T* qp = static_cast<const T*>(q);
  const T* kp = static_cast<const T*>(k);
  const T* vp = static_cast<const T*>(v);
  T* op = static_cast<T*>(o);
  if constexpr (sizeof(T) == 2)
    if (status != nullptr && group <= attn_decode::stream::kRows) {
      const route::DecodeStream plan = route::decode_stream(units, d->seq_len, D, std::min(sms, attn_decode::stream::kMaxCtas));
      if (plan.ctas > 0) {
        st = attention_decode_stream_launch<T, D>(err, d, qp, kp, vp, op, plan, status, s);
        if (st != kNoScratch) return st;
        st = TSM100_OK;
      }
    }
  if (sizeof(T) == 2 || group >= kDecodeF32TensorCoreGroup) {
    // 16-bit storage, or f32 with several query heads per cache: tensor cores, up to 16 query heads of a group per
    // pass; 4 warps per CTA, so the GPU is covered about four times before the ranges get shorter than 256 positions
    splits = 1;
    while (splits < attn_decode::kMaxSplits && units * splits < 4ll * sms && d->seq_len / (2 * splits) >= 256) splits *= 2;
    // a handful of sequences: clusters of 16 if the GPU holds all of them at once (one CTA per SM; a B200
    // holds 7), so that most SMs take part
    if (splits == attn_decode::kMaxSplits && d->seq_len / (2 * attn_decode::kMaxSplitsWide) >= 256 &&
        units <= decode_lone_clusters<T, D>(attn_decode::kMaxSplitsWide))
      splits = attn_decode::kMaxSplitsWide;
    // so few units that clusters leave a third of the SMs or more idle: one CTA per SM with 512 positions or more each,
    // merged by a second kernel.  Eight KV heads: 35.2 us as clusters, 30.2 this way at 32768 positions, 15.3 / 11.0 at 8192;
    // one KV head, 32768 positions 22.6 / 13.4.
    if constexpr (sizeof(T) == 2) {
      const int64_t wide = std::min<int64_t>({attn_decode::mma::kMaxGlobalSplits, sms / std::max<int64_t>(units, 1), d->seq_len / 512});
      if (wide * 2 >= 3 * splits && wide > 1) {
        st = attention_decode_global_launch<T, D>(err, d, qp, kp, vp, op, static_cast<int>(wide), s);
        if (st != kNoScratch) return st;
        st = TSM100_OK;
      }
    }
    // every CTA alone on its SM from start to end: eight warps and a deeper ring, so that it hides its own latencies
    const bool lone = units * splits <= sms && (splits < attn_decode::kMaxSplits || units <= decode_lone_clusters<T, D>(splits));
    for (int base = 0; base < group && st == TSM100_OK; base += 16)
      st = lone ? attention_decode_mma_launch<T, D, 3, 8>(err, d, qp, kp, vp, op, base, std::min(16, group - base), splits, s)
                : attention_decode_mma_launch<T, D, 2, 4>(err, d, qp, kp, vp, op, base, std::min(16, group - base), splits, s);
    return st;
  }
  // groups wider than 8 query heads run in passes of 8 (the cache is then re-read, from L2 when it fits)
  for (int base = 0; base < group && st == TSM100_OK; base += 8) {
    const int here = std::min(8, group - base);
    if (here == 1) st = attention_decode_launch<T, 1, D>(err, d, qp, kp, vp, op, base, here, splits, s);
    else if (here == 2) st = attention_decode_launch<T, 2, D>(err, d, qp, kp, vp, op, base, here, splits, s);
    else if (here <= 4) st = attention_decode_launch<T, 4, D>(err, d, qp, kp, vp, op, base, here, splits, s);
    else st = attention_decode_launch<T, 8, D>(err, d, qp, kp, vp, op, base, here, splits, s);
  }
  return st;
}

inline int32_t attention_decode(std::string* err, const tsm100_attention_decode_desc* d, const void* q, const void* k,
                                const void* v, void* o, void* stream, uint32_t* status = nullptr) {
  if (!d || !q || !k || !v || !o) return op_fail(err, TSM100_ERR_INVALID, "attention_decode: null argument");
  if (!dtype_valid(d->dtype)) return op_fail(err, TSM100_ERR_INVALID, "attention_decode: unknown dtype");
  if (d->batch < 0 || d->heads_q <= 0 || d->heads_kv <= 0 || d->seq_len < 0 || d->max_seq < d->seq_len)
    return op_fail(err, TSM100_ERR_INVALID, "attention_decode: bad shape (need heads > 0 and 0 <= seq_len <= max_seq)");
  if (d->heads_q % d->heads_kv != 0)
    return op_fail(err, TSM100_ERR_INVALID, "attention_decode: heads_q must be a multiple of heads_kv");
  if (d->head_dim != 64 && d->head_dim != 128)
    return op_fail(err, TSM100_ERR_INVALID, "attention_decode: head_dim must be 64 or 128");
  if (!aligned16(q) || !aligned16(k) || !aligned16(v) || !aligned16(o))
    return op_fail(err, TSM100_ERR_INVALID, "attention_decode: buffers must be 16-byte aligned");
  if (d->batch == 0) return TSM100_OK;
  if (static_cast<int64_t>(d->batch) * d->heads_kv * attn_decode::kMaxSplitsWide > 0x7fffffff)
    return op_fail(err, TSM100_ERR_INVALID, "attention_decode: too many (batch, KV head) units for one launch");
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const bool d128 = d->head_dim == 128;
  switch (d->dtype) {
    case TSM100_F32:
      return d128 ? attention_decode_typed<float, 128>(err, d, q, k, v, o, status, s) : attention_decode_typed<float, 64>(err, d, q, k, v, o, status, s);
    case TSM100_BF16:
      return d128 ? attention_decode_typed<__nv_bfloat16, 128>(err, d, q, k, v, o, status, s)
                  : attention_decode_typed<__nv_bfloat16, 64>(err, d, q, k, v, o, status, s);
    default:
      return d128 ? attention_decode_typed<__half, 128>(err, d, q, k, v, o, status, s) : attention_decode_typed<__half, 64>(err, d, q, k, v, o, status, s);
  }
}

template <bool kBf16, int D>
inline int32_t attention_tc_launch(std::string* err, const tsm100_attention_desc* d, const void* q, const void* k,
                                   const void* v, void* o, uint32_t* status, cudaStream_t s) {
  namespace at = attn;
  CUtensorMap tq, tk, tv;
  const uint64_t S = d->seq, d_row = d->head_dim;
  const uint64_t nq = static_cast<uint64_t>(d->batch) * d->heads_q, nkv = static_cast<uint64_t>(d->batch) * d->heads_kv;
  int32_t st = make_tmap_16bit_3d(err, &tq, q, d_row, S, nq, d_row, S * d_row, 64, at::kBQ, kBf16);
  if (st == TSM100_OK) st = make_tmap_16bit_3d(err, &tk, k, d_row, S, nkv, d_row, S * d_row, 64, at::kBKV, kBf16);
  if (st == TSM100_OK) st = make_tmap_16bit_3d(err, &tv, v, d_row, S, nkv, d_row, S * d_row, 64, at::kBKV, kBf16);
  if (st != TSM100_OK) return st;
  at::Params p;
  p.seq = d->seq;
  p.heads_q = d->heads_q;
  p.heads_kv = d->heads_kv;
  p.batch = d->batch;
  p.causal = d->causal ? 1 : 0;
  p.kv_band = attention_kv_band(S, static_cast<int64_t>(nkv), d_row);
  p.scale_log2 = static_cast<float>((1.0 / std::sqrt(static_cast<double>(d->head_dim))) * 1.4426950408889634);
  p.status = status;
  p.seq_kv = d->seq;
  p.q_offset = 0;
  p.o_row_stride = p.o_head_stride = 0;
  p.head_dim = d->head_dim;
  return attention_fwd_launch<kBf16, false, D>(err, tq, tk, tv, o, p, static_cast<int64_t>(nq), d->seq, s);
}

inline int32_t attention(std::string* err, const tsm100_attention_desc* d, const void* q, const void* k,
                         const void* v, void* o, uint32_t* status, void* stream) {
  if (!d || !q || !k || !v || !o) return op_fail(err, TSM100_ERR_INVALID, "attention: null argument");
  if (!dtype_valid(d->dtype)) return op_fail(err, TSM100_ERR_INVALID, "attention: unknown dtype");
  if (d->batch < 0 || d->heads_q < 0 || d->heads_kv < 0 || d->seq < 0 || d->head_dim < 0)
    return op_fail(err, TSM100_ERR_INVALID, "attention: negative shape");
  if (d->batch == 0 || d->heads_q == 0 || d->seq == 0 || d->head_dim == 0) return TSM100_OK;
  if (d->heads_kv <= 0 || d->heads_q % d->heads_kv != 0)
    return op_fail(err, TSM100_ERR_INVALID, "attention: heads_q must be a positive multiple of heads_kv");
  if (d->head_dim > attn_simt::kMaxD) return op_fail(err, TSM100_ERR_INVALID, "attention: head_dim > 256 unsupported");
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  if (attention_tc_ok(d->dtype, d->head_dim, d->seq, static_cast<int64_t>(d->batch) * d->heads_q, d->seq, status, q, k, v, o)) {
    const bool wide = d->head_dim == attn::kD;
    if (d->dtype == TSM100_BF16)
      return wide ? attention_tc_launch<true, 128>(err, d, q, k, v, o, status, s) : attention_tc_launch<true, 64>(err, d, q, k, v, o, status, s);
    return wide ? attention_tc_launch<false, 128>(err, d, q, k, v, o, status, s) : attention_tc_launch<false, 64>(err, d, q, k, v, o, status, s);
  }
  if (d->dtype == TSM100_F32) return attention_simt_launch<float>(err, d, q, k, v, o, status, s);
  if (d->dtype == TSM100_BF16) return attention_simt_launch<__nv_bfloat16>(err, d, q, k, v, o, status, s);
  return attention_simt_launch<__half>(err, d, q, k, v, o, status, s);
}

}  // namespace ops
}  // namespace tsm100
