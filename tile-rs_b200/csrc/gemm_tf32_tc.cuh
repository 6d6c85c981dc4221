// f32 GEMM on the 5th-generation tensor cores (tcgen05, kind::tf32) with f32-grade results.
//
//   C[b][M,N] = A[b][M,K] * B[b]       all f32, row-major; B [K,N] or stored [N,K]
//   __tile_matmul_f32 / __tile_matmul_transposed_f32 (crates/tile_std/src/tile.rs:192-193, :2017-2031);
//   semantics linalg.fill 0 + linalg.matmul (crates/rustc_codegen_tile/src/mlir_to_linalg.rs:1345-1393).
//
// One TF32 product keeps 11 significant bits, which cannot meet a 1e-5 bar; three can.  Every operand x is
// split once, by a streaming pass, into hi = tf32(x) (round to nearest) and lo = tf32(x - hi); a product is
// then  lo*hi + hi*lo + hi*hi  on the tensor cores, f32 accumulation in tensor memory; what is dropped (lo*lo,
// the rounding of lo) is below 2^-21 of |a||b|.  The same pass writes B's planes K-major ([N][K]), so the
// contraction kernel sees K-major operands only, whatever layout B came in.
//
// The tensor core rounds its f32 accumulator toward zero at every instruction, so a long K accumulated in one go
// drifts by about 2^-25.6 per instruction, all in one direction (3e-5 of the result at K = 4096).  The K loop is
// therefore cut into chunks of p.chunk_kb k-blocks: each chunk is accumulated from zero in one of two tensor-memory
// accumulators and then added, round-to-nearest, to running sums that the eight epilogue warps keep in registers
// (128 x 256 tile / 256 threads = 128 sums per thread) while the tensor core works on the next chunk.
//
// Per CTA (one per SM, persistent over 128 x 256 output tiles): warp 0 TMA producer (four planes per 32-deep
// k-block, 96 KiB per stage, two stages, no multicast), warp 1 tensor-memory allocation and MMA issue (12
// instructions of 128 x 256 x 8 per k-block), warps 2..9 chunk drain and output.
// Roofline: tensor pipe at the TF32 rate / 3.  Algorithmic work 2*M*N*K flop per problem.
#pragma once

#include "ptx.cuh"

namespace tsm100 {
namespace gemm_tf32_tc {

constexpr int kBM = 128;
constexpr int kBN = 256;
constexpr int kBK = 32;                  // 32 x f32 = one 128-byte swizzle row
constexpr int kStages = 2;
constexpr int kUmmaK = 8;                // 32 bytes of K per instruction
constexpr int kThreads = 320;            // warp 0 TMA, warp 1 MMA, warps 2..9 epilogue
constexpr int kAPlane = kBM * kBK * 4;   // 16 KiB
constexpr int kBPlane = kBN * kBK * 4;   // 32 KiB
constexpr int kStageBytes = 2 * kAPlane + 2 * kBPlane;  // 96 KiB: A_hi, A_lo, B_hi, B_lo
constexpr int kTmemCols = 512;           // two 256-column accumulators
constexpr int kGroupM = 16;              // m-blocks per rasterisation band (L2 reuse)

struct Redo {            // of a CTA's second pass (kRedo kernels)
  uint32_t any;          // one of its blocks holds an infinity or a NaN
  uint32_t pick, got;
};

struct alignas(8) Barriers {
  uint64_t full[kStages];
  uint64_t empty[kStages];
  uint64_t acc_full[2];
  uint64_t acc_empty[2];
  uint32_t tmem_base;
  uint32_t abort_flag;
  Redo redo;
};
// C is written in 32 x 32 blocks through shared memory, so that a warp's store covers whole 128-byte pieces of rows.
constexpr int kStagingFloats = 32 * 32;                       // per epilogue warp
constexpr int kStagingBytes = 8 * kStagingFloats * 4;
constexpr int kSmemBytes = kStages * kStageBytes + kStagingBytes + sizeof(Barriers) + 1024;
static_assert(kSmemBytes <= 227 * 1024, "shared memory budget of one CTA");

struct Params {
  int32_t m, n, k, batch;
  int32_t m_blocks, n_blocks;
  int64_t c_batch_stride;  // elements
  int64_t ldc;             // row pitch of C in elements
  uint32_t* status;
  int32_t vec_store;       // every row of C starts on a 16-byte boundary
  int32_t chunk_kb;        // 32-deep k-blocks per accumulation chunk
  // kRedo kernels: the operands as they came, and a word per 128 x 128 block of C, [batch][ceil(m / 128)][ceil(n / 128)], zero
  // at the start (see second_pass)
  uint32_t* flags;
  int32_t b_transposed;
  const float *a, *b;
  int64_t lda, ldb, a_batch_stride, b_batch_stride;
  // pair kernels: tiles from whole_tiles on are worked on by `splits` pairs each (see pair::Walk); their partial sums, and a counter
  // per CTA's half of such a tile, zero at the start
  int32_t whole_tiles, splits;
  float4* part;
  uint32_t* arrivals;
};

// x rounded to the nearest TF32 number (10 explicit mantissa bits; ties away from zero).  The conversion instruction, not
// an add on the bits: that would carry a NaN of all ones into a zero.
__device__ __forceinline__ float tf32_rn(float x) {
  uint32_t r;
  asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(r) : "f"(x));
  return __uint_as_float(r & 0xffffe000u);
}

// ---------------------------------------------------------------------------
// the split pass
// ---------------------------------------------------------------------------
// One launch splits both operands (two launches cost a ramp and a tail more).
// rows: src [rows][cols] with row pitch ld -> hi, lo [rows][cols] with row pitch kp, a multiple of 4 >= cols, so that every
// plane row starts on a 16-byte boundary whatever cols is (the columns from cols to kp are never read: the tensor maps
// end at cols).  One thread per four values; kVec: rows of src start on 16-byte boundaries and cols % 4 == 0, else the
// four values are loaded one by one.
// transposed: src [cols][rows] with row pitch ld -> the same planes, 32 x 32 tiles through shared memory.
struct SplitOperand {
  const float* src;
  float *hi, *lo;
  int64_t ld, batch_stride;   // of src, in elements
  int64_t rows;
  int32_t cols, kp;
  int32_t blocks;             // blocks of the launch that work on it
};

template <bool kVec>
__device__ __forceinline__ void split_rows(const SplitOperand& p, int block, int batch) {
  const int64_t vec_per_row = p.kp >> 2;
  const int64_t total = p.rows * vec_per_row;
  const float* s = p.src + batch * p.batch_stride;
  float* h = p.hi + batch * p.rows * p.kp;
  float* l = p.lo + batch * p.rows * p.kp;
  for (int64_t i = block * static_cast<int64_t>(blockDim.x) + threadIdx.x; i < total; i += static_cast<int64_t>(p.blocks) * blockDim.x) {
    const int64_t r = i / vec_per_row, c4 = (i - r * vec_per_row) << 2;
    float4 x;
    if (kVec) {
      x = *reinterpret_cast<const float4*>(s + r * p.ld + c4);
    } else {
      const float* q = s + r * p.ld + c4;
      x.x = q[0];  // c4 < cols, because kp - cols < 4
      x.y = c4 + 1 < p.cols ? q[1] : 0.f;
      x.z = c4 + 2 < p.cols ? q[2] : 0.f;
      x.w = c4 + 3 < p.cols ? q[3] : 0.f;
    }
    float4 a, b;
    a.x = tf32_rn(x.x), a.y = tf32_rn(x.y), a.z = tf32_rn(x.z), a.w = tf32_rn(x.w);
    b.x = tf32_rn(x.x - a.x), b.y = tf32_rn(x.y - a.y), b.z = tf32_rn(x.z - a.z), b.w = tf32_rn(x.w - a.w);
    *reinterpret_cast<float4*>(h + r * p.kp + c4) = a;
    *reinterpret_cast<float4*>(l + r * p.kp + c4) = b;
  }
}

// One 32 x 32 tile per block, 256 threads (32 x 8).
__device__ __forceinline__ void split_transposed(const SplitOperand& p, int block, int batch, float (&tile)[32][33]) {
  const float* s = p.src + batch * p.batch_stride;
  float* h = p.hi + batch * p.rows * p.kp;
  float* l = p.lo + batch * p.rows * p.kp;
  const int row_tiles = static_cast<int>((p.rows + 31) / 32);
  const int n0 = block % row_tiles * 32, k0 = block / row_tiles * 32;
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const int kk = k0 + ty + 8 * j, nn = n0 + tx;
    tile[ty + 8 * j][tx] = (kk < p.cols && nn < p.rows) ? s[static_cast<int64_t>(kk) * p.ld + nn] : 0.f;
  }
  __syncthreads();
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const int nn = n0 + ty + 8 * j, kk = k0 + tx;
    if (nn < p.rows && kk < p.cols) {
      const float x = tile[tx][ty + 8 * j];
      const float a = tf32_rn(x);
      h[static_cast<int64_t>(nn) * p.kp + kk] = a;
      l[static_cast<int64_t>(nn) * p.kp + kk] = tf32_rn(x - a);
    }
  }
}

// grid (a.blocks + b.blocks, batch); the blocks of the transposed operand come first.  zero[0 .. n_zero) is cleared on the way:
// the flags of the contraction's second pass.
template <bool kVec, bool kTransposeB>
__global__ void __launch_bounds__(256)
split_operands_kernel(const SplitOperand a, const SplitOperand b, uint32_t* zero, int64_t n_zero) {
  ptx::launch_dependents();
  ptx::wait_prior_grid();
  if (blockIdx.y == 0)
    for (int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; i < n_zero; i += static_cast<int64_t>(gridDim.x) * blockDim.x) zero[i] = 0u;
  __shared__ float tile[kTransposeB ? 32 : 1][33];
  const int block = static_cast<int>(blockIdx.x);
  if (block < b.blocks) {
    if constexpr (kTransposeB) split_transposed(b, block, blockIdx.y, tile);
    else split_rows<kVec>(b, block, blockIdx.y);
  } else {
    split_rows<kVec>(a, block - b.blocks, blockIdx.y);
  }
}

// ---------------------------------------------------------------------------
// the contraction
// ---------------------------------------------------------------------------
// One warp writes its 32 rows x 32 columns of C (lane = row of `sum`, first element C[row0][col0]), transposed through
// `staging`: 16-byte unit u of row r lies at unit u ^ (r & 7), so neither side has bank conflicts.  vec_store: 16-byte
// stores, four rows at a time, otherwise 4-byte stores of one row.  Writing rows from the lanes that hold them costs more
// even where they are aligned: every store then touches 32 rows (2000 x 3000 x 1500 on 256 x 128 tiles: 127 us against 117).
// Columns of an accumulator read at a time.  32 leave the kRedo kernels, whose second pass holds registers too, with spills: 1999 x 3001 x
// 1501 130.2 us with 32, 124.7 with 16; no difference for the others.
constexpr int kDrain = 16;
// kRedo (problems that the FP32 pipe could take as well): a block with an infinity or a NaN is marked for second_pass.
template <bool kRedo>
__device__ __forceinline__ void store_block_32x32(float* __restrict__ c, const Params& p, int batch, int row0, int col0,
                                                  const float (&sum)[32], float* staging, int lane, Redo* redo) {
  float* cb = c + batch * p.c_batch_stride;
  if (kRedo && row0 < p.m && col0 < p.n) {
    float z = 0.f;  // NaN where anything is infinite or NaN (rows and columns past C are so only beside such ones of C)
#pragma unroll
    for (int i = 0; i < 32; ++i) z = fmaf(sum[i], 0.f, z);
    if (__any_sync(0xffffffffu, z != 0.f) && lane == 0) {
      p.flags[(static_cast<int64_t>(batch) * ((p.m + 127) / 128) + row0 / 128) * ((p.n + 127) / 128) + col0 / 128] = 2u + blockIdx.x;
      redo->any = 1u;
    }
  }
  float4* st4 = reinterpret_cast<float4*>(staging);
  __syncwarp();  // the previous block has been read
#pragma unroll
  for (int i = 0; i < 8; ++i) st4[lane * 8 + (i ^ (lane & 7))] = make_float4(sum[4 * i], sum[4 * i + 1], sum[4 * i + 2], sum[4 * i + 3]);
  __syncwarp();
  const int rows = min(32, p.m - row0);
  if (p.vec_store && col0 + 32 <= p.n) {
    const int u = lane & 7;
    float* dst = cb + static_cast<int64_t>(row0) * p.ldc + col0 + u * 4;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int r = i * 4 + (lane >> 3);
      if (r < rows) *reinterpret_cast<float4*>(dst + r * p.ldc) = st4[r * 8 + (u ^ (r & 7))];
    }
  } else if (col0 + lane < p.n) {
    float* dst = cb + static_cast<int64_t>(row0) * p.ldc + col0 + lane;
    for (int r = 0; r < rows; ++r) dst[r * p.ldc] = staging[r * 32 + (((lane >> 2) ^ (r & 7)) << 2) + (lane & 3)];
  }
}

// ---------------------------------------------------------------------------
// the second pass of kRedo kernels
// ---------------------------------------------------------------------------
// An infinity split into hi + lo is infinity + NaN, and a hi part can round up to infinity, so outputs that come out infinite or
// NaN are summed again in plain f32 and replaced.  That runs when a CTA has written all of its tiles: no barrier of the
// pipeline waits for it, however long it takes, and a CTA whose outputs are all finite does nothing.  A CTA that marked
// blocks publishes them then, walks over the published blocks and sums those it can claim until it finds none, so that CTAs with few tiles
// help those with many.  Nobody waits for a block to be published: its own CTA comes for it.
// Every output infinite: 2049 x 2051 x 1501 590 us (610 on the FP32-pipe kernel), 1999 x 3001 x 1501 840 (770), 4097 x 4097 x
// 2001 2900 (2650); 2049 x 2051 x 301 0.19 ms, 20 with one dependent sum per lane inside the epilogue.
constexpr int kEpilogueThreads = 256;
__device__ __forceinline__ void epilogue_sync() { asm volatile("barrier.cta.sync 1, 256;" ::: "memory"); }
__device__ __forceinline__ bool epilogue_any(bool x) {
  uint32_t r;
  asm volatile(
      "{\n"
      ".reg .pred p, q;\n"
      "setp.ne.u32 p, %1, 0;\n"
      "barrier.cta.red.or.pred q, 1, 256, p;\n"
      "selp.u32 %0, 1, 0, q;\n"
      "}\n" : "=r"(r) : "r"(static_cast<uint32_t>(x)) : "memory");
  return r != 0;
}
// One 128 x 128 block, 256 threads with 8 x 8 sums each, in the order of k; the next 16 of k are loaded meanwhile.
// `panels`: kPanelFloats of shared memory.
constexpr int kPanelK = 16, kPanelPitch = 132;
constexpr int kPanelFloats = 2 * kPanelK * kPanelPitch;
static_assert(kPanelFloats * 4 <= kStages * kStageBytes, "the panels take the place of the stages");
__device__ __forceinline__ void sum_block_again(const Params& p, float* c, float* panels, int batch, int row0, int col0, int tid) {
  float *sa = panels, *sb = panels + kPanelK * kPanelPitch;
  const int tx = tid & 15, ty = tid >> 4;
  // this thread's eight values of a panel of A: row (tid >> 4) + 16 i, k = tid & 15; of B the same, or, stored [K][N], column
  // tid & 127, k = (tid >> 7) + 2 i
  const bool bt = p.b_transposed != 0;
  const int m = p.m, n = p.n, k = p.k;
  const float* a = p.a + batch * p.a_batch_stride + (row0 + ty) * p.lda + tx;
  const float* b = p.b + batch * p.b_batch_stride + (bt ? (col0 + ty) * p.ldb + tx : (tid >> 7) * p.ldb + col0 + (tid & 127));
  const int64_t a_step = 16 * p.lda, b_step = (bt ? 16 : 2) * p.ldb, b_panel = bt ? kPanelK : kPanelK * p.ldb;
  const int b_col = col0 + (bt ? ty : tid & 127), b_col_step = bt ? 16 : 0, b_k = bt ? tx : tid >> 7, b_k_step = bt ? 0 : 2;
  float* const sa_at = sa + tx * kPanelPitch + ty;
  float* const sb_at = bt ? sb + tx * kPanelPitch + ty : sb + (tid >> 7) * kPanelPitch + (tid & 127);
  const int sb_step = bt ? 16 : 2 * kPanelPitch;
  float acc[8][8], na[8], nb[8];
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int j = 0; j < 8; ++j) acc[i][j] = 0.f;
  auto fetch = [&](int k0) {
    const float *pa = a, *pb = b;
#pragma unroll
    for (int i = 0; i < 8; ++i, pa += a_step, pb += b_step) {
      na[i] = row0 + ty + 16 * i < m && k0 + tx < k ? *pa : 0.f;
      nb[i] = b_col + i * b_col_step < n && k0 + b_k + i * b_k_step < k ? *pb : 0.f;
    }
    a += kPanelK;
    b += b_panel;
  };
  fetch(0);
  for (int k0 = 0; k0 < k; k0 += kPanelK) {
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      sa_at[i * 16] = na[i];
      sb_at[i * sb_step] = nb[i];
    }
    epilogue_sync();
    fetch(k0 + kPanelK);
#pragma unroll 2
    for (int kk = 0; kk < kPanelK; ++kk) {
      alignas(16) float x[8], w[8];
#pragma unroll
      for (int i = 0; i < 8; i += 4) {
        *reinterpret_cast<float4*>(x + i) = *reinterpret_cast<const float4*>(sa + kk * kPanelPitch + ty * 8 + i);
        *reinterpret_cast<float4*>(w + i) = *reinterpret_cast<const float4*>(sb + kk * kPanelPitch + tx * 4 + i * 16);
      }
#pragma unroll
      for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < 8; ++j) acc[i][j] = fmaf(x[i], w[j], acc[i][j]);
    }
    epilogue_sync();
  }
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int r = row0 + ty * 8 + i;
    if (r >= m) break;
    float* out = c + batch * p.c_batch_stride + r * p.ldc + col0 + tx * 4;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const int at = (j & 3) + (j >> 2) * 64;
      if (col0 + tx * 4 + at < n && !(fabsf(__ldcg(out + at)) < INFINITY)) out[at] = acc[i][j];
    }
  }
}
// Called by all eight epilogue warps after their last tile, with `ok` false if a wait of theirs gave up.  The stages are free: the last
// accumulator is complete, so every copy into them and every product from them has retired.
__device__ __noinline__ void second_pass(const Params& p, float* c, float* panels, Redo* redo, bool ok) {
  const int tid = static_cast<int>(threadIdx.x) - 64;
  if (!epilogue_any(redo->any != 0u) || epilogue_any(!ok)) return;
  const int rows = (p.m + 127) / 128, cols = (p.n + 127) / 128;
  const int total = p.batch * rows * cols;
  volatile uint32_t* flags = p.flags;
  __threadfence();  // this thread's part of C before the flags that say it is there
  epilogue_sync();
  for (int i = tid; i < total; i += kEpilogueThreads)
    if (flags[i] == 2u + blockIdx.x) atomicExch(&p.flags[i], 1u);
  epilogue_sync();
  const int start = static_cast<int>(static_cast<int64_t>(blockIdx.x) * total / gridDim.x);
  bool found = true;
  while (found) {
    found = false;
    for (int at = 0; at < total; at += kEpilogueThreads) {
      const int i = (start + at + tid) % total;
      for (;;) {
        const bool ready = at + tid < total && flags[i] == 1u;
        if (!epilogue_any(ready)) break;
        if (tid == 0) redo->pick = kEpilogueThreads;
        epilogue_sync();
        if (ready) atomicMin(&redo->pick, static_cast<uint32_t>(tid));
        epilogue_sync();
        const int pick = static_cast<int>(redo->pick);
        if (tid == pick) redo->got = atomicCAS(&p.flags[i], 1u, 0u) == 1u ? 1u : 0u;
        epilogue_sync();
        if (redo->got != 0u) {
          __threadfence();
          const int block = (start + at + pick) % total;
          sum_block_again(p, c, panels, block / (rows * cols), block / cols % rows * 128, block % cols * 128, tid);
          found = true;
        }
      }
    }
  }
}

__device__ __forceinline__ void tile_coords(const Params& p, int tile, int& b, int& mb, int& nb) {
  const int per_batch = p.m_blocks * p.n_blocks;
  b = tile / per_batch;
  int t = tile - b * per_batch;
  const int band_tiles = kGroupM * p.n_blocks;
  const int band = t / band_tiles;
  const int first_m = band * kGroupM;
  const int rows_in_band = min(kGroupM, p.m_blocks - first_m);
  t -= band * band_tiles;
  mb = first_m + t % rows_in_band;
  nb = t / rows_in_band;
}

// 32-bit instruction descriptor for kind::tf32 with f32 accumulation, both operands K-major.
//   [4,6) D format (1 = f32)  [7,10) A format  [10,13) B format (2 = tf32)  [17,23) N >> 3  [24,29) M >> 4
__host__ __device__ constexpr uint32_t make_idesc_tf32(uint32_t m, uint32_t n) {
  return (1u << 4) | (2u << 7) | (2u << 10) | ((n >> 3) << 17) | ((m >> 4) << 24);
}

__device__ __forceinline__ void tcgen05_mma_tf32_ss(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc,
                                                    uint32_t accumulate) {
  asm volatile(
      "{\n"
      ".reg .pred p;\n"
      "setp.ne.b32 p, %4, 0;\n"
      "tcgen05.mma.cta_group::1.kind::tf32 [%0], %1, %2, %3, p;\n"
      "}\n" ::"r"(d_tmem),
      "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate)
      : "memory");
}

template <bool kRedo>
__global__ void __launch_bounds__(kThreads, 1)
gemm_tf32_tc_kernel(const __grid_constant__ CUtensorMap tmap_a_hi, const __grid_constant__ CUtensorMap tmap_a_lo,
                    const __grid_constant__ CUtensorMap tmap_b_hi, const __grid_constant__ CUtensorMap tmap_b_lo,
                    float* __restrict__ c, const __grid_constant__ Params p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  Barriers* bars = reinterpret_cast<Barriers*>(smem + kStages * kStageBytes + kStagingBytes);

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const int num_tiles = p.batch * p.m_blocks * p.n_blocks;
  const int num_kb = (p.k + kBK - 1) / kBK;
  const int num_chunks = (num_kb + p.chunk_kb - 1) / p.chunk_kb;
  volatile uint32_t* abort_flag = &bars->abort_flag;

  if (threadIdx.x == 0) {
    for (int s = 0; s < kStages; ++s) {
      ptx::mbar_init(&bars->full[s], 1);
      ptx::mbar_init(&bars->empty[s], 1);
    }
    for (int a = 0; a < 2; ++a) {
      ptx::mbar_init(&bars->acc_full[a], 1);
      ptx::mbar_init(&bars->acc_empty[a], 8);  // one arrival per epilogue warp
    }
    bars->abort_flag = 0;
    bars->redo.any = 0;
    ptx::fence_mbar_init();
  }
  if (warp == 1) {
    ptx::tmem_alloc(&bars->tmem_base, kTmemCols);
    ptx::tmem_relinquish_alloc_permit();
  }
  ptx::tcgen05_fence_before_thread_sync();
  __syncthreads();
  ptx::tcgen05_fence_after_thread_sync();
  const uint32_t tmem_base = bars->tmem_base;
  ptx::launch_dependents();
  ptx::wait_prior_grid();

  if (warp == 0) {
    // ------------------------------ TMA producer ------------------------------
    if (lane == 0) {
      ptx::prefetch_tensormap(&tmap_a_hi);
      ptx::prefetch_tensormap(&tmap_a_lo);
      ptx::prefetch_tensormap(&tmap_b_hi);
      ptx::prefetch_tensormap(&tmap_b_lo);
      int stage = 0;
      uint32_t phase = 0;
      bool ok = true;
      for (int tile = blockIdx.x; tile < num_tiles && ok; tile += gridDim.x) {
        int b, mb, nb;
        tile_coords(p, tile, b, mb, nb);
        for (int kb = 0; kb < num_kb; ++kb) {
          if (!ptx::mbar_wait(&bars->empty[stage], phase ^ 1u, abort_flag, p.status, 41)) {
            ok = false;
            break;
          }
          uint8_t* st = smem + stage * kStageBytes;
          ptx::mbar_arrive_expect_tx(&bars->full[stage], kStageBytes);
          ptx::tma_load_3d(st, &tmap_a_hi, &bars->full[stage], kb * kBK, mb * kBM, b);
          ptx::tma_load_3d(st + kAPlane, &tmap_a_lo, &bars->full[stage], kb * kBK, mb * kBM, b);
          ptx::tma_load_3d(st + 2 * kAPlane, &tmap_b_hi, &bars->full[stage], kb * kBK, nb * kBN, b);
          ptx::tma_load_3d(st + 2 * kAPlane + kBPlane, &tmap_b_lo, &bars->full[stage], kb * kBK, nb * kBN, b);
          if (++stage == kStages) {
            stage = 0;
            phase ^= 1u;
          }
        }
      }
    }
  } else if (warp == 1) {
    // ------------------------------ MMA issuer --------------------------------
    if (lane == 0) {
      constexpr uint32_t idesc = make_idesc_tf32(kBM, kBN);
      constexpr uint64_t kmajor = ptx::make_smem_desc_base(16, 1024);  // 8-row groups 1024 B apart
      constexpr uint32_t kstep = kUmmaK * 4;                            // 32 B inside the swizzle row
      int stage = 0;
      uint32_t phase = 0;
      bool ok = true;
      uint32_t chunk_count = 0;  // chunks issued by this CTA so far: picks the accumulator and its barrier phase
      for (int tile = blockIdx.x; tile < num_tiles && ok; tile += gridDim.x) {
        for (int ch = 0; ch < num_chunks && ok; ++ch, ++chunk_count) {
          const uint32_t acc = chunk_count & 1u;
          const uint32_t acc_phase = (chunk_count >> 1) & 1u;
          if (!ptx::mbar_wait_relaxed(&bars->acc_empty[acc], acc_phase ^ 1u, abort_flag, p.status, 42)) {
            ok = false;
            break;
          }
          ptx::tcgen05_fence_after_thread_sync();
          const uint32_t d_tmem = tmem_base + acc * kBN;
          const int kb_end = min(num_kb, (ch + 1) * p.chunk_kb);
          for (int kb = ch * p.chunk_kb; kb < kb_end; ++kb) {
            if (!ptx::mbar_wait_relaxed(&bars->full[stage], phase, abort_flag, p.status, 43)) {
              ok = false;
              break;
            }
            ptx::tcgen05_fence_after_thread_sync();
            const uint32_t a_hi = ptx::smem_u32(smem + stage * kStageBytes);
            const uint32_t a_lo = a_hi + kAPlane;
            const uint32_t b_hi = a_hi + 2 * kAPlane;
            const uint32_t b_lo = b_hi + kBPlane;
            const bool first_kb = kb == ch * p.chunk_kb;
            // the small products first, then the large ones
#pragma unroll
            for (int kk = 0; kk < kBK / kUmmaK; ++kk) {
              const uint32_t off = kk * kstep;
              tcgen05_mma_tf32_ss(d_tmem, ptx::smem_desc(kmajor, a_lo + off), ptx::smem_desc(kmajor, b_hi + off), idesc,
                                  (first_kb && kk == 0) ? 0u : 1u);
              tcgen05_mma_tf32_ss(d_tmem, ptx::smem_desc(kmajor, a_hi + off), ptx::smem_desc(kmajor, b_lo + off), idesc, 1u);
            }
#pragma unroll
            for (int kk = 0; kk < kBK / kUmmaK; ++kk)
              tcgen05_mma_tf32_ss(d_tmem, ptx::smem_desc(kmajor, a_hi + kk * kstep), ptx::smem_desc(kmajor, b_hi + kk * kstep), idesc, 1u);
            ptx::tcgen05_commit(&bars->empty[stage]);  // stage reusable once these MMAs retire
            if (++stage == kStages) {
              stage = 0;
              phase ^= 1u;
            }
          }
          if (ok) ptx::tcgen05_commit(&bars->acc_full[acc]);
        }
      }
    }
  } else {
    // ------------------------------ chunk drain and output ----------------------
    const int quad = warp & 3;            // TMEM lanes [32*quad, 32*quad+32) belong to this warp
    const int half = (warp - 2) >> 2;     // which 128 columns of the 256-column accumulator
    float* staging = reinterpret_cast<float*>(smem + kStages * kStageBytes) + (warp - 2) * kStagingFloats;
    const uint32_t lane_addr = tmem_base + (static_cast<uint32_t>(quad * 32) << 16) + half * 128;
    uint32_t chunk_count = 0;
    bool alive = true;
    for (int tile = blockIdx.x; tile < num_tiles && alive; tile += gridDim.x) {
      int b, mb, nb;
      tile_coords(p, tile, b, mb, nb);
      float sum[4][32];
#pragma unroll
      for (int cc = 0; cc < 4; ++cc)
#pragma unroll
        for (int i = 0; i < 32; ++i) sum[cc][i] = 0.f;
      for (int ch = 0; ch < num_chunks; ++ch, ++chunk_count) {
        const uint32_t acc = chunk_count & 1u;
        const uint32_t acc_phase = (chunk_count >> 1) & 1u;
        // tcgen05.ld is warp-collective: leave the loop only as a whole warp
        const bool ready = ptx::mbar_wait(&bars->acc_full[acc], acc_phase, abort_flag, p.status, 44);
        if (!__all_sync(0xffffffffu, ready)) {
          alive = false;
          break;
        }
        ptx::tcgen05_fence_after_thread_sync();
#pragma unroll
        for (int cc = 0; cc < 4; ++cc) {
#pragma unroll
          for (int h = 0; h < 32; h += kDrain) {
            uint32_t v[kDrain];
            ptx::tmem_ld_32x32b_x16(lane_addr + acc * kBN + cc * 32 + h, v);
            ptx::tmem_ld_wait();
#pragma unroll
            for (int i = 0; i < kDrain; ++i) sum[cc][h + i] += __uint_as_float(v[i]);  // round-to-nearest add of the chunk
          }
        }
        ptx::tcgen05_fence_before_thread_sync();
        __syncwarp();
        if (lane == 0) ptx::mbar_arrive(&bars->acc_empty[acc]);
      }
      if (!alive) break;
#pragma unroll
      for (int cc = 0; cc < 4; ++cc)
        store_block_32x32<kRedo>(c, p, b, mb * kBM + quad * 32, nb * kBN + half * 128 + cc * 32, sum[cc], staging, lane, &bars->redo);
    }
    if (kRedo) second_pass(p, c, reinterpret_cast<float*>(smem), &bars->redo, alive);
  }

  // ------------------------------ teardown ------------------------------------
  if (*abort_flag != 0u) {
    // A wait gave up: give copies and MMAs already in flight time to land before
    // shared and tensor memory are released.
    const unsigned long long t0 = ptx::globaltimer_ns();
    while (ptx::globaltimer_ns() - t0 < 1000000ull) {
    }
  }
  ptx::tcgen05_fence_before_thread_sync();
  __syncthreads();
  if (warp == 1) {
    ptx::tcgen05_fence_after_thread_sync();
    ptx::tmem_dealloc(tmem_base, kTmemCols);
  }
}

// ---------------------------------------------------------------------------
// the contraction on CTA pairs (tcgen05 cta_group::2): a 256 x 256 output tile per pair of SMs
// ---------------------------------------------------------------------------
// With hi and lo planes a single CTA's stage is 96 KiB: two stages fit, and the loads of a stage have one
// stage of MMA time to arrive (measured: tensor pipe 75 % busy).  In a pair each CTA stages its own 128 rows of
// A and its own 128 columns of B (64 KiB per k-block, three stages), the hardware feeds both halves of B to both
// SMs, and the leader's thread issues for both.  No TMA multicast: every CTA loads exactly the bytes it keeps,
// completion bytes counted on the leader's mbarrier.  Chunked accumulation as above; each CTA's eight epilogue
// warps keep the running sums of its own 128 x 256 half.
namespace pair {
constexpr int kPairM = 256;
constexpr int kCtaM = 128;
constexpr int kGroupM = 8;             // pair tiles per band
constexpr int kMaxStages = 4;

// BN: columns of a pair's tile, 256 or 128.  Half the width means twice the tiles, which fill the last wave better
// (the host picks, see gemm_tf32_tc_launch), at 4/3 of the operand traffic per product.
template <int BN>
struct Shape {
  static constexpr int kCtaN = BN / 2;                // columns of B staged by each CTA
  static constexpr int kStages = BN == 256 ? 3 : 4;
  static constexpr int kAPlane = kCtaM * kBK * 4;     // 16 KiB
  static constexpr int kBPlane = kCtaN * kBK * 4;     // 16 or 8 KiB
  static constexpr int kStageBytes = 2 * (kAPlane + kBPlane);  // A_hi, A_lo, B_hi, B_lo
};

struct alignas(8) Barriers {
  uint64_t full[kMaxStages];   // used in the leader: both CTAs' bytes of a stage have landed
  uint64_t empty[kMaxStages];  // in each CTA: the MMAs reading the stage have retired
  uint64_t acc_full[2];        // in each CTA: chunk accumulator complete
  uint64_t acc_empty[2];       // used in the leader: 16 epilogue warps of the pair have drained it
  uint32_t tmem_base;
  uint32_t abort_flag;
  Redo redo;
};
template <int BN>
constexpr int smem_bytes() {
  return Shape<BN>::kStages * Shape<BN>::kStageBytes + kStagingBytes + sizeof(Barriers) + 1024;
}
static_assert(smem_bytes<256>() <= 227 * 1024 && smem_bytes<128>() <= 227 * 1024, "shared memory budget of one CTA");

__device__ __forceinline__ void tile_coords(const Params& p, int tile, int& b, int& mb, int& nb) {
  const int per_batch = p.m_blocks * p.n_blocks;
  b = tile / per_batch;
  int t = tile - b * per_batch;
  const int band_tiles = kGroupM * p.n_blocks;
  const int band = t / band_tiles;
  const int first_m = band * kGroupM;
  const int rows_in_band = min(kGroupM, p.m_blocks - first_m);
  t -= band * band_tiles;
  mb = first_m + t % rows_in_band;
  nb = t / rows_in_band;
}

// A pair's work, in order: whole tiles pair_id, pair_id + pairs, ... below whole_tiles, then a share of K of one of the tiles left, which
// by themselves would occupy `splits` times fewer pairs.  (Dealing all their k-blocks out evenly gives a pair pieces of two tiles: the
// sums of the first have to leave before the second goes on, and that cost more than the even shares gave.)
struct Piece {
  int tile, kb0, kb1;
};
struct Walk {
  const Params& p;
  const int pair, pairs, num_kb;
  int next_tile;
  bool shared;
  __device__ __forceinline__ Walk(const Params& params, int pair_id, int num_pairs, int num_kb_)
      : p(params), pair(pair_id), pairs(num_pairs), num_kb(num_kb_), next_tile(pair_id),
        shared(pair_id < (params.batch * params.m_blocks * params.n_blocks - params.whole_tiles) * params.splits) {}
  __device__ __forceinline__ bool next(Piece& w) {
    if (next_tile < p.whole_tiles) {
      w = Piece{next_tile, 0, num_kb};
      next_tile += pairs;
      return true;
    }
    if (!shared) return false;
    shared = false;
    const int t = pair / p.splits, i = pair - t * p.splits, per = (num_kb + p.splits - 1) / p.splits;
    w = Piece{p.whole_tiles + t, i * per, min(num_kb, (i + 1) * per)};
    return true;
  }
};

__device__ __forceinline__ void tcgen05_mma_tf32_ss_pair(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc,
                                                         uint32_t accumulate) {
  asm volatile(
      "{\n"
      ".reg .pred p;\n"
      "setp.ne.b32 p, %4, 0;\n"
      "tcgen05.mma.cta_group::2.kind::tf32 [%0], %1, %2, %3, p;\n"
      "}\n" ::"r"(d_tmem),
      "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate)
      : "memory");
}

// m_blocks / n_blocks of Params count 256 x BN pair tiles here.
template <int BN, bool kRedo>
__global__ void __launch_bounds__(kThreads, 1)
gemm_tf32_tc2_kernel(const __grid_constant__ CUtensorMap tmap_a_hi, const __grid_constant__ CUtensorMap tmap_a_lo,
                     const __grid_constant__ CUtensorMap tmap_b_hi, const __grid_constant__ CUtensorMap tmap_b_lo,
                     float* __restrict__ c, const __grid_constant__ Params p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  using S = Shape<BN>;
  constexpr int kStages = S::kStages, kStageBytes = S::kStageBytes, kCtaN = S::kCtaN;
  constexpr int kAPlane = S::kAPlane, kBPlane = S::kBPlane;
  Barriers* bars = reinterpret_cast<Barriers*>(smem + kStages * kStageBytes + kStagingBytes);

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const uint32_t rank = ptx::cluster_ctarank();  // 0 = leader
  const int pair_id = blockIdx.x >> 1;
  const int num_pairs = gridDim.x >> 1;
  const int num_kb = (p.k + kBK - 1) / kBK;
  volatile uint32_t* abort_flag = &bars->abort_flag;

  if (threadIdx.x == 0) {
    for (int s = 0; s < kStages; ++s) {
      ptx::mbar_init(&bars->full[s], 1);
      ptx::mbar_init(&bars->empty[s], 1);
    }
    for (int a = 0; a < 2; ++a) {
      ptx::mbar_init(&bars->acc_full[a], 1);
      ptx::mbar_init(&bars->acc_empty[a], 16);  // 8 epilogue warps in each CTA of the pair
    }
    bars->abort_flag = 0;
    bars->redo.any = 0;
    ptx::fence_mbar_init();
  }
  if (warp == 1) {
    ptx::tmem_alloc_pair(&bars->tmem_base, kTmemCols);
    ptx::tmem_relinquish_alloc_permit_pair();
  }
  ptx::tcgen05_fence_before_thread_sync();
  ptx::cluster_sync_all();  // the peer's barriers are initialised before anything signals them
  ptx::tcgen05_fence_after_thread_sync();
  const uint32_t tmem_base = bars->tmem_base;
  ptx::launch_dependents();
  ptx::wait_prior_grid();

  if (warp == 0) {
    // ------------------------------ TMA producer (both CTAs) ------------------
    if (lane == 0) {
      ptx::prefetch_tensormap(&tmap_a_hi);
      ptx::prefetch_tensormap(&tmap_a_lo);
      ptx::prefetch_tensormap(&tmap_b_hi);
      ptx::prefetch_tensormap(&tmap_b_lo);
      int stage = 0;
      uint32_t phase = 0;
      bool ok = true;
      Walk walk(p, pair_id, num_pairs, num_kb);
      for (Piece w; ok && walk.next(w);) {
        int b, mb, nb;
        pair::tile_coords(p, w.tile, b, mb, nb);
        const int row0 = mb * kPairM + static_cast<int>(rank) * kCtaM;
        const int col0 = nb * BN + static_cast<int>(rank) * kCtaN;
        for (int kb = w.kb0; kb < w.kb1; ++kb) {
          if (!ptx::mbar_wait(&bars->empty[stage], phase ^ 1u, abort_flag, p.status, 45)) {
            ok = false;
            break;
          }
          const uint32_t full_leader = ptx::mapa_shared(ptx::smem_u32(&bars->full[stage]), 0);
          if (rank == 0) ptx::mbar_arrive_expect_tx(&bars->full[stage], 2 * kStageBytes);
          uint8_t* st = smem + stage * kStageBytes;
          ptx::tma_load_3d_pair(st, &tmap_a_hi, full_leader, kb * kBK, row0, b);
          ptx::tma_load_3d_pair(st + kAPlane, &tmap_a_lo, full_leader, kb * kBK, row0, b);
          ptx::tma_load_3d_pair(st + 2 * kAPlane, &tmap_b_hi, full_leader, kb * kBK, col0, b);
          ptx::tma_load_3d_pair(st + 2 * kAPlane + kBPlane, &tmap_b_lo, full_leader, kb * kBK, col0, b);
          if (++stage == kStages) {
            stage = 0;
            phase ^= 1u;
          }
        }
      }
    }
  } else if (warp == 1) {
    // ------------------------------ MMA issuer (leader CTA only) --------------
    if (lane == 0 && rank == 0) {
      constexpr uint32_t idesc = make_idesc_tf32(kPairM, BN);
      constexpr uint64_t kmajor = ptx::make_smem_desc_base(16, 1024);
      constexpr uint32_t kstep = kUmmaK * 4;
      int stage = 0;
      uint32_t phase = 0;
      bool ok = true;
      uint32_t chunk_count = 0;
      Walk walk(p, pair_id, num_pairs, num_kb);
      for (Piece w; ok && walk.next(w);) {
        for (int kb_begin = w.kb0; kb_begin < w.kb1 && ok; kb_begin += p.chunk_kb, ++chunk_count) {
          const uint32_t acc = chunk_count & 1u;
          const uint32_t acc_phase = (chunk_count >> 1) & 1u;
          if (!ptx::mbar_wait_relaxed(&bars->acc_empty[acc], acc_phase ^ 1u, abort_flag, p.status, 46)) {
            ok = false;
            break;
          }
          ptx::tcgen05_fence_after_thread_sync();
          const uint32_t d_tmem = tmem_base + acc * BN;
          const int kb_end = min(w.kb1, kb_begin + p.chunk_kb);
          for (int kb = kb_begin; kb < kb_end; ++kb) {
            if (!ptx::mbar_wait_relaxed(&bars->full[stage], phase, abort_flag, p.status, 47)) {
              ok = false;
              break;
            }
            ptx::tcgen05_fence_after_thread_sync();
            const uint32_t a_hi = ptx::smem_u32(smem + stage * kStageBytes);
            const uint32_t a_lo = a_hi + kAPlane, b_hi = a_lo + kAPlane, b_lo = b_hi + kBPlane;
            const bool first_kb = kb == kb_begin;
#pragma unroll
            for (int kk = 0; kk < kBK / kUmmaK; ++kk) {
              const uint32_t off = kk * kstep;
              tcgen05_mma_tf32_ss_pair(d_tmem, ptx::smem_desc(kmajor, a_lo + off), ptx::smem_desc(kmajor, b_hi + off), idesc,
                                       (first_kb && kk == 0) ? 0u : 1u);
              tcgen05_mma_tf32_ss_pair(d_tmem, ptx::smem_desc(kmajor, a_hi + off), ptx::smem_desc(kmajor, b_lo + off), idesc, 1u);
            }
#pragma unroll
            for (int kk = 0; kk < kBK / kUmmaK; ++kk)
              tcgen05_mma_tf32_ss_pair(d_tmem, ptx::smem_desc(kmajor, a_hi + kk * kstep), ptx::smem_desc(kmajor, b_hi + kk * kstep), idesc, 1u);
            ptx::tcgen05_commit_pair(&bars->empty[stage], 3);  // frees the stage in both CTAs
            if (++stage == kStages) {
              stage = 0;
              phase ^= 1u;
            }
          }
          if (ok) ptx::tcgen05_commit_pair(&bars->acc_full[acc], 3);
        }
      }
    }
  } else {
    // ------------------------------ chunk drain and output (both CTAs) ----------
    const int quad = warp & 3;
    const int half = (warp - 2) >> 2;
    constexpr int kChunks = BN / 64;      // 32-column blocks per warp
    const uint32_t lane_addr = tmem_base + (static_cast<uint32_t>(quad * 32) << 16) + half * (BN / 2);
    float* staging = reinterpret_cast<float*>(smem + kStages * kStageBytes) + (warp - 2) * kStagingFloats;
    uint32_t chunk_count = 0;
    bool alive = true;
    Walk walk(p, pair_id, num_pairs, num_kb);
    for (Piece w; walk.next(w);) {
      float sum[kChunks][32];
#pragma unroll
      for (int cc = 0; cc < kChunks; ++cc)
#pragma unroll
        for (int i = 0; i < 32; ++i) sum[cc][i] = 0.f;
      for (int kb = w.kb0; kb < w.kb1 && alive; kb += p.chunk_kb, ++chunk_count) {
        const uint32_t acc = chunk_count & 1u;
        const uint32_t acc_phase = (chunk_count >> 1) & 1u;
        const bool ready = ptx::mbar_wait(&bars->acc_full[acc], acc_phase, abort_flag, p.status, 48);
        if (!__all_sync(0xffffffffu, ready)) {
          alive = false;
          break;
        }
        ptx::tcgen05_fence_after_thread_sync();
#pragma unroll
        for (int cc = 0; cc < kChunks; ++cc) {
#pragma unroll
          for (int h = 0; h < 32; h += kDrain) {
            uint32_t v[kDrain];
            ptx::tmem_ld_32x32b_x16(lane_addr + acc * BN + cc * 32 + h, v);
            ptx::tmem_ld_wait();
#pragma unroll
            for (int i = 0; i < kDrain; ++i) sum[cc][h + i] += __uint_as_float(v[i]);
          }
        }
        ptx::tcgen05_fence_before_thread_sync();
        __syncwarp();
        if (lane == 0) ptx::mbar_arrive_cluster(ptx::mapa_shared(ptx::smem_u32(&bars->acc_empty[acc]), 0));
      }
      if (w.kb1 - w.kb0 != num_kb) {
        // every warp comes here, also one whose wait gave up: the barrier is for all eight
        if (epilogue_any(!alive)) {
          alive = false;
          continue;
        }
        const int tid = static_cast<int>(threadIdx.x) - 64;
        constexpr int kVecs = BN / 8;  // float4 per thread
        float4* mine = p.part + (static_cast<int64_t>(pair_id) * 2 + rank) * (kVecs * kEpilogueThreads) + tid;
#pragma unroll
        for (int cc = 0; cc < kChunks; ++cc)
#pragma unroll
          for (int i = 0; i < 8; ++i)
            __stcg(mine + (cc * 8 + i) * kEpilogueThreads, make_float4(sum[cc][4 * i], sum[cc][4 * i + 1], sum[cc][4 * i + 2], sum[cc][4 * i + 3]));
        __threadfence();
        epilogue_sync();
        const int first = (w.tile - p.whole_tiles) * p.splits;
        if (tid == 0) bars->redo.got = atomicAdd(&p.arrivals[2 * (w.tile - p.whole_tiles) + rank], 1u);
        epilogue_sync();
        if (bars->redo.got + 1u != static_cast<uint32_t>(p.splits)) continue;
        // the last one here adds all pieces, in order
        __threadfence();
#pragma unroll
        for (int cc = 0; cc < kChunks; ++cc)
#pragma unroll
          for (int i = 0; i < 32; ++i) sum[cc][i] = 0.f;
        for (int q = first; q < first + p.splits; ++q) {
          const float4* from = p.part + (static_cast<int64_t>(q) * 2 + rank) * (kVecs * kEpilogueThreads) + tid;
#pragma unroll
          for (int cc = 0; cc < kChunks; ++cc)
#pragma unroll
            for (int i = 0; i < 8; ++i) {
              const float4 x = __ldcg(from + (cc * 8 + i) * kEpilogueThreads);
              sum[cc][4 * i] += x.x, sum[cc][4 * i + 1] += x.y, sum[cc][4 * i + 2] += x.z, sum[cc][4 * i + 3] += x.w;
            }
        }
      }
      if (!alive) continue;
      int b, mb, nb;
      pair::tile_coords(p, w.tile, b, mb, nb);
      const int row0 = mb * kPairM + static_cast<int>(rank) * kCtaM + quad * 32;
#pragma unroll
      for (int cc = 0; cc < kChunks; ++cc)
        store_block_32x32<kRedo>(c, p, b, row0, nb * BN + half * (BN / 2) + cc * 32, sum[cc], staging, lane, &bars->redo);
    }
    if (kRedo) second_pass(p, c, reinterpret_cast<float*>(smem), &bars->redo, alive);
  }

  // ------------------------------ teardown ------------------------------------
  if (*abort_flag != 0u) {
    const unsigned long long t0 = ptx::globaltimer_ns();
    while (ptx::globaltimer_ns() - t0 < 1000000ull) {
    }
  }
  ptx::tcgen05_fence_before_thread_sync();
  // Neither CTA may leave while the other can still read its shared memory (the leader's MMAs) or signal its barriers.
  ptx::cluster_sync_all();
  if (warp == 1) {
    ptx::tcgen05_fence_after_thread_sync();
    ptx::tmem_dealloc_pair(tmem_base, kTmemCols);
  }
}
}  // namespace pair

}  // namespace gemm_tf32_tc
}  // namespace tsm100
