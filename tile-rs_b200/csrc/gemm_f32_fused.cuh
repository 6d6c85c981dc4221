// f32 GEMM on the tensor cores (tcgen05, kind::f16) for problems of few tiles, the operands split on the way in.
//
//   C[b][M,N] = A[b][M,K] * B[b], semantics as in gemm_tf32_tc.cuh (crates/tile_std/src/tile.rs:192-193, :2017-2031;
//   crates/rustc_codegen_tile/src/mlir_to_linalg.rs:1345-1393), accumulation in chunks as there.
//
// There a launch of its own writes hi / lo planes for TMA.  Here eight warps read the operands where they are, any alignment and
// either layout of B, split them in registers and store K-major, swizzled tiles: no second launch, no planes in memory, and no
// tensor maps to build.  Tiles are 128 x BN, BN = 64 or 128, and where they are fewer than the SMs a cluster of up to 8 CTAs splits K;
// the partial tiles are summed in rank order through distributed shared memory.
//
// A value is split into three bf16 numbers, hi + mid + lo, 24 bits together, so nothing of it is lost; of the nine products the six from
// 2^-16 on are taken (mid * lo and lo * mid, 2^-25 of the term and less and of either sign, and lo * lo are left out).  At twice the rate of
// TF32 that is the tensor-core time of three products of two TF32 numbers (which keep 22 bits) and the same traffic to feed them.
// What no bf16 number holds, bits below 2^-133 and infinities, is noticed: see redo_tile.
//
// Per CTA (one per SM): warps 8..15 load, split and store; warps 0..7 drain the accumulators, keep the sums in registers and write C; warp
// 0 also issues the products.  Bound, per 32 of K and 128 x 128 tile: shared memory, 768 cycles to feed the tensor core (which needs
// as many) and 384 for the stores of the split tiles.  Below 512^3 the fixed 4 to 5 us of a launch, its first loads and its last stores.
//
// As graph replays, warp-level kernel / two TF32 numbers (hi + lo, three products, chunks as below) / here: 512^3 11.9 / 9.3 / 9.4 us; FP32 pipe /
// TF32 / here: 1001 x 1003 x 1005 133 / 26.1 / 25.8, 301 x 301 x 2501 198 / 18.9 / 19.1, 600 x 2401 x 201 41 / 16.1 / 15.1, 3001 x 3003 x 101 86 /
// 36.1 / 32.5; 1024^3 24 us.
#pragma once

#include "attention_decode.cuh"  // cp.async helpers
#include "attention_tc.cuh"  // 16-bit pairs
#include "gemm_tf32_tc.cuh"
#include "ptx.cuh"

namespace tsm100 {
namespace gemm_f32_fused {

namespace tc = gemm_tf32_tc;

constexpr int kBM = 128;
constexpr int kBK = 32;                 // one 64-byte swizzle row of bf16
constexpr int kRow = kBK * 2;
constexpr int kUmmaK = 16;
constexpr int kDrainWarps = 8, kLoadWarps = 8;
constexpr int kThreads = (kDrainWarps + kLoadWarps) * 32;
constexpr int kMaxSplit = 8;
constexpr int kStages = 4;
constexpr int kAPlane = kBM * kRow;     // 8 KiB
enum : int { kOdd = 0, kLost = 1 };
constexpr int kRedoTiles = 256;         // tiles of one CTA that have bits of their own in Barriers
// An accumulator takes 256 of K of aligned rows and 128 of others, however long K is, and is then added to the sums in registers: it cuts
// every term off at its own last place, so the error grows with what it takes.  The products with mid and lo, 2^-8 of the others and less,
// have one to themselves, for 16 times as long.  Off the 64-bit result, normally distributed / all-positive data: 64 of K 0.9e-7 / 0.9e-7, 128
// 1.3e-7 / 1.8e-7, 256 2.4e-7 / 3.9e-7, all products in one accumulator of 128 7.9e-7 / 2.0e-6.  Beside it, for rows that start anywhere, the FP32
// pipe: 1.5e-7 / 1.2e-7 at K = 65, 3.3e-7 / 2.6e-7 at 333, 5.7e-7 / 4.9e-7 at 1005; for aligned ones the warp-level kernel: 9.2e-7 / 1.2e-6
// at K = 512, 7.2e-6 / 1.1e-5 at 1024.
constexpr int kChunkKb = 128 / kBK, kChunkKbAligned = 256 / kBK, kSmallChunks = 16;
// its bounded waits report sites 91 .. 94

template <int BN>
struct Shape {
  static constexpr int kBPlane = BN * kRow;
  static constexpr int kStageBytes = 3 * kAPlane + 3 * kBPlane;  // hi, mid and lo of A, then of B
  static constexpr int kStagingOff = kStages * kStageBytes;
  static constexpr int kBarsOff = kStagingOff + tc::kStagingBytes;
  static constexpr int kTmemCols = 4 * BN;  // two accumulators of hi * hi, two of the other products
};
struct alignas(8) Barriers {
  uint64_t full[kStages], empty[kStages];
  uint64_t acc_full[2], acc_empty[2];
  uint32_t tmem_base;
  uint32_t abort_flag;
  // a bit per tile, the last for all further ones: an output is infinite or NaN; an operand is not the sum of its parts
  uint32_t marks[2][kRedoTiles / 32];
};
template <int BN>
constexpr int smem_bytes() {
  return Shape<BN>::kBarsOff + static_cast<int>(sizeof(Barriers)) + 1024;
}
static_assert(Shape<64>::kStageBytes % 1024 == 0 && Shape<128>::kStageBytes % 1024 == 0 && Shape<64>::kBPlane % 512 == 0, "the swizzle repeats after 512 bytes");
static_assert(smem_bytes<64>() <= 227 * 1024 && smem_bytes<128>() <= 227 * 1024, "shared memory budget of one CTA");
struct Params {
  tc::Params g;             // m_blocks, n_blocks count 128 x BN tiles; a, b are the operands
  int32_t vec_a, vec_b;     // rows of A, and of B stored [N][K], start on 16-byte boundaries and K is a multiple of 4
  int32_t kb_per_cta;       // k-blocks per CTA of the cluster
};

// Four values of row `row` from k on, zeros outside [0, rows) x [0, k_end).
__device__ __forceinline__ void load4(float (&v)[4], const float* src, int64_t ld, int row, int rows, int k, int k_end, bool vec) {
  const float* p = src + row * ld + k;
  if (vec) {
    float4 x = make_float4(0.f, 0.f, 0.f, 0.f);
    if (row < rows && k < k_end) x = *reinterpret_cast<const float4*>(p);
    v[0] = x.x, v[1] = x.y, v[2] = x.z, v[3] = x.w;
  } else {
#pragma unroll
    for (int j = 0; j < 4; ++j) v[j] = row < rows && k + j < k_end ? p[j] : 0.f;
  }
}
// Two values as three pairs of bf16 numbers: hi truncated (the largest f32 numbers would round up to infinity), mid rounded to nearest
// (so that what the products leave out has either sign), lo the rest.  All differences are exact, and lo has 8 bits; in the lower half of
// the f32 number that it is cut from something stands only if it falls below 2^-133, or for infinities and NaNs: `lost` collects that.
__device__ __forceinline__ void split2(float x0, float x1, uint32_t& hi, uint32_t& mid, uint32_t& lo, uint32_t& lost) {
  const uint32_t b0 = __float_as_uint(x0), b1 = __float_as_uint(x1);
  hi = __byte_perm(b0, b1, 0x7632);
  const float r0 = x0 - __uint_as_float(b0 & 0xffff0000u), r1 = x1 - __uint_as_float(b1 & 0xffff0000u);
  mid = attn::pack16x2<true>(r0, r1);
  const uint32_t l0 = __float_as_uint(r0 - attn::unpack16_lo<true>(mid)), l1 = __float_as_uint(r1 - attn::unpack16_hi<true>(mid));
  lo = __byte_perm(l0, l1, 0x7632);
  lost |= l0 | l1;
}
// Four values of a row -> 8 bytes of each plane, `plane` bytes apart.
__device__ __forceinline__ void split_store4(uint32_t at, uint32_t plane, const float (&v)[4], uint32_t& lost) {
  uint32_t hi[2], mid[2], lo[2];
#pragma unroll
  for (int j = 0; j < 2; ++j) split2(v[2 * j], v[2 * j + 1], hi[j], mid[j], lo[j], lost);
  ptx::st_shared_v2(at, hi[0], hi[1]);
  ptx::st_shared_v2(at + plane, mid[0], mid[1]);
  ptx::st_shared_v2(at + 2 * plane, lo[0], lo[1]);
}
__device__ __forceinline__ void split_store8(uint32_t at, uint32_t plane, const float (&v)[8], uint32_t& lost) {
  uint32_t hi[4], mid[4], lo[4];
#pragma unroll
  for (int j = 0; j < 4; ++j) split2(v[2 * j], v[2 * j + 1], hi[j], mid[j], lo[j], lost);
  ptx::st_shared_v4(at, hi[0], hi[1], hi[2], hi[3]);
  ptx::st_shared_v4(at + plane, mid[0], mid[1], mid[2], mid[3]);
  ptx::st_shared_v4(at + 2 * plane, lo[0], lo[1], lo[2], lo[3]);
}
// The largest finite magnitude among rows [row0, row_end) x columns [col0, col_end) of `src`, over all 256 threads; `red`: 8 floats.
__device__ __forceinline__ float largest(const float* src, int64_t ld, int row0, int row_end, int col0, int col_end, float* red, int tid) {
  float most = 0.f;
  for (int i = col0 + (tid & 31); i < col_end; i += 32)
#pragma unroll 8
    for (int r = row0 + (tid >> 5); r < row_end; r += 8) {
      const float v = fabsf(src[r * ld + i]);
      if (v < INFINITY) most = fmaxf(most, v);
    }
  for (int off = 16; off > 0; off >>= 1) most = fmaxf(most, __shfl_xor_sync(0xffffffffu, most, off));
  tc::epilogue_sync();
  if ((tid & 31) == 0) red[tid >> 5] = most;
  tc::epilogue_sync();
  for (int i = 0; i < 8; ++i) most = fmaxf(most, red[i]);
  return most;
}
// The outputs of rows [row_begin, row_end) of a tile that the parts of the operands do not give are summed again in plain f32, in the
// order of k.  Infinities and NaNs always (an infinity split into parts is infinity + NaN).  Where an operand's parts miss bits (`lost`), which
// are below 2^-133, outputs beside which K times those bits and the largest operand are more than 2^-25; all, if there are infinities or NaNs too
// (`odd`).  256 threads, 64 x 64 outputs at a time, 4 x 4 each (with what more registers take, the whole kernel spills), the next 32 of k copied
// meanwhile.  1001 x 1003 x 1005, 29 us, with one infinity 235 us, all outputs infinite 437, a hundredth of A
// 1e-36 102 (FP32 pipe 137).
constexpr int kPanelK = 32, kPanelPitch = 68, kPanelBytes = 2 * kPanelK * kPanelPitch * 4;
static_assert(2 * kPanelBytes <= kStages * Shape<64>::kStageBytes, "two panels of both operands take the place of the stages");
template <int BN>
__device__ __noinline__ void redo_tile(const Params& p, float* c, float* panels, int tile, int row_begin, int row_end, bool lost, bool odd, int tid) {
  const tc::Params& g = p.g;
  int bz, mb, nb;
  tc::tile_coords(g, tile, bz, mb, nb);
  row_begin += mb * kBM, row_end = min(row_end + mb * kBM, g.m);
  const bool bt = g.b_transposed != 0;
  float least = lost ? INFINITY : 0.f;
  if (lost && !odd) {
    const float* a = g.a + bz * g.a_batch_stride;
    const float* b = g.b + bz * g.b_batch_stride;
    const int col0 = nb * BN, col_end = min(col0 + BN, g.n);
    const float most_a = largest(a, g.lda, row_begin, row_end, 0, g.k, panels, tid);
    const float most_b = bt ? largest(b, g.ldb, col0, col_end, 0, g.k, panels, tid) : largest(b, g.ldb, 0, g.k, col0, col_end, panels, tid);
    least = static_cast<float>(g.k) * 0x1p-108f * (most_a + most_b);
  }
  const int tx = tid & 15, ty = tid >> 4;
  // this thread's eight values of a panel of A: k = tid & 31, rows (tid >> 5) + 8 i; of B the same, or, stored [K][N], column tid & 63, k = (tid >>
  // 6) + 4 i
  const int ak = tid & 31, ar = tid >> 5, bk = bt ? ak : tid >> 6, bn = bt ? ar : tid & 63, bk_step = bt ? 0 : 4, bn_step = bt ? 8 : 0;
  for (int block = 0; block < 2 * (BN / 64); ++block) {
    const int row0 = mb * kBM + (block & 1) * 64, col0 = nb * BN + (block >> 1) * 64;
    if (row0 >= row_end || row0 + 64 <= row_begin || col0 >= g.n) continue;
    float* out = c + bz * g.c_batch_stride + (row0 + ty * 4) * g.ldc + col0 + tx * 4;
    uint32_t again = 0;
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int row = row0 + ty * 4 + i;
        if (row < row_begin || row >= row_end || col0 + tx * 4 + j >= g.n) continue;
        const float v = fabsf(__ldcg(out + i * g.ldc + j));
        if (!(v < INFINITY) || v < least) again |= 1u << (i * 4 + j);
      }
    if (!tc::epilogue_any(again != 0u)) continue;
    const float* a = g.a + bz * g.a_batch_stride + (row0 + ar) * g.lda + ak;
    const float* b = g.b + bz * g.b_batch_stride + (bt ? (col0 + bn) * g.ldb + bk : bk * g.ldb + col0 + bn);
    const int64_t b_step = (bt ? 8 : 4) * g.ldb;
    auto copy = [&](int k0, uint32_t to) {
#pragma unroll 1
      for (int i = 0; i < 8; ++i) {
        const bool in_a = row0 + ar + 8 * i < g.m && k0 + ak < g.k, in_b = col0 + bn + i * bn_step < g.n && k0 + bk + i * bk_step < g.k;
        ptx::cp_async_4(to + (ak * kPanelPitch + ar + 8 * i) * 4, in_a ? a + i * 8 * g.lda : g.a, in_a);
        ptx::cp_async_4(to + kPanelBytes / 2 + ((bk + i * bk_step) * kPanelPitch + bn + i * bn_step) * 4, in_b ? b + i * b_step : g.b, in_b);
      }
      a += kPanelK;
      b += bt ? kPanelK : kPanelK * g.ldb;
      attn_decode::mma::cp_async_commit();
    };
    float acc[4][4] = {};
    uint32_t second = 0;
    copy(0, ptx::smem_u32(panels));
    for (int k0 = 0; k0 < g.k; k0 += kPanelK, second ^= 1u) {
      copy(k0 + kPanelK, ptx::smem_u32(panels) + (second ^ 1u) * kPanelBytes);
      attn_decode::mma::cp_async_wait<1>();
      tc::epilogue_sync();
      const float* sa = panels + second * (kPanelBytes / 4) + ty * 4;
      const float* sb = panels + second * (kPanelBytes / 4) + kPanelBytes / 8 + tx * 4;
#pragma unroll 2
      for (int kk = 0; kk < kPanelK; ++kk, sa += kPanelPitch, sb += kPanelPitch) {
        const float4 x = *reinterpret_cast<const float4*>(sa);
        const float4 w = *reinterpret_cast<const float4*>(sb);
        const float xs[4] = {x.x, x.y, x.z, x.w}, ws[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
          for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(xs[i], ws[j], acc[i][j]);
      }
      tc::epilogue_sync();
    }
    attn_decode::mma::cp_async_wait<0>();
    tc::epilogue_sync();
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j)
        if ((again >> (i * 4 + j)) & 1u) out[i * g.ldc + j] = acc[i][j];
  }
}

// grid: a persistent CTA per SM over all tiles, or, in clusters, one tile per cluster.
// kShortK: the stages hold all of a CTA's K at once (kStages k-blocks at most).  The products with mid and lo come first then, before there
// is anything large beside which they would be cut off, and one accumulator does.
template <int BN, bool kBTransposed, bool kShortK>
__global__ void __launch_bounds__(kThreads, 1)
gemm_f32_fused_kernel(float* __restrict__ c, const __grid_constant__ Params p) {
  using S = Shape<BN>;
  constexpr int kCols = BN / 2;  // columns per drain warp
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  Barriers* bars = reinterpret_cast<Barriers*>(smem + S::kBarsOff);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  volatile uint32_t* abort_flag = &bars->abort_flag;
  const tc::Params& g = p.g;

  const int splits = static_cast<int>(ptx::cluster_nctarank()), rank = static_cast<int>(ptx::cluster_ctarank());
  const int num_tiles = g.batch * g.m_blocks * g.n_blocks;
  const int first_tile = static_cast<int>(blockIdx.x) / splits, tile_step = static_cast<int>(gridDim.x) / splits;
  const int kb_all = (g.k + kBK - 1) / kBK;
  const int kb0 = rank * p.kb_per_cta;
  const int num_kb = min(kb_all - kb0, p.kb_per_cta);
  const int num_chunks = (num_kb + g.chunk_kb - 1) / g.chunk_kb;

  if (threadIdx.x == 0) {
    for (int s = 0; s < kStages; ++s) {
      ptx::mbar_init(&bars->full[s], kLoadWarps);
      ptx::mbar_init(&bars->empty[s], 1);
    }
    for (int a = 0; a < 2; ++a) {
      ptx::mbar_init(&bars->acc_full[a], 1);
      ptx::mbar_init(&bars->acc_empty[a], kDrainWarps);
    }
    bars->abort_flag = 0;
    ptx::fence_mbar_init();
  }
  if (threadIdx.x < kRedoTiles / 32) bars->marks[kOdd][threadIdx.x] = bars->marks[kLost][threadIdx.x] = 0;
  if (warp == 0) {
    ptx::tmem_alloc(&bars->tmem_base, S::kTmemCols);
    ptx::tmem_relinquish_alloc_permit();
  }
  ptx::tcgen05_fence_before_thread_sync();
  __syncthreads();
  ptx::tcgen05_fence_after_thread_sync();
  const uint32_t tmem_base = bars->tmem_base;
  ptx::wait_prior_grid();

  if (warp >= kDrainWarps) {
    // ------------------------------ load, split, store --------------------------
    const int t = static_cast<int>(threadIdx.x) - kDrainWarps * 32;
    const float* a_all = ptx::wait_prior_grid(g.a);
    const float* b_all = ptx::wait_prior_grid(g.b);
    // The swizzle: 16-byte unit u of row r of a plane lies at unit u ^ ((r >> 1) & 3).
    // A (and B stored [N][K]): values 4 u to 4 u + 3 of rows r, r + 32, ...; eight lanes read 128 bytes of a row
    const int r = t >> 3, u = t & 7;
    const uint32_t at = r * kRow + (((u >> 1) ^ ((r >> 1) & 3)) << 4) + (u & 1) * 8;
    // B stored [K][N]: column n, units g0, g0 + kGroups, ... of eight values; a warp reads 128 bytes of a row of K
    constexpr int kGroups = kLoadWarps * 32 / BN, kBRows = BN / 32, kBUnits = BN / 64;
    const int n = t % BN, g0 = t / BN;
    struct Regs {
      float a[4][4];
      float b[kBTransposed ? kBRows : kBUnits][kBTransposed ? 4 : 8];
    };
    // the next k-block to load: two are in registers, across tiles
    int lt = first_tile, lk = 0, row0 = 0, col0 = 0;
    const float *a = a_all, *b = b_all;
    auto load = [&](Regs& x) -> bool {
      if (lt >= num_tiles) return false;
      if (lk == 0) {
        int bz, mb, nb;
        tc::tile_coords(g, lt, bz, mb, nb);
        row0 = mb * kBM, col0 = nb * BN;
        a = a_all + bz * g.a_batch_stride;
        b = b_all + bz * g.b_batch_stride;
      }
      const int k = (kb0 + lk) * kBK;
#pragma unroll
      for (int i = 0; i < 4; ++i) load4(x.a[i], a, g.lda, row0 + r + 32 * i, g.m, k + u * 4, g.k, p.vec_a != 0);
      if constexpr (kBTransposed) {
#pragma unroll
        for (int i = 0; i < kBRows; ++i) load4(x.b[i], b, g.ldb, col0 + r + 32 * i, g.n, k + u * 4, g.k, p.vec_b != 0);
      } else {
        const int col = col0 + n;
#pragma unroll
        for (int i = 0; i < kBUnits; ++i) {
          const int k8 = k + (g0 + i * kGroups) * 8;
          const float* q = b + k8 * g.ldb + col;
#pragma unroll
          for (int j = 0; j < 8; ++j) x.b[i][j] = col < g.n && k8 + j < g.k ? q[j * g.ldb] : 0.f;
        }
      }
      if (++lk == num_kb) lk = 0, lt += tile_step;
      return true;
    };
    int stage = 0, seq = 0, sk = 0;
    uint32_t phase = 0, lost = 0;
    auto store = [&](const Regs& x) -> bool {
      if (!__all_sync(0xffffffffu, ptx::mbar_wait(&bars->empty[stage], phase ^ 1u, abort_flag, g.status, 91))) return false;
      const uint32_t base = ptx::smem_u32(smem + stage * S::kStageBytes);
#pragma unroll
      for (int i = 0; i < 4; ++i) split_store4(base + at + i * 32 * kRow, kAPlane, x.a[i], lost);
      const uint32_t bb = base + 3 * kAPlane;
      if constexpr (kBTransposed) {
#pragma unroll
        for (int i = 0; i < kBRows; ++i) split_store4(bb + at + i * 32 * kRow, S::kBPlane, x.b[i], lost);
      } else {
#pragma unroll
        for (int i = 0; i < kBUnits; ++i) split_store8(bb + n * kRow + (((g0 + i * kGroups) ^ ((n >> 1) & 3)) << 4), S::kBPlane, x.b[i], lost);
      }
      if (++sk == num_kb) {  // the tile's last
        const int bit = min(seq, kRedoTiles - 1);
        if (__any_sync(0xffffffffu, (lost & 0xffffu) != 0u) && lane == 0) atomicOr(&bars->marks[kLost][bit >> 5], 1u << (bit & 31));
        sk = 0, lost = 0, ++seq;
      }
      ptx::fence_proxy_async_smem();  // the tensor core reads the tiles through the async proxy
      __syncwarp();
      if (lane == 0) ptx::mbar_arrive(&bars->full[stage]);
      if (++stage == kStages) stage = 0, phase ^= 1u;
      return true;
    };
    Regs x0, x1;
    bool have0 = load(x0), have1 = load(x1);
    while (have0) {
      if (!store(x0)) break;
      have0 = load(x0);
      if (!have1 || !store(x1)) break;
      have1 = load(x1);
    }
    __syncwarp();
    ptx::launch_dependents();
  } else {
    // ------------------------------ chunk drain and output ----------------------
    const int quad = warp & 3, half = warp >> 2;  // TMEM lanes, and which half of the columns
    const uint32_t lane_addr = tmem_base + (static_cast<uint32_t>(quad * 32) << 16) + half * kCols;
    float* staging = reinterpret_cast<float*>(smem + S::kStagingOff) + warp * tc::kStagingFloats;
    // The products, issued by warp 0 a chunk ahead of the drain: two accumulators, and the tensor core has the next chunk queued
    // while all warps drain this one.
    constexpr uint32_t idesc = ptx::make_idesc_f16(kBM, BN, false, false, true);
    constexpr uint64_t kmajor = ptx::make_smem_desc_base(16, 8 * kRow, ptx::kSwizzle64B);
    constexpr uint32_t hi32 = static_cast<uint32_t>(kmajor >> 32), lo32 = static_cast<uint32_t>(kmajor);
    auto desc = [](uint32_t lo) -> uint64_t { return (static_cast<uint64_t>(hi32) << 32) | lo; };
    const uint32_t smem_lo = lo32 | (ptx::smem_u32(smem) >> 4);
    int stage = 0, next_tile = first_tile, next_chunk = 0;
    uint32_t phase = 0, issued = 0, groups = 0;
    auto issue_chunk = [&]() -> bool {
      if (next_tile >= num_tiles) return true;
      const uint32_t acc = issued & 1u;
      if (!__all_sync(0xffffffffu, ptx::mbar_wait_relaxed(&bars->acc_empty[acc], ((issued >> 1) & 1u) ^ 1u, abort_flag, g.status, 92))) return false;
      if (next_chunk % kSmallChunks == 0) ++groups;
      const uint32_t large = tmem_base + acc * BN, small = kShortK ? large : tmem_base + (2 + (groups & 1u)) * BN;
      const int kb_begin = next_chunk * g.chunk_kb, kb_end = min(num_kb, kb_begin + g.chunk_kb);
      auto products = [&](uint32_t d, uint32_t x, uint32_t w, bool first) {
#pragma unroll
        for (int kk = 0; kk < kBK / kUmmaK; ++kk)
          ptx::tcgen05_mma_f16_ss(d, desc(x + kk * (kUmmaK * 2 >> 4)), desc(w + kk * (kUmmaK * 2 >> 4)), idesc, first && kk == 0 ? 0u : 1u);
      };
      auto small_products = [&](uint32_t a, bool first) {  // `a`: where the stage's hi part of A lies
        const uint32_t b = a + (3 * kAPlane >> 4);
        products(small, a + (2 * kAPlane >> 4), b, first);
        products(small, a, b + (2 * S::kBPlane >> 4), false);
        products(small, a + (kAPlane >> 4), b + (S::kBPlane >> 4), false);
        products(small, a + (kAPlane >> 4), b, false);
        products(small, a, b + (S::kBPlane >> 4), false);
      };
      int late = stage;  // kShortK: the stage that the large products are at
      for (int kb = kb_begin; kb < kb_end; ++kb) {
        if (!__all_sync(0xffffffffu, ptx::mbar_wait(&bars->full[stage], phase, abort_flag, g.status, 93))) return false;
        ptx::tcgen05_fence_after_thread_sync();
        if (ptx::elect_one_sync()) {
          const uint32_t a = smem_lo + stage * (S::kStageBytes >> 4);
          small_products(a, kb == kb_begin && next_chunk % kSmallChunks == 0);
          if (!kShortK) {
            products(large, a, a + (3 * kAPlane >> 4), kb == kb_begin);
            ptx::tcgen05_commit(&bars->empty[stage]);
            if (kb == kb_end - 1) ptx::tcgen05_commit(&bars->acc_full[acc]);
          }
        }
        __syncwarp();
        if (++stage == kStages) stage = 0, phase ^= 1u;
      }
      if (kShortK) {
        for (int kb = 0; kb < num_kb; ++kb) {
          if (ptx::elect_one_sync()) {
            const uint32_t a = smem_lo + late * (S::kStageBytes >> 4);
            products(large, a, a + (3 * kAPlane >> 4), false);
            ptx::tcgen05_commit(&bars->empty[late]);
            if (kb == num_kb - 1) ptx::tcgen05_commit(&bars->acc_full[acc]);
          }
          __syncwarp();
          if (++late == kStages) late = 0;
        }
      }
      ++issued;
      if (++next_chunk == num_chunks) next_chunk = 0, next_tile += tile_step;
      return true;
    };
    uint32_t chunk_count = 0, group_count = 0;
    bool alive = warp != 0 || issue_chunk();
    int seq = 0;
    for (int tile = first_tile; tile < num_tiles; tile += tile_step, ++seq) {
      float sum[kCols / 32][32];
#pragma unroll
      for (int cc = 0; cc < kCols / 32; ++cc)
#pragma unroll
        for (int i = 0; i < 32; ++i) sum[cc][i] = 0.f;
      for (int ch = 0; ch < (kShortK ? 1 : num_chunks); ++ch, ++chunk_count) {
        const uint32_t acc = chunk_count & 1u;
        if (warp == 0) alive = alive && issue_chunk();
        if (!alive) break;
        if (!__all_sync(0xffffffffu, ptx::mbar_wait(&bars->acc_full[acc], (chunk_count >> 1) & 1u, abort_flag, g.status, 94))) {
          alive = false;
          break;
        }
        ptx::tcgen05_fence_after_thread_sync();
        auto drain = [&](uint32_t from) {
#pragma unroll
          for (int cc = 0; cc < kCols / 32; ++cc) {
            uint32_t v[32];
            ptx::tmem_ld_32x32b_x32(lane_addr + from + cc * 32, v);
            ptx::tmem_ld_wait();
#pragma unroll
            for (int i = 0; i < 32; ++i) sum[cc][i] = kShortK ? __uint_as_float(v[i]) : sum[cc][i] + __uint_as_float(v[i]);
          }
        };
        drain(acc * BN);
        if (ch % kSmallChunks == 0) ++group_count;
        if (!kShortK && (ch % kSmallChunks == kSmallChunks - 1 || ch == num_chunks - 1)) drain((2 + (group_count & 1u)) * BN);
        ptx::tcgen05_fence_before_thread_sync();
        __syncwarp();
        if (lane == 0) ptx::mbar_arrive(&bars->acc_empty[acc]);
      }
      if (!alive) break;
      if (splits > 1) {
        // the partial tile takes the place of the stages (the last accumulator is complete: every product has retired), 16-byte unit
        // q of row r at q ^ (r & 7)
        const int row = quad * 32 + lane;
        const uint32_t part = ptx::smem_u32(smem) + row * (BN * 4);
#pragma unroll
        for (int cc = 0; cc < kCols / 32; ++cc)
#pragma unroll
          for (int i = 0; i < 8; ++i)
            ptx::st_shared_v4(part + (((half * kCols / 4 + cc * 8 + i) ^ (row & 7)) << 4), __float_as_uint(sum[cc][4 * i]),
                              __float_as_uint(sum[cc][4 * i + 1]), __float_as_uint(sum[cc][4 * i + 2]), __float_as_uint(sum[cc][4 * i + 3]));
      } else {
        int b, mb, nb;
        tc::tile_coords(g, tile, b, mb, nb);
        float z4[4] = {};  // NaN where anything is infinite or NaN (rows and columns past C are so only beside such ones of C)
#pragma unroll
        for (int cc = 0; cc < kCols / 32; ++cc)
#pragma unroll
          for (int i = 0; i < 32; ++i) z4[i & 3] = fmaf(sum[cc][i], 0.f, z4[i & 3]);
        const float z = (z4[0] + z4[1]) + (z4[2] + z4[3]);
        const int bit = min(seq, kRedoTiles - 1);
        if (__any_sync(0xffffffffu, z != 0.f) && lane == 0) atomicOr(&bars->marks[kOdd][bit >> 5], 1u << (bit & 31));
#pragma unroll
        for (int cc = 0; cc < kCols / 32; ++cc)
          tc::store_block_32x32<false>(c, g, b, mb * kBM + quad * 32, nb * BN + half * kCols + cc * 32, sum[cc], staging, lane, nullptr);
      }
    }
    if (splits == 1 && !tc::epilogue_any(!alive)) {
      if (tc::epilogue_any(threadIdx.x < kRedoTiles / 32 && (bars->marks[kOdd][threadIdx.x] | bars->marks[kLost][threadIdx.x]) != 0u)) {
        seq = 0;
        for (int tile = first_tile; tile < num_tiles; tile += tile_step, ++seq) {
          const int bit = min(seq, kRedoTiles - 1);
          const bool lost = (bars->marks[kLost][bit >> 5] >> (bit & 31)) & 1u, odd = (bars->marks[kOdd][bit >> 5] >> (bit & 31)) & 1u;
          if (lost || odd) redo_tile<BN>(p, c, reinterpret_cast<float*>(smem), tile, 0, kBM, lost, odd, threadIdx.x);
        }
      }
    }
  }

  if (splits > 1) {
    ptx::cluster_sync_all();
    // every CTA adds its share of the rows, in rank order
    int b, mb, nb;
    tc::tile_coords(g, first_tile, b, mb, nb);
    const int rows = min(kBM, g.m - mb * kBM);
    const uint32_t part = ptx::smem_u32(smem);
    float* cb = c + b * g.c_batch_stride;
    const int per = (rows + splits - 1) / splits, row_end = min(rows, (rank + 1) * per);
    bool odd = false;
    // an operand's missing bits in one share of K concern all rows
    if (static_cast<int>(threadIdx.x) < splits && bars->marks[kLost][0] != 0u)
      ptx::st_shared_cluster_u32(ptx::mapa_shared(ptx::smem_u32(&bars->marks[kLost][0]), threadIdx.x), 1u);
    if (*abort_flag == 0u) {
      for (int i = rank * per * (BN / 4) + static_cast<int>(threadIdx.x); i < row_end * (BN / 4); i += kThreads) {
        const int row = i / (BN / 4), q = i % (BN / 4);
        const uint32_t at = part + row * (BN * 4) + ((q ^ (row & 7)) << 4);
        float4 v[kMaxSplit];
#pragma unroll
        for (int s = 0; s < kMaxSplit; ++s)
          if (s < splits) v[s] = ptx::ld_shared_cluster_f32x4(ptx::mapa_shared(at, s));
        float4 x = v[0];
#pragma unroll
        for (int s = 1; s < kMaxSplit; ++s)
          if (s < splits) x.x += v[s].x, x.y += v[s].y, x.z += v[s].z, x.w += v[s].w;
        const int col = nb * BN + q * 4;
        float* dst = cb + static_cast<int64_t>(mb * kBM + row) * g.ldc + col;
        if (g.vec_store && col + 4 <= g.n) {
          *reinterpret_cast<float4*>(dst) = x;
        } else {
          if (col < g.n) dst[0] = x.x;
          if (col + 1 < g.n) dst[1] = x.y;
          if (col + 2 < g.n) dst[2] = x.z;
          if (col + 3 < g.n) dst[3] = x.w;
        }
        odd |= !(fabsf(x.x) < INFINITY && fabsf(x.y) < INFINITY && fabsf(x.z) < INFINITY && fabsf(x.w) < INFINITY);
      }
    }
    if (odd) bars->marks[kOdd][0] = 1u;
    ptx::cluster_sync_all();  // nobody's partial tile goes while a peer reads it; all of the tile is in memory
    const bool lost = bars->marks[kLost][0] != 0u, any_odd = bars->marks[kOdd][0] != 0u;
    if ((lost || any_odd) && *abort_flag == 0u && threadIdx.x < 256)
      redo_tile<BN>(p, c, reinterpret_cast<float*>(smem), first_tile, rank * per, row_end, lost, any_odd, threadIdx.x);
  }

  // ------------------------------ teardown ------------------------------------
  if (*abort_flag != 0u) {
    const unsigned long long t0 = ptx::globaltimer_ns();
    while (ptx::globaltimer_ns() - t0 < 1000000ull) {
    }
  }
  ptx::tcgen05_fence_before_thread_sync();
  __syncthreads();
  if (warp == 0) {
    ptx::tcgen05_fence_after_thread_sync();
    ptx::tmem_dealloc(tmem_base, S::kTmemCols);
  }
}

}  // namespace gemm_f32_fused
}  // namespace tsm100
