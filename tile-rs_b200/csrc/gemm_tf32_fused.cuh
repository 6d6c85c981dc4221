// f32 GEMM on the tensor cores (tcgen05, kind::tf32) for problems of few tiles, the operands split on the way in.
//
//   C[b][M,N] = A[b][M,K] * B[b], semantics, the three TF32 products per product and the accumulation in chunks as in
//   gemm_tf32_tc.cuh (crates/tile_std/src/tile.rs:192-193, :2017-2031; crates/rustc_codegen_tile/src/mlir_to_linalg.rs:1345-1393).
//
// There a launch of its own writes hi / lo planes for TMA.  Here eight warps read the operands where they are, any alignment and
// either layout of B, split them in registers and store K-major, swizzled tiles: no second launch, no planes in memory, and no
// tensor maps to build.  Tiles are 128 x BN, BN = 64 or 128, and where they are fewer than the SMs a cluster of up to 8 CTAs splits K;
// the partial tiles are summed in rank order through distributed shared memory.
//
// 512^3 12.9 us on the warp-level kernel, 9.1 here (as graph replays); 1024^3 51 / 23; rows that start anywhere, FP32 pipe / here:
// 1001 x 1003 x 1005 133 / 25, 301 x 301 x 2501 199 / 15, 601 x 2401 x 201 40 / 16.  Error against 64 bits 8.2e-7 of the result in
// chunks of 128, whatever K is (warp level 9.1e-7 at K = 512, 7.2e-6 at 1024, 1.4e-4 at 20000), 3.7e-7 and 1.4e-7 in chunks of 64 and 32 (FP32 pipe 5.7e-7 at 1005).
//
// Per CTA (one per SM): warps 8..15 load, split and store; warps 0..7 drain the chunks, keep the sums in registers and write C; warp
// 0 also issues the products.  Bound, per 32 of K and 128 x 128 tile: shared memory, 768 cycles to feed the tensor core (which needs
// as many) and 512 for the stores of the split tiles; measured 1900 (0.63 us of products and 0.55 of splitting, each alone, take 1.0
// together, loads from the L2 included).  Below 512^3 the fixed 4 to 5 us of a launch, its first loads and its last stores.
#pragma once

#include "gemm_tf32_tc.cuh"
#include "ptx.cuh"

namespace tsm100 {
namespace gemm_tf32_fused {

namespace tc = gemm_tf32_tc;

constexpr int kBM = 128;
constexpr int kBK = 32;                 // one 128-byte swizzle row of f32
constexpr int kDrainWarps = 8, kLoadWarps = 8;
constexpr int kThreads = (kDrainWarps + kLoadWarps) * 32;
constexpr int kMaxSplit = 8;
constexpr int kMaxStages = 4;
constexpr int kAPlane = kBM * kBK * 4;  // 16 KiB
constexpr int kRedoTiles = 256;         // tiles of one CTA that a bit of their own says hold an infinity or a NaN
// its bounded waits report sites 91 .. 94

template <int BN>
struct Shape {
  static constexpr int kBPlane = BN * kBK * 4;
  static constexpr int kStageBytes = 2 * kAPlane + 2 * kBPlane;  // A_hi, A_lo, B_hi, B_lo
  static constexpr int kStages = BN == 64 ? 4 : 3;
  static constexpr int kStagingOff = kStages * kStageBytes;
  static constexpr int kBarsOff = kStagingOff + tc::kStagingBytes;
  static constexpr int kTmemCols = 2 * BN;
};
struct alignas(8) Barriers {
  uint64_t full[kMaxStages], empty[kMaxStages];
  uint64_t acc_full[2], acc_empty[2];
  uint32_t tmem_base;
  uint32_t abort_flag;
  uint32_t redo[kRedoTiles / 32];
};
template <int BN>
constexpr int smem_bytes() {
  return Shape<BN>::kBarsOff + static_cast<int>(sizeof(Barriers)) + 1024;
}
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
// hi = x rounded to TF32, lo = x - hi (exact) rounded again, without the conversion instruction (two of them for every value made 1.2 us
// per 32 of K and 128 x 128 tile, 1.04 this way).  A NaN stays one in hi.
__device__ __forceinline__ void split_store(uint32_t hi, uint32_t lo, const float (&v)[4]) {
  float h[4], l[4];
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    h[j] = tc::tf32_rn_fast(v[j]);
    l[j] = tc::tf32_rn_finite(v[j] - h[j]);
  }
  ptx::st_shared_v4(hi, __float_as_uint(h[0]), __float_as_uint(h[1]), __float_as_uint(h[2]), __float_as_uint(h[3]));
  ptx::st_shared_v4(lo, __float_as_uint(l[0]), __float_as_uint(l[1]), __float_as_uint(l[2]), __float_as_uint(l[3]));
}
// A tile that came out infinite or NaN somewhere: those outputs are summed again in plain f32, in the order of k (an infinity split
// into hi + lo is infinity + NaN, and a hi part can round up to infinity).  256 threads, 64 x 64 outputs at a time, 4 x 4 each.
constexpr int kPanelK = 16, kPanelPitch = 68;
template <int BN>
__device__ __noinline__ void redo_tile(const Params& p, float* c, float* panels, int tile, int tid) {
  const tc::Params& g = p.g;
  int bz, mb, nb;
  tc::tile_coords(g, tile, bz, mb, nb);
  const float* a = g.a + bz * g.a_batch_stride;
  const float* b = g.b + bz * g.b_batch_stride;
  float *sa = panels, *sb = panels + kPanelK * kPanelPitch;
  const int tx = tid & 15, ty = tid >> 4;
  for (int block = 0; block < 2 * (BN / 64); ++block) {
    const int row0 = mb * kBM + (block & 1) * 64, col0 = nb * BN + (block >> 1) * 64;
    if (row0 >= g.m || col0 >= g.n) continue;
    float acc[4][4] = {};
    for (int k0 = 0; k0 < g.k; k0 += kPanelK) {
      tc::epilogue_sync();
      for (int i = tid; i < 64 * kPanelK; i += 256) {
        const int r = i / kPanelK, kk = i % kPanelK;
        sa[kk * kPanelPitch + r] = row0 + r < g.m && k0 + kk < g.k ? a[(row0 + r) * g.lda + k0 + kk] : 0.f;
        const int n = g.b_transposed ? r : i % 64, kb = g.b_transposed ? kk : i / 64;
        sb[kb * kPanelPitch + n] = col0 + n < g.n && k0 + kb < g.k ? b[g.b_transposed ? (col0 + n) * g.ldb + k0 + kb : (k0 + kb) * g.ldb + col0 + n] : 0.f;
      }
      tc::epilogue_sync();
#pragma unroll 4
      for (int kk = 0; kk < kPanelK; ++kk) {
        const float4 x = *reinterpret_cast<const float4*>(sa + kk * kPanelPitch + ty * 4);
        const float4 w = *reinterpret_cast<const float4*>(sb + kk * kPanelPitch + tx * 4);
        const float xs[4] = {x.x, x.y, x.z, x.w}, ws[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
          for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(xs[i], ws[j], acc[i][j]);
      }
    }
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int row = row0 + ty * 4 + i, col = col0 + tx * 4 + j;
        if (row >= g.m || col >= g.n) continue;
        float* out = c + bz * g.c_batch_stride + row * g.ldc + col;
        if (!(fabsf(__ldcg(out)) < INFINITY)) *out = acc[i][j];
      }
  }
}

// grid: a persistent CTA per SM over all tiles, or, in clusters, one tile per cluster.
template <int BN, bool kBTransposed, bool kRedo>
__global__ void __launch_bounds__(kThreads, 1)
gemm_tf32_fused_kernel(float* __restrict__ c, const __grid_constant__ Params p) {
  using S = Shape<BN>;
  constexpr int kStages = S::kStages;
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
  if (threadIdx.x < kRedoTiles / 32) bars->redo[threadIdx.x] = 0;
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
    // A (and B stored [N][K]): 16-byte unit u of rows r, r + 32, ...; eight lanes read 128 bytes of a row
    const int r = t >> 3, u = t & 7;
    const uint32_t at = r * 128 + ((u ^ (r & 7)) << 4);
    // B stored [K][N]: column n, units g0, g0 + kGroups, ...; a warp reads 128 bytes of a row of K
    constexpr int kGroups = kLoadWarps * 32 / BN, kBUnits = BN / 32;
    const int n = t % BN, g0 = t / BN;
    struct Regs {
      float a[4][4], b[kBUnits][4];
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
        for (int i = 0; i < kBUnits; ++i) load4(x.b[i], b, g.ldb, col0 + r + 32 * i, g.n, k + u * 4, g.k, p.vec_b != 0);
      } else {
        const int col = col0 + n;
#pragma unroll
        for (int i = 0; i < kBUnits; ++i) {
          const int k4 = k + (g0 + i * kGroups) * 4;
          const float* q = b + k4 * g.ldb + col;
#pragma unroll
          for (int j = 0; j < 4; ++j) x.b[i][j] = col < g.n && k4 + j < g.k ? q[j * g.ldb] : 0.f;
        }
      }
      if (++lk == num_kb) lk = 0, lt += tile_step;
      return true;
    };
    int stage = 0;
    uint32_t phase = 0;
    auto store = [&](const Regs& x) -> bool {
      if (!__all_sync(0xffffffffu, ptx::mbar_wait(&bars->empty[stage], phase ^ 1u, abort_flag, g.status, 91))) return false;
      const uint32_t base = ptx::smem_u32(smem + stage * S::kStageBytes);
#pragma unroll
      for (int i = 0; i < 4; ++i) split_store(base + at + i * 4096, base + kAPlane + at + i * 4096, x.a[i]);
      const uint32_t bb = base + 2 * kAPlane;
#pragma unroll
      for (int i = 0; i < kBUnits; ++i) {
        const uint32_t to = kBTransposed ? at + i * 4096 : n * 128 + (((g0 + i * kGroups) ^ (n & 7)) << 4);
        split_store(bb + to, bb + S::kBPlane + to, x.b[i]);
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
    constexpr uint32_t idesc = tc::make_idesc_tf32(kBM, BN);
    constexpr uint64_t kmajor = ptx::make_smem_desc_base(16, 1024);
    constexpr uint32_t hi32 = static_cast<uint32_t>(kmajor >> 32), lo32 = static_cast<uint32_t>(kmajor);
    auto desc = [](uint32_t lo) -> uint64_t { return (static_cast<uint64_t>(hi32) << 32) | lo; };
    const uint32_t smem_lo = lo32 | (ptx::smem_u32(smem) >> 4);
    int stage = 0, next_tile = first_tile, next_chunk = 0;
    uint32_t phase = 0, issued = 0;
    auto issue_chunk = [&]() -> bool {
      if (next_tile >= num_tiles) return true;
      const uint32_t acc = issued & 1u;
      if (!__all_sync(0xffffffffu, ptx::mbar_wait_relaxed(&bars->acc_empty[acc], ((issued >> 1) & 1u) ^ 1u, abort_flag, g.status, 92))) return false;
      const uint32_t d = tmem_base + acc * BN;
      const int kb_begin = next_chunk * g.chunk_kb, kb_end = min(num_kb, kb_begin + g.chunk_kb);
      for (int kb = kb_begin; kb < kb_end; ++kb) {
        if (!__all_sync(0xffffffffu, ptx::mbar_wait(&bars->full[stage], phase, abort_flag, g.status, 93))) return false;
        ptx::tcgen05_fence_after_thread_sync();
        const uint32_t a_hi = smem_lo + stage * (S::kStageBytes >> 4), a_lo = a_hi + (kAPlane >> 4);
        const uint32_t b_hi = a_hi + (2 * kAPlane >> 4), b_lo = b_hi + (S::kBPlane >> 4);
        if (ptx::elect_one_sync()) {
          // the small products first, then the large ones: what rounding the accumulator toward zero costs grows with what it holds
#pragma unroll
          for (int kk = 0; kk < kBK / tc::kUmmaK; ++kk) {
            tc::tcgen05_mma_tf32_ss(d, desc(a_lo + kk * 2), desc(b_hi + kk * 2), idesc, kk == 0 && kb == kb_begin ? 0u : 1u);
            tc::tcgen05_mma_tf32_ss(d, desc(a_hi + kk * 2), desc(b_lo + kk * 2), idesc, 1u);
          }
#pragma unroll
          for (int kk = 0; kk < kBK / tc::kUmmaK; ++kk) tc::tcgen05_mma_tf32_ss(d, desc(a_hi + kk * 2), desc(b_hi + kk * 2), idesc, 1u);
          ptx::tcgen05_commit(&bars->empty[stage]);
          if (kb == kb_end - 1) ptx::tcgen05_commit(&bars->acc_full[acc]);
        }
        __syncwarp();
        if (++stage == kStages) stage = 0, phase ^= 1u;
      }
      ++issued;
      if (++next_chunk == num_chunks) next_chunk = 0, next_tile += tile_step;
      return true;
    };
    uint32_t chunk_count = 0;
    bool alive = warp != 0 || issue_chunk();
    int seq = 0;
    for (int tile = first_tile; tile < num_tiles; tile += tile_step, ++seq) {
      float sum[kCols / 32][32];
#pragma unroll
      for (int cc = 0; cc < kCols / 32; ++cc)
#pragma unroll
        for (int i = 0; i < 32; ++i) sum[cc][i] = 0.f;
      for (int ch = 0; ch < num_chunks; ++ch, ++chunk_count) {
        const uint32_t acc = chunk_count & 1u;
        if (warp == 0) alive = alive && issue_chunk();
        if (!alive) break;
        if (!__all_sync(0xffffffffu, ptx::mbar_wait(&bars->acc_full[acc], (chunk_count >> 1) & 1u, abort_flag, g.status, 94))) {
          alive = false;
          break;
        }
        ptx::tcgen05_fence_after_thread_sync();
#pragma unroll
        for (int cc = 0; cc < kCols / 32; ++cc) {
          uint32_t v[32];
          ptx::tmem_ld_32x32b_x32(lane_addr + acc * BN + cc * 32, v);
          ptx::tmem_ld_wait();
#pragma unroll
          for (int i = 0; i < 32; ++i) sum[cc][i] += __uint_as_float(v[i]);
        }
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
        if (kRedo) {
          float z = 0.f;  // NaN where anything is infinite or NaN (rows and columns past C are so only beside such ones of C)
#pragma unroll
          for (int cc = 0; cc < kCols / 32; ++cc)
#pragma unroll
            for (int i = 0; i < 32; ++i) z = fmaf(sum[cc][i], 0.f, z);
          const int bit = min(seq, kRedoTiles - 1);
          if (__any_sync(0xffffffffu, z != 0.f) && lane == 0) atomicOr(&bars->redo[bit >> 5], 1u << (bit & 31));
        }
#pragma unroll
        for (int cc = 0; cc < kCols / 32; ++cc)
          tc::store_block_32x32<false>(c, g, b, mb * kBM + quad * 32, nb * BN + half * kCols + cc * 32, sum[cc], staging, lane, nullptr);
      }
    }
    if (kRedo && splits == 1 && !tc::epilogue_any(!alive)) {
      __threadfence();
      tc::epilogue_sync();
      seq = 0;
      for (int tile = first_tile; tile < num_tiles; tile += tile_step, ++seq) {
        const int bit = min(seq, kRedoTiles - 1);
        if ((bars->redo[bit >> 5] >> (bit & 31)) & 1u) redo_tile<BN>(p, c, reinterpret_cast<float*>(smem), tile, threadIdx.x);
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
        if (kRedo) odd |= !(fabsf(x.x) < INFINITY && fabsf(x.y) < INFINITY && fabsf(x.z) < INFINITY && fabsf(x.w) < INFINITY);
      }
    }
    if (kRedo && odd) bars->redo[0] = 1u;
    __threadfence();
    ptx::cluster_sync_all();  // nobody's partial tile goes while a peer reads it; all of the tile is in memory
    if (kRedo && bars->redo[0] != 0u && *abort_flag == 0u && threadIdx.x < 256) redo_tile<BN>(p, c, reinterpret_cast<float*>(smem), first_tile, threadIdx.x);
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

}  // namespace gemm_tf32_fused
}  // namespace tsm100
