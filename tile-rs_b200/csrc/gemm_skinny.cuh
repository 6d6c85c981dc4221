// 16-bit GEMM for problems with few output tiles: a handful of rows of A against a large B (the projections of a decoding
// step), and any shape whose 256 x 256 tiles leave most SM pairs of gemm_tc2.cuh without one (the rule is in route.hpp).
//
//   C[b][M,N] = A[b][M,K] * B[b], semantics and operand forms as in gemm_tc.cuh (crates/tile_std/src/tile.rs:1982-1986,
//   :2017-2031; crates/rustc_codegen_tile/src/mlir_to_linalg.rs:1345-1393).
//
// Bound for a few rows: HBM, B is read once.  So the roles are swapped: B fills the 128-row side of the tensor core and
// the rows of A its N side, NT = 16 .. 128 wide (a 16-row problem then costs 16 columns of tensor work instead of 128
// rows of it), and where 128-column tiles are fewer than the SMs can take, a cluster of up to 8 CTAs splits K.  The
// partial tiles are summed in rank order through distributed shared memory, so results do not depend on timing.
// 16 rows against [16384][4096]: 32.9 us on the 128 x 256 tiles of gemm_tc.cuh (64 CTAs), 25.8 here (5.2 TB/s); against
// [4096][16384] 98.8 us (16 CTAs) and 26.1.  One CTA per SM instead of two, unsplit where it can be: 26.8 and 27.2.
// About 100 KiB of shared memory per CTA: two CTAs per SM, one of which loads while the other starts or ends.
//
// One CTA = one (128 columns of C, NT rows, K range).  128 threads: warp 0 TMA producer, warp 1 tensor-memory allocation
// and MMA issue, then all four warps read the accumulator (lane = column of C, TMEM column = row of C).
#pragma once

#include "gemm_tc.cuh"
#include "ptx.cuh"

namespace tsm100 {
namespace gemm_skinny {

constexpr int kBN = 128;                 // columns of C per tile: the tensor core's M side
constexpr int kBK = 64;
constexpr int kThreads = 128;
constexpr int kMaxSplit = 8;
constexpr int kWBytes = kBN * kBK * 2;   // 16 KiB of B per stage
constexpr int kMaxStages = 6;
constexpr int kAhead = 8;                // tiles of B that a CTA fetches into the L2 before the kernel before it has ended

template <int NT>
struct Shape {
  static constexpr int kXBytes = NT * kBK * 2;  // rows of A per stage
  static constexpr int kStageBytes = kWBytes + kXBytes;
  static constexpr int kStages = NT <= 16 ? 6 : NT <= 32 ? 5 : NT <= 64 ? 4 : 3;
  static constexpr int kTmemCols = NT < 32 ? 32 : NT;
};

struct alignas(8) Barriers {
  uint64_t full[kMaxStages];
  uint64_t empty[kMaxStages];
  uint64_t acc_full;
  uint32_t tmem_base;
  uint32_t abort_flag;
};

template <int NT>
constexpr int smem_bytes() {
  return Shape<NT>::kStages * Shape<NT>::kStageBytes + static_cast<int>(sizeof(Barriers)) + 1024;
}
// the partial tile of a split (NT rows x 128 columns, f32) takes the place of the stages
static_assert(Shape<128>::kStages * Shape<128>::kStageBytes >= 128 * kBN * 4 && Shape<16>::kStages * Shape<16>::kStageBytes >= 16 * kBN * 4,
              "the partial tile fits the stages");
static_assert(2 * (smem_bytes<128>() + 1024) <= 227 * 1024 && 2 * (smem_bytes<16>() + 1024) <= 227 * 1024 &&
              2 * (smem_bytes<64>() + 1024) <= 227 * 1024 && 2 * (smem_bytes<32>() + 1024) <= 227 * 1024, "two CTAs per SM");

struct Params {
  int32_t m, n, k, batch;
  int32_t m_blocks, n_blocks;
  int32_t kb_per_cta;       // 64-deep k-blocks per CTA of the cluster (every CTA has at least one)
  int64_t c_batch_stride;
  int64_t ldc;
  uint32_t* status;
  int32_t early;            // the next kernel may be placed from the start
};

template <typename OutT>
__device__ __forceinline__ OutT narrow(float f);
template <>
__device__ __forceinline__ float narrow<float>(float f) { return f; }
template <>
__device__ __forceinline__ __nv_bfloat16 narrow<__nv_bfloat16>(float f) { return __float2bfloat16_rn(f); }
template <>
__device__ __forceinline__ __half narrow<__half>(float f) { return __float2half_rn(f); }

// grid: ((batch * n_blocks + nb) * m_blocks + mb) * cluster size + rank; CTAs that share a tile of B are neighbours.
// kLoose: rows of C start anywhere.
template <typename OutT, bool kBTransposed, bool kIsBf16, int NT, bool kLoose>
__global__ void __launch_bounds__(kThreads)
gemm_skinny_kernel(const __grid_constant__ CUtensorMap tmap_a, const __grid_constant__ CUtensorMap tmap_b,
                   OutT* __restrict__ c, const Params p) {
  using S = Shape<NT>;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  Barriers* bars = reinterpret_cast<Barriers*>(smem + S::kStages * S::kStageBytes);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  volatile uint32_t* abort_flag = &bars->abort_flag;

  const uint32_t splits = ptx::cluster_nctarank(), rank = ptx::cluster_ctarank();
  int t = static_cast<int>(blockIdx.x / splits);
  const int mb = t % p.m_blocks;
  t /= p.m_blocks;
  const int nb = t % p.n_blocks;
  const int b = t / p.n_blocks;
  const int kb_all = (p.k + kBK - 1) / kBK;
  const int kb0 = static_cast<int>(rank) * p.kb_per_cta;
  const int num_kb = min(kb_all - kb0, p.kb_per_cta);

  if (threadIdx.x == 0) {
    for (int s = 0; s < S::kStages; ++s) {
      ptx::mbar_init(&bars->full[s], 1);
      ptx::mbar_init(&bars->empty[s], 1);
    }
    ptx::mbar_init(&bars->acc_full, 1);
    bars->abort_flag = 0;
    ptx::fence_mbar_init();
  }
  if (warp == 1) {
    ptx::tmem_alloc(&bars->tmem_base, S::kTmemCols);
    ptx::tmem_relinquish_alloc_permit();
  }
  ptx::tcgen05_fence_before_thread_sync();
  __syncthreads();
  ptx::tcgen05_fence_after_thread_sync();
  const uint32_t tmem_base = bars->tmem_base;
  if (p.early) ptx::launch_dependents();
  if (threadIdx.x == 0) {
    ptx::prefetch_tensormap(&tmap_a);
    ptx::prefetch_tensormap(&tmap_b);
    // while the kernel before this one runs: its first tiles of B
    for (int i = 0; i < min(num_kb, kAhead); ++i) {
      const int k0 = (kb0 + i) * kBK;
      if (kBTransposed) {
        ptx::prefetch_l2_3d(&tmap_b, k0, nb * kBN, b);
      } else {
        ptx::prefetch_l2_3d(&tmap_b, nb * kBN, k0, b);
        ptx::prefetch_l2_3d(&tmap_b, nb * kBN + 64, k0, b);
      }
    }
  }
  ptx::wait_prior_grid();

  if (warp == 0) {
    if (lane == 0) {
      int stage = 0;
      uint32_t phase = 0;
      for (int i = 0; i < num_kb; ++i) {
        if (!ptx::mbar_wait(&bars->empty[stage], phase ^ 1u, abort_flag, p.status, 51)) break;
        uint8_t* w = smem + stage * S::kStageBytes;
        const int k0 = (kb0 + i) * kBK;
        ptx::mbar_arrive_expect_tx(&bars->full[stage], S::kStageBytes);
        if (kBTransposed) {
          ptx::tma_load_3d(w, &tmap_b, &bars->full[stage], k0, nb * kBN, b);
        } else {  // [K][N]: two 64-column groups of 64 k rows
          ptx::tma_load_3d(w, &tmap_b, &bars->full[stage], nb * kBN, k0, b);
          ptx::tma_load_3d(w + kWBytes / 2, &tmap_b, &bars->full[stage], nb * kBN + 64, k0, b);
        }
        ptx::tma_load_3d(w + kWBytes, &tmap_a, &bars->full[stage], k0, mb * NT, b);
        if (++stage == S::kStages) {
          stage = 0;
          phase ^= 1u;
        }
      }
    }
  } else if (warp == 1) {
    if (lane == 0) {
      constexpr uint32_t idesc = ptx::make_idesc_f16(kBN, NT, !kBTransposed, false, kIsBf16);
      constexpr uint64_t kmajor = ptx::make_smem_desc_base(16, 1024);
      constexpr uint64_t mnmajor = ptx::make_smem_desc_base(kWBytes / 2, 1024);
      int stage = 0;
      uint32_t phase = 0;
      bool ok = true;
      for (int i = 0; i < num_kb; ++i) {
        if (!(ok = ptx::mbar_wait_relaxed(&bars->full[stage], phase, abort_flag, p.status, 52))) break;
        ptx::tcgen05_fence_after_thread_sync();
        const uint32_t w = ptx::smem_u32(smem + stage * S::kStageBytes), x = w + kWBytes;
#pragma unroll
        for (int kk = 0; kk < kBK / 16; ++kk) {
          const uint64_t wd = kBTransposed ? ptx::smem_desc(kmajor, w + kk * 32) : ptx::smem_desc(mnmajor, w + kk * 2048);
          ptx::tcgen05_mma_f16_ss(tmem_base, wd, ptx::smem_desc(kmajor, x + kk * 32), idesc, (i | kk) != 0 ? 1u : 0u);
        }
        ptx::tcgen05_commit(&bars->empty[stage]);
        if (++stage == S::kStages) {
          stage = 0;
          phase ^= 1u;
        }
      }
      if (ok) ptx::tcgen05_commit(&bars->acc_full);
    }
  }
  __syncwarp();

  // ------------------------------ accumulator -> C ------------------------------
  const bool ready = __all_sync(0xffffffffu, ptx::mbar_wait(&bars->acc_full, 0, abort_flag, p.status, 53));
  ptx::tcgen05_fence_after_thread_sync();
  // not before, unless the host says so (route.hpp: skinny_places_early): 11 x 4104 x 2064 of a batch of 4 in a row of calls 16.8 us with this at
  // the start of the kernel, 14.2 here
  ptx::launch_dependents();
  const uint32_t lane_addr = tmem_base + (static_cast<uint32_t>(warp * 32) << 16);
  constexpr int kStep = NT < 32 ? 16 : 32;  // rows of C (TMEM columns) per read
  OutT* cb = c + static_cast<int64_t>(b) * p.c_batch_stride;
  const int rows = min(NT, p.m - mb * NT);
  if (splits == 1) {
    const int col = nb * kBN + warp * 32 + lane;
    if (ready) {
#pragma unroll
      for (int r0 = 0; r0 < NT; r0 += kStep) {
        if (r0 >= rows) break;
        uint32_t v[kStep];
        if constexpr (kStep == 16) ptx::tmem_ld_32x32b_x16(lane_addr + r0, v);
        else ptx::tmem_ld_32x32b_x32(lane_addr + r0, v);
        ptx::tmem_ld_wait();
        OutT* dst = cb + static_cast<int64_t>(mb * NT + r0) * p.ldc + col;
        if (col < p.n) {
#pragma unroll
          for (int i = 0; i < kStep; ++i)
            if (r0 + i < rows) dst[i * p.ldc] = narrow<OutT>(__uint_as_float(v[i]));
        }
      }
    }
  } else {
    // every CTA leaves its partial tile in its stages (all copies into them and products from them have retired) ...
    float* part = reinterpret_cast<float*>(smem);
    if (ready) {
#pragma unroll
      for (int r0 = 0; r0 < NT; r0 += kStep) {
        if (r0 >= rows) break;
        uint32_t v[kStep];
        if constexpr (kStep == 16) ptx::tmem_ld_32x32b_x16(lane_addr + r0, v);
        else ptx::tmem_ld_32x32b_x32(lane_addr + r0, v);
        ptx::tmem_ld_wait();
#pragma unroll
        for (int i = 0; i < kStep; ++i) part[(r0 + i) * kBN + warp * 32 + lane] = __uint_as_float(v[i]);
      }
    }
    ptx::cluster_sync_all();
    // ... and sums its share of the rows over all of them, in rank order
    const uint32_t part_addr = ptx::smem_u32(part);
    const int items = rows * (kBN / 4);  // four columns each
    for (int i = static_cast<int>(rank) * kThreads + threadIdx.x; i < items; i += static_cast<int>(splits) * kThreads) {
      float4 v[kMaxSplit];
#pragma unroll
      for (int q = 0; q < kMaxSplit; ++q)
        if (q < static_cast<int>(splits)) v[q] = ptx::ld_shared_cluster_f32x4(ptx::mapa_shared(part_addr + i * 16, q));
      float4 s = v[0];
#pragma unroll
      for (int q = 1; q < kMaxSplit; ++q)
        if (q < static_cast<int>(splits)) s.x += v[q].x, s.y += v[q].y, s.z += v[q].z, s.w += v[q].w;
      const int col = nb * kBN + (i % (kBN / 4)) * 4;
      if (col < p.n) {  // N is a multiple of 4 and rows of C start on 16-byte boundaries, unless loose
        OutT* dst = cb + static_cast<int64_t>(mb * NT + i / (kBN / 4)) * p.ldc + col;
        if constexpr (kLoose) {
          const float x[4] = {s.x, s.y, s.z, s.w};
#pragma unroll
          for (int j = 0; j < 4; ++j)
            if (col + j < p.n) dst[j] = narrow<OutT>(x[j]);
        } else if constexpr (sizeof(OutT) == 4) {
          *reinterpret_cast<float4*>(dst) = s;
        } else {
          OutT o4[4] = {narrow<OutT>(s.x), narrow<OutT>(s.y), narrow<OutT>(s.z), narrow<OutT>(s.w)};
          *reinterpret_cast<uint2*>(dst) = *reinterpret_cast<const uint2*>(o4);
        }
      }
    }
    ptx::cluster_sync_all();  // nobody's partial tile goes while a peer reads it
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
    ptx::tmem_dealloc(tmem_base, S::kTmemCols);
  }
}

}  // namespace gemm_skinny
}  // namespace tsm100
