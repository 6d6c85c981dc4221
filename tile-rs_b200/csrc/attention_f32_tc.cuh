// Fused attention forward for f32 tensors on the 5th-generation tensor cores (tcgen05, kind::tf32), f32-grade results.
//
// Semantics as attention_tf32x3.cuh (__tile_attention_f32, crates/tile_std/src/tile.rs:218-224;
// crates/rustc_codegen_tile/src/mlir_to_linalg.rs:1781-1902, :1191-1244; grouped heads
// crates/rustc_codegen_tile/src/mlir_to_gpu.rs:1657-1673); the scheme of three TF32 products per product on hi / lo
// parts, and of accumulating in short chunks, is that of gemm_tf32_tc.cuh.
//
// One streaming launch writes the hi / lo planes of K ([keys][D]) and of V, transposed ([D][keys]), so that both products
// see K-major operands only.  Then one CTA owns 128 query rows of one head and walks the keys in steps of 32:
//   warp 8       TMA producer: K_0, K_1, V_0, K_2, V_1, ... (hi and lo together, 256 * D bytes a unit) through a 5-deep
//                ring.  No multicast.
//   warp 9       S = Q K^T: the hi tile of Q stays in tensor memory for the CTA's life, the lo tile in shared memory.  A
//                128 x 32 x 8 product reads 4 KiB of A against 1 KiB of B; from shared memory that takes 40 cycles, 16 of which
//                the tensor core needs, so two of the three products take A from tensor memory.
//   warp 10      O += P V: P_hi, P_lo are read from tensor memory.
//   warps 0..3   softmax, one thread per query row; the running maximum is raised freely where a chunk of O begins and
//                otherwise only when it grows by more than 2^8 (the chunk in tensor memory is then rescaled).
//   warps 4..7   drain: the tensor core rounds its accumulator toward zero, so O is accumulated over kChunkSteps steps
//                (128 keys) from zero and then added, round to nearest, to running sums in registers (D per thread).
// S and the chunk of O are double-buffered, so that the products of one step run during the softmax of the next; P is not
// (tensor memory at D = 128: 2 * 128 of O, 2 * 32 of S, 32 + 32 of P, 128 of Q: all 512 columns).
// Bound: tensor pipe at the TF32 rate / 3; shared-memory reads of Q by the 32-wide S products come close behind.  16 heads of
// 4096 x 128, causal: 170 TFLOP/s as graph replays (0.63 of a third of the TF32 rate; 137 with both parts of Q in shared memory), 156 per
// call in a row of calls; 48 on the warp-level kernel.
#pragma once

#include "attention_simt.cuh"  // Params
#include "gemm_tf32_tc.cuh"    // split passes, tf32_rn, descriptors
#include "ptx.cuh"

namespace tsm100 {
namespace attn_f32_tc {

using gemm_tf32_tc::tf32_rn;

constexpr int kBQ = 128;           // query rows per CTA
constexpr int kBKV = 32;           // keys per step: one 128-byte swizzle row of f32
constexpr int kChunkSteps = 4;     // steps per accumulation chunk of O
constexpr int kThreads = 384;
constexpr int kRing = 5;
constexpr int kRegsOther = 56, kRegsSoftmax = 168, kRegsDrain = 224;
static_assert(128 * (kRegsOther + kRegsSoftmax + kRegsDrain) <= kThreads * 168, "setmaxnreg draws on the launch's registers");
constexpr int kTmemCols = 512;
constexpr int kTmemO = 0, kTmemS = 256, kTmemP = 320, kTmemQ = 384;  // two accumulators of 128, two of 32, 32 hi + 32 lo, 128
constexpr float kRescaleThreshold = 8.0f;              // log2 units
// its bounded waits report sites 71 .. 84

template <int D>
struct Shape {
  static constexpr int kQPlane = kBQ * D * 4;           // D / 32 groups of 128 rows x 128 bytes
  static constexpr int kUnitPlane = kBKV * D * 4;       // K: D / 32 groups of 32 rows x 128 bytes; V: D rows x 128 bytes
  static constexpr int kUnitBytes = 2 * kUnitPlane;     // hi, lo
  static constexpr int kRingOff = kQPlane;              // behind the lo tile of Q
  static constexpr int kRowsOff = kRingOff + kRing * kUnitBytes;  // float [3][128]: per chunk, the maximum it is scaled by
  static constexpr int kBarsOff = kRowsOff + 3 * kBQ * 4;
};
struct alignas(8) Barriers {
  uint64_t q_ready;
  uint64_t kv_full[kRing], kv_empty[kRing];
  uint64_t s_full[2], s_free[2];
  uint64_t p_ready, pv_done;
  uint64_t o_full[2], o_empty[2];
  uint64_t m_ready[3];   // the maximum of a chunk is in its row slot
  uint64_t l_ready;      // the row sums are in the slot after the last chunk's
  uint32_t tmem_base;
  uint32_t abort_flag;
  uint32_t pv_steps;     // steps whose P V has been issued (only grows)
};
template <int D>
constexpr int smem_bytes() {
  return Shape<D>::kBarsOff + static_cast<int>(sizeof(Barriers)) + 1024;
}
static_assert(smem_bytes<128>() <= 227 * 1024, "shared memory budget of one CTA");

struct Params {
  attn_simt::Params a;      // shapes, and the strides of Q and O
  uint32_t* status;
};

__device__ __forceinline__ void mma_tf32_ts(uint32_t d_tmem, uint32_t a_tmem, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n"
      ".reg .pred p;\n"
      "setp.ne.b32 p, %4, 0;\n"
      "tcgen05.mma.cta_group::1.kind::tf32 [%0], [%1], %2, %3, p;\n"
      "}\n" ::"r"(d_tmem),
      "r"(a_tmem), "l"(b_desc), "r"(idesc), "r"(accumulate)
      : "memory");
}

template <int D>
__global__ void __launch_bounds__(kThreads, 1)
attention_f32_tc_kernel(const __grid_constant__ CUtensorMap tmap_k_hi, const __grid_constant__ CUtensorMap tmap_k_lo,
                        const __grid_constant__ CUtensorMap tmap_v_hi, const __grid_constant__ CUtensorMap tmap_v_lo,
                        const float* __restrict__ q, float* __restrict__ o, const Params pp) {
  using Sh = Shape<D>;
  const attn_simt::Params& p = pp.a;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* ring = smem + Sh::kRingOff;
  float* row_slot = reinterpret_cast<float*>(smem + Sh::kRowsOff);
  Barriers* bars = reinterpret_cast<Barriers*>(smem + Sh::kBarsOff);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  volatile uint32_t* abort_flag = &bars->abort_flag;
  uint32_t* status = pp.status;

  // block -> (query block, head): the heads vary fastest, the heaviest query blocks of all heads come first when causal
  const int heads = p.batch * p.heads_q;
  const int q_blocks = (p.seq + kBQ - 1) / kBQ;
  const int bh = static_cast<int>(blockIdx.x) % heads;
  const int qb_raw = static_cast<int>(blockIdx.x) / heads;
  const int q0 = (p.causal ? q_blocks - 1 - qb_raw : qb_raw) * kBQ;
  const int kvh = bh / p.heads_q * p.heads_kv + bh % p.heads_q / (p.heads_q / p.heads_kv);
  const int n_all = (p.seq_kv + kBKV - 1) / kBKV;
  const int n = p.causal ? min(n_all, (min(q0 + kBQ, p.seq) - 1 + p.q_offset) / kBKV + 1) : n_all;  // steps, >= 1
  const int chunks = (n + kChunkSteps - 1) / kChunkSteps;

  if (threadIdx.x == 0) {
    ptx::mbar_init(&bars->q_ready, 128);
    ptx::mbar_init(&bars->p_ready, 128);
    ptx::mbar_init(&bars->pv_done, 1);
    for (int s = 0; s < kRing; ++s) {
      ptx::mbar_init(&bars->kv_full[s], 1);
      ptx::mbar_init(&bars->kv_empty[s], 1);
    }
    for (int i = 0; i < 2; ++i) {
      ptx::mbar_init(&bars->s_full[i], 1);
      ptx::mbar_init(&bars->s_free[i], 128);
      ptx::mbar_init(&bars->o_full[i], 1);
      ptx::mbar_init(&bars->o_empty[i], 128);
    }
    for (int i = 0; i < 3; ++i) ptx::mbar_init(&bars->m_ready[i], 128);
    ptx::mbar_init(&bars->l_ready, 128);
    bars->abort_flag = 0;
    bars->pv_steps = 0;
    ptx::fence_mbar_init();
  }
  if (warp == 9) {
    ptx::tmem_alloc(&bars->tmem_base, kTmemCols);
    ptx::tmem_relinquish_alloc_permit();
  }
  ptx::tcgen05_fence_before_thread_sync();
  __syncthreads();
  ptx::tcgen05_fence_after_thread_sync();
  const uint32_t tmem = bars->tmem_base;
  // ring positions: K_0, K_1, V_0, K_2, V_1, ..., K_{n-1}, V_{n-2}, V_{n-1}
  auto k_pos = [&](int j) { return j == 0 ? 0 : 2 * j - 1; };
  auto v_pos = [&](int j) { return j == n - 1 ? 2 * n - 1 : 2 * j + 2; };

  // Q, split (warps 0..3, one row each): hi to tensor memory, lo to the swizzled K-major tile in shared memory (16-byte unit u
  // of row r at position u ^ (r & 7) of its group of 32 columns)
  if (warp < 4) {
    const int r = warp * 32 + lane;
    const bool valid = q0 + r < p.seq;
    const float4* qr = reinterpret_cast<const float4*>(q + bh * p.q_head_stride + (q0 + r) * p.q_row_stride);
    const uint32_t base = ptx::smem_u32(smem) + r * 128;
#pragma unroll
    for (int c = 0; c < D / 32; ++c) {
      uint32_t hi[32];
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        const float4 x = valid ? qr[c * 8 + u] : make_float4(0.f, 0.f, 0.f, 0.f);
        const float4 h = make_float4(tf32_rn(x.x), tf32_rn(x.y), tf32_rn(x.z), tf32_rn(x.w));
        hi[4 * u] = __float_as_uint(h.x), hi[4 * u + 1] = __float_as_uint(h.y), hi[4 * u + 2] = __float_as_uint(h.z), hi[4 * u + 3] = __float_as_uint(h.w);
        ptx::st_shared_v4(base + c * (kBQ * 128) + ((u ^ (r & 7)) << 4), __float_as_uint(tf32_rn(x.x - h.x)), __float_as_uint(tf32_rn(x.y - h.y)),
                          __float_as_uint(tf32_rn(x.z - h.z)), __float_as_uint(tf32_rn(x.w - h.w)));
      }
      __syncwarp();
      ptx::tmem_st_32x32b_x32(tmem + (static_cast<uint32_t>(warp * 32) << 16) + kTmemQ + c * 32, hi);
    }
    ptx::tmem_st_wait();
    ptx::tcgen05_fence_before_thread_sync();
    ptx::fence_proxy_async_smem();
    ptx::mbar_arrive(&bars->q_ready);
  }

  if (warp == 8) {
    // ------------------------------ TMA producer ------------------------------
    ptx::setmaxnreg_dec<kRegsOther>();
    if (lane == 0) {
      const int total = 2 * n;
      for (int idx = 0; idx < total; ++idx) {
        const int slot = idx % kRing;
        if (!ptx::mbar_wait(&bars->kv_empty[slot], ((idx / kRing) & 1u) ^ 1u, abort_flag, status, 71)) break;
        ptx::mbar_arrive_expect_tx(&bars->kv_full[slot], Sh::kUnitBytes);
        const bool is_v = idx == total - 1 || (idx >= 2 && (idx & 1) == 0);
        const int step = idx == 0 ? 0 : idx == total - 1 ? n - 1 : is_v ? (idx >> 1) - 1 : (idx + 1) >> 1;
        uint8_t* dst = ring + slot * Sh::kUnitBytes;
        if (is_v) {
          ptx::tma_load_3d(dst, &tmap_v_hi, &bars->kv_full[slot], step * kBKV, 0, kvh);
          ptx::tma_load_3d(dst + Sh::kUnitPlane, &tmap_v_lo, &bars->kv_full[slot], step * kBKV, 0, kvh);
        } else {
#pragma unroll
          for (int c = 0; c < D / 32; ++c) {
            ptx::tma_load_3d(dst + c * (kBKV * 128), &tmap_k_hi, &bars->kv_full[slot], c * 32, step * kBKV, kvh);
            ptx::tma_load_3d(dst + Sh::kUnitPlane + c * (kBKV * 128), &tmap_k_lo, &bars->kv_full[slot], c * 32, step * kBKV, kvh);
          }
        }
      }
    }
  } else if (warp == 9 || warp == 10) {
    // ------------------------------ MMA issuers --------------------------------
    ptx::setmaxnreg_dec<kRegsOther>();
    constexpr uint64_t kmajor = ptx::make_smem_desc_base(16, 1024);
    constexpr uint32_t k_hi32 = static_cast<uint32_t>(kmajor >> 32), k_lo32 = static_cast<uint32_t>(kmajor);
    auto desc = [](uint32_t lo) -> uint64_t { return (static_cast<uint64_t>(k_hi32) << 32) | lo; };
    const uint32_t ring_lo = k_lo32 | (ptx::smem_u32(ring) >> 4);
    auto wait_kv = [&](int idx) -> bool {
      const bool r = ptx::mbar_wait_relaxed(&bars->kv_full[idx % kRing], (idx / kRing) & 1u, abort_flag, status, 72);
      return __all_sync(0xffffffffu, r);
    };
    bool ok = true;
    if (warp == 9) {
      constexpr uint32_t idesc = gemm_tf32_tc::make_idesc_tf32(kBQ, kBKV);
      const uint32_t q_lo32 = k_lo32 | (ptx::smem_u32(smem) >> 4);
      ok = __all_sync(0xffffffffu, ptx::mbar_wait(&bars->q_ready, 0, abort_flag, status, 73));
      ptx::tcgen05_fence_after_thread_sync();
      volatile uint32_t* pv_steps = &bars->pv_steps;
      for (int j = 0; j < n && ok; ++j) {
        // not before the P V of step j - 2 is queued: the tensor core would take this product first
        if (j >= 2 && !(ok = __all_sync(0xffffffffu, ptx::wait_counter_ge(pv_steps, static_cast<uint32_t>(j - 1), abort_flag, status, 74)))) break;
        if (!(ok = wait_kv(k_pos(j)))) break;
        if (j >= 2 && !(ok = __all_sync(0xffffffffu, ptx::mbar_wait_relaxed(&bars->s_free[j & 1], ((j - 2) >> 1) & 1u, abort_flag, status, 75)))) break;
        ptx::tcgen05_fence_after_thread_sync();
        const uint32_t d = tmem + kTmemS + (j & 1) * kBKV;
        const uint32_t b_hi = ring_lo + (k_pos(j) % kRing) * (Sh::kUnitBytes >> 4), b_lo = b_hi + (Sh::kUnitPlane >> 4);
        if (ptx::elect_one_sync()) {
          // the small products first, then the large ones: the accumulator is rounded toward zero at every product, and
          // what that costs grows with what it holds
#pragma unroll
          for (int kk = 0; kk < D / 8; ++kk) {
            const uint32_t a_off = (kk >> 2) * ((kBQ * 128) >> 4) + (kk & 3) * 2, b_off = (kk >> 2) * ((kBKV * 128) >> 4) + (kk & 3) * 2;
            gemm_tf32_tc::tcgen05_mma_tf32_ss(d, desc(q_lo32 + a_off), desc(b_hi + b_off), idesc, kk != 0 ? 1u : 0u);
            mma_tf32_ts(d, tmem + kTmemQ + kk * 8, desc(b_lo + b_off), idesc, 1u);
          }
#pragma unroll
          for (int kk = 0; kk < D / 8; ++kk) {
            const uint32_t b_off = (kk >> 2) * ((kBKV * 128) >> 4) + (kk & 3) * 2;
            mma_tf32_ts(d, tmem + kTmemQ + kk * 8, desc(b_hi + b_off), idesc, 1u);
          }
          ptx::tcgen05_commit(&bars->s_full[j & 1]);
          ptx::tcgen05_commit(&bars->kv_empty[k_pos(j) % kRing]);
        }
        __syncwarp();
      }
    } else {
      constexpr uint32_t idesc = gemm_tf32_tc::make_idesc_tf32(kBQ, D);
      for (int j = 0; j < n && ok; ++j) {
        const int c = j / kChunkSteps, acc = c & 1;
        const bool first = j % kChunkSteps == 0, last = j % kChunkSteps == kChunkSteps - 1 || j == n - 1;
        if (!(ok = wait_kv(v_pos(j)))) break;
        if (first && c >= 2 && !(ok = __all_sync(0xffffffffu, ptx::mbar_wait_relaxed(&bars->o_empty[acc], ((c - 2) >> 1) & 1u, abort_flag, status, 76)))) break;
        if (!(ok = __all_sync(0xffffffffu, ptx::mbar_wait(&bars->p_ready, j & 1u, abort_flag, status, 77)))) break;
        ptx::tcgen05_fence_after_thread_sync();
        const uint32_t d = tmem + kTmemO + acc * 128;
        const uint32_t a_hi = tmem + kTmemP, a_lo = a_hi + kBKV;
        const uint32_t b_hi = ring_lo + (v_pos(j) % kRing) * (Sh::kUnitBytes >> 4), b_lo = b_hi + (Sh::kUnitPlane >> 4);
        if (ptx::elect_one_sync()) {
#pragma unroll
          for (int kk = 0; kk < kBKV / 8; ++kk) {
            mma_tf32_ts(d, a_lo + kk * 8, desc(b_hi + kk * 2), idesc, (first && kk == 0) ? 0u : 1u);
            mma_tf32_ts(d, a_hi + kk * 8, desc(b_lo + kk * 2), idesc, 1u);
            mma_tf32_ts(d, a_hi + kk * 8, desc(b_hi + kk * 2), idesc, 1u);
          }
          ptx::tcgen05_commit(&bars->pv_done);
          ptx::tcgen05_commit(&bars->kv_empty[v_pos(j) % kRing]);
          if (last) ptx::tcgen05_commit(&bars->o_full[acc]);
          *const_cast<volatile uint32_t*>(&bars->pv_steps) = static_cast<uint32_t>(j + 1);
        }
        __syncwarp();
      }
    }
  } else if (warp == 11) {
    ptx::setmaxnreg_dec<kRegsOther>();
  } else if (warp < 4) {
    // ------------------------------ softmax ------------------------------------
    ptx::setmaxnreg_inc<kRegsSoftmax>();
    const int r = warp * 32 + lane;        // row of the tile == TMEM lane
    const int qrow = q0 + r;
    const int limit = p.causal ? min(qrow + p.q_offset, p.seq_kv - 1) : p.seq_kv - 1;  // last visible key
    const uint32_t lane_base = tmem + (static_cast<uint32_t>(warp * 32) << 16);
    const float sl2 = p.scale * 1.4426950408889634f;
    float m_used = -INFINITY, l = 0.f;     // running maximum in raw score units, row sum scaled by it
    bool alive = true;
    for (int j = 0; j < n; ++j) {
      const int b = j & 1;
      if (!__all_sync(0xffffffffu, ptx::mbar_wait(&bars->s_full[b], (j >> 1) & 1u, abort_flag, status, 78))) {
        alive = false;
        break;
      }
      ptx::tcgen05_fence_after_thread_sync();
      uint32_t v[32];
      ptx::tmem_ld_32x32b_x32(lane_base + kTmemS + b * kBKV, v);
      ptx::tmem_ld_wait();
      ptx::tcgen05_fence_before_thread_sync();
      ptx::mbar_arrive(&bars->s_free[b]);
      const int key0 = j * kBKV;
      if (key0 + kBKV - 1 > limit) {
#pragma unroll
        for (int i = 0; i < 32; ++i)
          if (key0 + i > limit) v[i] = 0xff800000u;  // -inf
      }
      float mx4[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
      for (int i = 0; i < 32; i += 2)
        mx4[(i >> 1) & 3] = ptx::fmax3(mx4[(i >> 1) & 3], __uint_as_float(v[i]), __uint_as_float(v[i + 1]));
      const float m_new = fmaxf(m_used, fmaxf(fmaxf(mx4[0], mx4[1]), fmaxf(mx4[2], mx4[3])));
      const bool chunk_start = j % kChunkSteps == 0;
      if (chunk_start) {
        // nothing of this chunk is in tensor memory yet; the drain warps rescale their sums
        if (m_new != m_used) {
          l *= ptx::ex2_approx((m_used - m_new) * sl2);  // l = 0 while m_used = -inf
          m_used = m_new;
        }
      } else if (__any_sync(0xffffffffu, (m_new - m_used) * sl2 > kRescaleThreshold)) {
        if (!__all_sync(0xffffffffu, ptx::mbar_wait(&bars->pv_done, (j - 1) & 1u, abort_flag, status, 79))) {
          alive = false;
          break;
        }
        ptx::tcgen05_fence_after_thread_sync();
        const bool need = (m_new - m_used) * sl2 > kRescaleThreshold;
        const float alpha = need ? ptx::ex2_approx((m_used - m_new) * sl2) : 1.0f;
        if (need) m_used = m_new;
        l *= alpha;
        const uint32_t to = lane_base + kTmemO + ((j / kChunkSteps) & 1) * 128;
#pragma unroll 1
        for (int c = 0; c < D / 32; ++c) {
          uint32_t ov[32];
          ptx::tmem_ld_32x32b_x32(to + c * 32, ov);
          ptx::tmem_ld_wait();
#pragma unroll
          for (int i = 0; i < 32; ++i) ov[i] = __float_as_uint(__uint_as_float(ov[i]) * alpha);
          ptx::tmem_st_32x32b_x32(to + c * 32, ov);
        }
        ptx::tmem_st_wait();
        ptx::tcgen05_fence_before_thread_sync();
      }
      // a row that has seen nothing but -inf so far: probabilities 0, not NaN
      const float nms = m_used == -INFINITY ? 0.f : -m_used * sl2;
      uint32_t hi[32], lo[32];
      float ls[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
      for (int i = 0; i < 32; ++i) {
        const float e = ptx::ex2_approx(fmaf(__uint_as_float(v[i]), sl2, nms));
        ls[i & 3] += e;
        const float h = tf32_rn(e);
        hi[i] = __float_as_uint(h);
        lo[i] = __float_as_uint(e - h);  // exact; the tensor core reads its top 11 bits
      }
      l += (ls[0] + ls[1]) + (ls[2] + ls[3]);
      // P of step j - 1 has been read
      if (j >= 1 && !__all_sync(0xffffffffu, ptx::mbar_wait(&bars->pv_done, (j - 1) & 1u, abort_flag, status, 80))) {
        alive = false;
        break;
      }
      __syncwarp();
      ptx::tcgen05_fence_after_thread_sync();
      const uint32_t tp = lane_base + kTmemP;
      ptx::tmem_st_32x32b_x32(tp, hi);
      ptx::tmem_st_32x32b_x32(tp + kBKV, lo);
      ptx::tmem_st_wait();
      ptx::tcgen05_fence_before_thread_sync();
      ptx::mbar_arrive(&bars->p_ready);
      if (j % kChunkSteps == kChunkSteps - 1 || j == n - 1) {
        // slot c % 3: the wait above says that P V of step j - 1 was issued, which (accumulators alternate) says that
        // the drain warps are done with chunk c - 3
        const int c3 = (j / kChunkSteps) % 3;
        row_slot[c3 * kBQ + r] = m_used;
        ptx::mbar_arrive(&bars->m_ready[c3]);
      }
    }
    // the row sum takes the slot after the last chunk's, once the last product has retired: by then the chunk that had it
    // (chunks - 3) is drained
    if (alive && __all_sync(0xffffffffu, ptx::mbar_wait(&bars->pv_done, (n - 1) & 1u, abort_flag, status, 81))) {
      row_slot[(chunks % 3) * kBQ + r] = l;
      ptx::mbar_arrive(&bars->l_ready);
    }
  } else {
    // ------------------------------ drain and output ---------------------------
    ptx::setmaxnreg_inc<kRegsDrain>();
    const int quad = warp & 3;
    const int r = quad * 32 + lane;
    const uint32_t lane_base = tmem + (static_cast<uint32_t>(quad * 32) << 16);
    const float sl2 = p.scale * 1.4426950408889634f;
    float sum[D];
#pragma unroll
    for (int i = 0; i < D; ++i) sum[i] = 0.f;
    float m_prev = -INFINITY;
    bool alive = true;
    for (int c = 0; c < chunks; ++c) {
      const int acc = c & 1;
      bool ready = ptx::mbar_wait(&bars->m_ready[c % 3], (c / 3) & 1u, abort_flag, status, 82);
      ready = ready && ptx::mbar_wait(&bars->o_full[acc], (c >> 1) & 1u, abort_flag, status, 83);
      if (!__all_sync(0xffffffffu, ready)) {
        alive = false;
        break;
      }
      ptx::tcgen05_fence_after_thread_sync();
      const float m_c = row_slot[(c % 3) * kBQ + r];
      const float alpha = m_c == m_prev ? 1.0f : ptx::ex2_approx((m_prev - m_c) * sl2);  // 0 before the first chunk
      m_prev = m_c;
#pragma unroll
      for (int cc = 0; cc < D / 32; ++cc) {
        uint32_t ov[32];
        ptx::tmem_ld_32x32b_x32(lane_base + kTmemO + acc * 128 + cc * 32, ov);
        ptx::tmem_ld_wait();
#pragma unroll
        for (int i = 0; i < 32; ++i) sum[cc * 32 + i] = fmaf(sum[cc * 32 + i], alpha, __uint_as_float(ov[i]));
      }
      ptx::tcgen05_fence_before_thread_sync();
      ptx::mbar_arrive(&bars->o_empty[acc]);
    }
    if (alive && __all_sync(0xffffffffu, ptx::mbar_wait(&bars->l_ready, 0, abort_flag, status, 84))) {
      const float inv = 1.0f / row_slot[(chunks % 3) * kBQ + r];
      if (q0 + r < p.seq) {
        float4* orow = reinterpret_cast<float4*>(o + bh * p.o_head_stride + (q0 + r) * p.o_row_stride);
#pragma unroll
        for (int i = 0; i < D / 4; ++i)
          orow[i] = make_float4(sum[4 * i] * inv, sum[4 * i + 1] * inv, sum[4 * i + 2] * inv, sum[4 * i + 3] * inv);
      }
    }
  }

  // ------------------------------ teardown ------------------------------------
  if (*abort_flag != 0u) {
    const unsigned long long t0 = ptx::globaltimer_ns();
    while (ptx::globaltimer_ns() - t0 < 1000000ull) {
    }
  }
  ptx::tcgen05_fence_before_thread_sync();
  __syncthreads();
  if (warp == 9) {
    ptx::tcgen05_fence_after_thread_sync();
    ptx::tmem_dealloc(tmem, kTmemCols);
  }
}

}  // namespace attn_f32_tc
}  // namespace tsm100
