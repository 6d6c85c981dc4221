// Fused attention forward for 16-bit heads of 64 and less: O = softmax(Q K^T / sqrt(d)) V, as attention_tc.cuh (semantics and citations
// there), with d any multiple of 8 up to 64 (the tensor maps end at d and fill the rest of a 64-wide row with zeros).
//
// The probabilities are handed to P V as hi + lo, two 16-bit numbers whose sum is the f32 value to 2^-17 of it (bf16), or to 2^-22 of
// it or 2^-32 of the row's largest (f16).  With 64 columns of O that is as much tensor work as one 128-wide product, but through shared
// memory it is twice the traffic: scores and products would read 256 KiB a step and the probabilities write 128, 3250 cycles of
// shared memory against 2048 of exponentials.  So the probabilities stay in tensor memory: they take the place of the scores they
// were made from (hi in the first half of a buffer's 128 columns, lo in the second), and P V reads them from there.
//
// One CTA owns 256 query rows of one (batch, head): two 128-row tiles A and B; keys go by in steps of 128.
//   warp 8       TMA producer: Q once, then K_0, K_1, V_0, K_2, V_1, ... (128 x 64 tiles, 128-byte swizzle) through a ring.  No multicast.
//   warp 9       issues every S = Q_g K_j^T, warp 10 every O_g += P V_j.
//   warps 0..3   softmax of tile A, warps 4..7 of tile B: one thread per query row (tensor-memory lane).
// Tensor memory: three buffers of 128 columns that the (tile, step) jobs A_0, B_0, A_1, B_1, ... take in turn, and O_A, O_B of 64: all 512.
// While both tiles are in their softmax the third buffer receives the scores that the tile to finish first needs next.
// kCache, kSplit: as in attention_tc.cuh.
#pragma once

#include "attention_tc.cuh"
#include "ptx.cuh"

namespace tsm100 {
namespace attn_narrow {

using attn::Params;

constexpr int kD = 64;
constexpr int kBQ = attn::kBQ, kBKV = attn::kBKV;
constexpr int kThreads = 384;            // warps 0..3 softmax A, 4..7 softmax B, 8 TMA, 9 scores, 10 products, 11 idle
constexpr int kRegsSoftmax = 224, kRegsOther = 56;
static_assert(2 * kRegsSoftmax + kRegsOther <= 3 * 168, "setmaxnreg draws on the launch's registers");
constexpr int kTmemCols = 512;
constexpr int kBuffers = 3;
constexpr int kTmemO = kBuffers * 128;
constexpr int kRing = 6;
constexpr int kTileBytes = 128 * 64 * 2;
constexpr int kRingOff = 2 * kTileBytes;
constexpr int kBarsOff = kRingOff + kRing * kTileBytes;
// its bounded waits report sites 101 .. 116

struct alignas(8) Barriers {
  uint64_t q_full;
  uint64_t kv_full[kRing], kv_empty[kRing];
  uint64_t s_full[kBuffers];    // the scores of a job are in its buffer
  uint64_t p_ready[kBuffers];   // its probabilities have taken their place
  uint64_t buf_free[kBuffers];  // its product has read them
  // Per tile, of even and of odd steps: the product of a step has retired.  A softmax thread may be two products ahead of the tensor
  // core when it waits for the last one, and the parity of one barrier cannot tell a phase from the one two before it.  With the steps
  // on two barriers the phase before on the same barrier is of step j - 2 or earlier, which the scores of step j have waited for.
  uint64_t pv_done[2][2];
  uint32_t tmem_base;
  uint32_t abort_flag;
};
constexpr int kSmemBytes = kBarsOff + static_cast<int>(sizeof(Barriers)) + 1024;
static_assert(kSmemBytes <= 227 * 1024, "shared memory budget of one CTA");

// f16 numbers end at 2^-24: the probabilities (2^8 at most, see kRescaleThreshold) and their sum are taken 2^7 times as large, so that
// a long tail of them down to 2^-32 of the largest counts in P V as it does in the sum
template <bool kIsBf16>
constexpr float kPShift = kIsBf16 ? 0.0f : 7.0f;

template <bool kIsBf16, bool kCache, bool kSplit, bool kLone = kSplit>
__global__ void __launch_bounds__(kThreads, 1)
attention_narrow_kernel(const __grid_constant__ CUtensorMap tmap_q, const __grid_constant__ CUtensorMap tmap_k,
                        const __grid_constant__ CUtensorMap tmap_v, uint16_t* __restrict__ o, const Params p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* smem_kv = smem + kRingOff;
  Barriers* bars = reinterpret_cast<Barriers*>(smem + kBarsOff);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  volatile uint32_t* abort_flag = &bars->abort_flag;

  const int splits = kSplit ? p.splits : 1;
  const int rank = kSplit ? static_cast<int>(blockIdx.x) % splits : 0;
  const int block = kSplit ? static_cast<int>(blockIdx.x) / splits : static_cast<int>(blockIdx.x);
  int bh, kvh, qb;
  attn::block_coords(p, block, bh, kvh, qb);
  const int q0 = kLone && !kSplit ? qb * p.block_rows : qb * (2 * kBQ);
  const int seq_kv = kCache ? p.seq_kv : p.seq;
  const int q_off = kCache ? p.q_offset : 0;
  const int n_kv_all = (seq_kv + kBKV - 1) / kBKV;
  // number of KV steps each tile needs (causal: up to and including the step of its last row's own position)
  const int n_a_all = p.causal ? min(n_kv_all, (q0 + kBQ - 1 + q_off) / kBKV + 1) : n_kv_all;
  const bool lone = kLone && ((!kSplit && p.block_rows == kBQ) || q0 + kBQ >= p.seq);  // no tile B, as in attention_tc.cuh
  const int n_b_all = lone ? n_a_all : p.causal ? min(n_kv_all, (q0 + 2 * kBQ - 1 + q_off) / kBKV + 1) : n_kv_all;
  // kSplit: this CTA's range [j0, j0 + n_b) of them, possibly empty
  const int per_rank = kSplit ? (n_b_all + splits - 1) / splits : n_b_all;
  const int j0 = kSplit ? min(rank * per_rank, n_b_all) : 0;
  const int n_b = kSplit ? min(per_rank, n_b_all - j0) : n_b_all;
  const int n_a = kSplit ? max(0, min(n_a_all - j0, n_b)) : n_a_all;
  // the place of step j of tile g among the jobs: A_0, B_0, A_1, B_1, ... and one tile alone once the other has no step any more
  auto job = [&](int g, int j) { return lone ? j : j < n_a ? 2 * j + g : n_a + j; };

  if (threadIdx.x == 0) {
    ptx::mbar_init(&bars->q_full, 1);
    for (int s = 0; s < kRing; ++s) {
      ptx::mbar_init(&bars->kv_full[s], 1);
      ptx::mbar_init(&bars->kv_empty[s], 1);
    }
    for (int b = 0; b < kBuffers; ++b) {
      ptx::mbar_init(&bars->s_full[b], 1);
      ptx::mbar_init(&bars->p_ready[b], 128);
      ptx::mbar_init(&bars->buf_free[b], 1);
    }
    for (int g = 0; g < 2; ++g)
      for (int e = 0; e < 2; ++e) ptx::mbar_init(&bars->pv_done[g][e], 1);
    bars->abort_flag = 0;
    ptx::fence_mbar_init();
  }
  if (warp == 9) {
    ptx::tmem_alloc(&bars->tmem_base, kTmemCols);
    ptx::tmem_relinquish_alloc_permit();
  }
  ptx::tcgen05_fence_before_thread_sync();
  __syncthreads();
  ptx::tcgen05_fence_after_thread_sync();
  const uint32_t tmem_base = bars->tmem_base;
  ptx::launch_dependents();
  ptx::wait_prior_grid();

  if (warp == 8) {
    // ------------------------------ TMA producer ------------------------------
    ptx::setmaxnreg_dec<kRegsOther>();
    if (lane == 0) {
      ptx::mbar_arrive_expect_tx(&bars->q_full, 2 * kTileBytes);
#pragma unroll
      for (int g = 0; g < 2; ++g) ptx::tma_load_3d(smem + g * kTileBytes, &tmap_q, &bars->q_full, 0, q0 + g * kBQ, bh);
      // ring order = the order the tensor core first needs the tiles in: K_0, K_1, V_0, K_2, V_1, ..., K_{n-1}, V_{n-2}, V_{n-1}
      const int total = 2 * n_b;
      for (int idx = 0; idx < total; ++idx) {
        const int slot = idx % kRing;
        if (!ptx::mbar_wait(&bars->kv_empty[slot], ((idx / kRing) & 1u) ^ 1u, abort_flag, p.status, 101)) break;
        ptx::mbar_arrive_expect_tx(&bars->kv_full[slot], kTileBytes);
        const bool is_v = idx == total - 1 || (idx >= 2 && (idx & 1) == 0);
        const int step = idx == 0 ? 0 : idx == total - 1 ? n_b - 1 : is_v ? (idx >> 1) - 1 : (idx + 1) >> 1;
        ptx::tma_load_3d(smem_kv + slot * kTileBytes, is_v ? &tmap_v : &tmap_k, &bars->kv_full[slot], 0, (j0 + step) * kBKV, kvh);
      }
    }
  } else if (warp == 9 || warp == 10) {
    // ------------------------------ MMA issuers --------------------------------
    ptx::setmaxnreg_dec<kRegsOther>();
    constexpr uint64_t kmajor = ptx::make_smem_desc_base(16, 1024);
    constexpr uint64_t v_mnmajor = ptx::make_smem_desc_base(kTileBytes, 1024);
    constexpr uint32_t k_hi = static_cast<uint32_t>(kmajor >> 32), v_hi = static_cast<uint32_t>(v_mnmajor >> 32);
    constexpr uint32_t k_lo = static_cast<uint32_t>(kmajor), v_lo = static_cast<uint32_t>(v_mnmajor);
    auto desc = [](uint32_t hi, uint32_t lo) -> uint64_t { return (static_cast<uint64_t>(hi) << 32) | lo; };
    // ring positions of the tiles (see the producer)
    auto k_pos = [&](int j) { return j == 0 ? 0 : 2 * j - 1; };
    auto v_pos = [&](int j) { return j == n_b - 1 ? 2 * n_b - 1 : 2 * j + 2; };
    auto wait_kv = [&](int idx) -> bool {
      const bool r = ptx::mbar_wait_relaxed(&bars->kv_full[idx % kRing], (idx / kRing) & 1u, abort_flag, p.status, 102);
      return __all_sync(0xffffffffu, r);  // the warp stays converged, also when a wait gives up
    };
    if (warp == 9) {
      constexpr uint32_t idesc = ptx::make_idesc_f16(kBQ, kBKV, false, false, kIsBf16);
      const uint32_t q_lo = k_lo | (ptx::smem_u32(smem) >> 4), ring_lo = k_lo | (ptx::smem_u32(smem_kv) >> 4);
      bool ok = __all_sync(0xffffffffu, ptx::mbar_wait_relaxed(&bars->q_full, 0, abort_flag, p.status, 103));
      for (int j = 0; j < n_b && ok; ++j) {
        if (!(ok = wait_kv(k_pos(j)))) break;
        const uint32_t b_lo = ring_lo + (k_pos(j) % kRing) * (kTileBytes >> 4);
#pragma unroll
        for (int g = 0; g < 2; ++g) {
          if (g == 0 ? j >= n_a : lone) continue;
          const int q = job(g, j), buf = q % kBuffers, use = q / kBuffers;
          // the product of the job that had this buffer has read it
          if (use > 0) ok = __all_sync(0xffffffffu, ptx::mbar_wait_relaxed(&bars->buf_free[buf], (use - 1) & 1u, abort_flag, p.status, 104));
          if (!ok) break;
          ptx::tcgen05_fence_after_thread_sync();
          if (ptx::elect_one_sync()) {
#pragma unroll
            for (int kk = 0; kk < kD / 16; ++kk)
              ptx::tcgen05_mma_f16_ss(tmem_base + buf * 128, desc(k_hi, q_lo + g * (kTileBytes >> 4) + kk * 2), desc(k_hi, b_lo + kk * 2), idesc,
                                      kk != 0 ? 1u : 0u);
            ptx::tcgen05_commit(&bars->s_full[buf]);
            if (g == 1 || lone) ptx::tcgen05_commit(&bars->kv_empty[k_pos(j) % kRing]);  // last reader of K_j
          }
          __syncwarp();
        }
      }
    } else {
      constexpr uint32_t idesc = ptx::make_idesc_f16(kBQ, kD, false, true, kIsBf16);
      const uint32_t ring_lo = v_lo | (ptx::smem_u32(smem_kv) >> 4);
      bool ok = true;
      for (int j = 0; j < n_b && ok; ++j) {
        if (!(ok = wait_kv(v_pos(j)))) break;
        const uint32_t b_lo = ring_lo + (v_pos(j) % kRing) * (kTileBytes >> 4);
#pragma unroll
        for (int g = 0; g < 2; ++g) {
          if (g == 0 ? j >= n_a : lone) continue;
          const int q = job(g, j), buf = q % kBuffers;
          ok = __all_sync(0xffffffffu, ptx::mbar_wait(&bars->p_ready[buf], (q / kBuffers) & 1u, abort_flag, p.status, 105));
          if (!ok) break;
          ptx::tcgen05_fence_after_thread_sync();
          const uint32_t d = tmem_base + kTmemO + g * kD, a = tmem_base + buf * 128;
          if (ptx::elect_one_sync()) {
#pragma unroll
            for (int kk = 0; kk < kBKV / 16; ++kk) {
              const uint64_t b = desc(v_hi, b_lo + kk * (2048 >> 4));
              ptx::tcgen05_mma_f16_ts(d, a + kk * 8, b, idesc, (j > 0 || kk != 0) ? 1u : 0u);
              ptx::tcgen05_mma_f16_ts(d, a + 64 + kk * 8, b, idesc, 1u);
            }
            ptx::tcgen05_commit(&bars->buf_free[buf]);
            ptx::tcgen05_commit(&bars->pv_done[g][j & 1]);
            if (g == 1 || lone) ptx::tcgen05_commit(&bars->kv_empty[v_pos(j) % kRing]);  // last reader of V_j
          }
          __syncwarp();
        }
      }
    }
  } else if (warp == 11) {
    ptx::setmaxnreg_dec<kRegsOther>();
  } else {
    // ------------------------------ softmax / output ---------------------------
    ptx::setmaxnreg_inc<kRegsSoftmax>();
    const int g = warp >> 2;                // 0: tile A, 1: tile B
    const int quad = warp & 3;              // tensor-memory lanes this warp may touch
    const int r = quad * 32 + lane;         // row inside the tile == lane
    const int n_g = g == 0 ? n_a : lone ? 0 : n_b;
    const int qrow = q0 + g * kBQ + r;
    const int limit = p.causal ? min(qrow + q_off, seq_kv - 1) : (seq_kv - 1);  // last visible column
    const uint32_t lane_base = tmem_base + (static_cast<uint32_t>(quad * 32) << 16);
    const uint32_t to = lane_base + kTmemO + g * kD;
    const float sl2 = p.scale_log2;

    float m_used = -INFINITY;  // running max in raw score units
    float l = 0.f;
    bool alive = true;
    for (int j = 0; j < n_g; ++j) {
      const int q = job(g, j), buf = q % kBuffers;
      const uint32_t ts = lane_base + buf * 128;
      bool ready = ptx::mbar_wait(&bars->s_full[buf], (q / kBuffers) & 1u, abort_flag, p.status, 106 + g);
      if (!__all_sync(0xffffffffu, ready)) {
        alive = false;
        break;
      }
      ptx::tcgen05_fence_after_thread_sync();
      const int col0 = (j0 + j) * kBKV;

      // the whole score row of this step, read once: the probabilities will take its place
      uint32_t v[4][32];
#pragma unroll
      for (int c = 0; c < 4; ++c) ptx::tmem_ld_32x32b_x32(ts + c * 32, v[c]);
      ptx::tmem_ld_wait();

      float mx = -INFINITY;
      if (col0 + kBKV - 1 > limit) {
#pragma unroll
        for (int c = 0; c < 4; ++c)
#pragma unroll
          for (int i = 0; i < 32; ++i) {
            if (col0 + c * 32 + i > limit) v[c][i] = 0xff800000u;  // -inf
            mx = fmaxf(mx, __uint_as_float(v[c][i]));
          }
      } else {
        float mx4[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
        for (int c = 0; c < 4; ++c)
#pragma unroll
          for (int i = 0; i < 32; i += 2)  // three-input max: 64 instructions for 128 values
            mx4[(i >> 1) & 3] = ptx::fmax3(mx4[(i >> 1) & 3], __uint_as_float(v[c][i]), __uint_as_float(v[c][i + 1]));
        mx = fmaxf(fmaxf(mx4[0], mx4[1]), fmaxf(mx4[2], mx4[3]));
      }
      // the running max is raised only when it grows by more than 2^8; O is rescaled then
      const float m_new = fmaxf(m_used, mx);
      if (j == 0) {
        m_used = m_new;
      } else {
        const bool need = (m_new - m_used) * sl2 > attn::kRescaleThreshold;
        if (__any_sync(0xffffffffu, need)) {
          // once the previous step's product has retired (the next one is not issued before this step's probabilities are handed over)
          ready = ptx::mbar_wait(&bars->pv_done[g][(j - 1) & 1], ((j - 1) >> 1) & 1u, abort_flag, p.status, 108 + g);
          if (!__all_sync(0xffffffffu, ready)) {
            alive = false;
            break;
          }
          ptx::tcgen05_fence_after_thread_sync();
          const float alpha = need ? ptx::ex2_approx((m_used - m_new) * sl2) : 1.0f;
          if (need) m_used = m_new;
          l *= alpha;
#pragma unroll 1
          for (int c = 0; c < kD / 32; ++c) {
            uint32_t ov[32];
            ptx::tmem_ld_32x32b_x32(to + c * 32, ov);
            ptx::tmem_ld_wait();
#pragma unroll
            for (int i = 0; i < 32; ++i) ov[i] = __float_as_uint(__uint_as_float(ov[i]) * alpha);
            ptx::tmem_st_32x32b_x32(to + c * 32, ov);
          }
        }
      }

      // Probabilities, 64 keys at a time: hi = p rounded to the storage type, lo = p - hi rounded again; the row sum adds the f32 values.
      // A row whose scores so far are all -inf (a step, or in kSplit a whole range, may lie behind the row's last visible key):
      // taking them against 0 gives them no weight, against their maximum of -inf NaN.
      const float ms = m_used == -INFINITY ? 0.f : m_used * sl2 - kPShift<kIsBf16>;
      const ptx::f32x2_t sl2x2 = ptx::pack_f32x2(sl2, sl2);
      const ptx::f32x2_t nmsx2 = ptx::pack_f32x2(-ms, -ms);
      ptx::f32x2_t lsum[2] = {0ull, 0ull};
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        uint32_t hi[32], lo[32];
#pragma unroll
        for (int i = 0; i < 32; ++i) {
          const int c = 2 * h + (i >> 4), e = (i & 15) * 2;
          const ptx::f32x2_t t2 =
              ptx::fma_f32x2(ptx::pack_f32x2(__uint_as_float(v[c][e]), __uint_as_float(v[c][e + 1])), sl2x2, nmsx2);
          float t0, t1;
          ptx::unpack_f32x2(t2, t0, t1);
          const float p0 = ptx::ex2_approx(t0), p1 = ptx::ex2_approx(t1);  // 2^(-inf) = 0
          const ptx::f32x2_t p2 = ptx::pack_f32x2(p0, p1);
          hi[i] = attn::pack16x2<kIsBf16>(p0, p1);
          float d0, d1;
          ptx::unpack_f32x2(ptx::fma_f32x2(ptx::pack_f32x2(attn::unpack16_lo<kIsBf16>(hi[i]), attn::unpack16_hi<kIsBf16>(hi[i])),
                                           ptx::pack_f32x2(-1.0f, -1.0f), p2), d0, d1);
          lo[i] = attn::pack16x2<kIsBf16>(d0, d1);
          lsum[i & 1] = ptx::add_f32x2(lsum[i & 1], p2);
        }
        ptx::tmem_st_32x32b_x32(ts + h * 32, hi);
        ptx::tmem_st_32x32b_x32(ts + 64 + h * 32, lo);
      }
      float l4[4];
      ptx::unpack_f32x2(lsum[0], l4[0], l4[1]);
      ptx::unpack_f32x2(lsum[1], l4[2], l4[3]);
      l += (l4[0] + l4[1]) + (l4[2] + l4[3]);
      ptx::tmem_st_wait();
      ptx::tcgen05_fence_before_thread_sync();  // probabilities, and a rescaled O, are ordered before the arrival
      ptx::mbar_arrive(&bars->p_ready[buf]);
    }

    if (kSplit && g == 1 && lone) {
      // nobody reads the records of rows that do not exist
    } else if constexpr (kSplit) {
      bool have = alive && n_g > 0;  // a range may be empty for this tile: weight 0, O zero
      if (have) have = __all_sync(0xffffffffu, ptx::mbar_wait(&bars->pv_done[g][(n_g - 1) & 1], ((n_g - 1) >> 1) & 1u, abort_flag, p.status, 110 + g));
      ptx::tcgen05_fence_after_thread_sync();
      const int64_t rec = static_cast<int64_t>(block) * splits + rank;
      const int row = g * kBQ + r;
      float4* part = p.part + rec * (kD / 4) * (2 * kBQ) + row;
#pragma unroll 1
      for (int c = 0; c < kD / 32; ++c) {
        uint32_t ov[32];
        ptx::tmem_ld_32x32b_x32(to + c * 32, ov);
        ptx::tmem_ld_wait();
#pragma unroll
        for (int i = 0; i < 8; ++i)
          part[(c * 8 + i) * (2 * kBQ)] =
              have ? make_float4(__uint_as_float(ov[4 * i]), __uint_as_float(ov[4 * i + 1]), __uint_as_float(ov[4 * i + 2]), __uint_as_float(ov[4 * i + 3]))
                   : make_float4(0.f, 0.f, 0.f, 0.f);
      }
      p.part_ml[rec * (2 * kBQ) + row] = have ? make_float2(m_used, l) : make_float2(-INFINITY, 0.f);
    } else if (alive && n_g > 0) {
      const bool ready = ptx::mbar_wait(&bars->pv_done[g][(n_g - 1) & 1], ((n_g - 1) >> 1) & 1u, abort_flag, p.status, 112 + g);
      if (__all_sync(0xffffffffu, ready)) {
        ptx::tcgen05_fence_after_thread_sync();
        // all scores -inf (or NaN): softmax is NaN there
        const float inv = m_used == -INFINITY ? NAN : 1.0f / l;
        const int cols = p.head_dim;
        uint16_t* orow = kCache ? o + bh * p.o_head_stride + qrow * p.o_row_stride
                                : o + (static_cast<int64_t>(bh) * p.seq + qrow) * cols;
#pragma unroll 1
        for (int c = 0; c < kD / 32; ++c) {
          uint32_t ov[32];
          ptx::tmem_ld_32x32b_x32(to + c * 32, ov);
          ptx::tmem_ld_wait();
          if (qrow < p.seq) {
#pragma unroll
            for (int t = 0; t < 4; ++t) {
              uint4 w;
              w.x = attn::pack16x2<kIsBf16>(__uint_as_float(ov[8 * t + 0]) * inv, __uint_as_float(ov[8 * t + 1]) * inv);
              w.y = attn::pack16x2<kIsBf16>(__uint_as_float(ov[8 * t + 2]) * inv, __uint_as_float(ov[8 * t + 3]) * inv);
              w.z = attn::pack16x2<kIsBf16>(__uint_as_float(ov[8 * t + 4]) * inv, __uint_as_float(ov[8 * t + 5]) * inv);
              w.w = attn::pack16x2<kIsBf16>(__uint_as_float(ov[8 * t + 6]) * inv, __uint_as_float(ov[8 * t + 7]) * inv);
              if (c * 32 + t * 8 < cols) reinterpret_cast<uint4*>(orow + c * 32)[t] = w;
            }
          }
        }
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
    ptx::tmem_dealloc(tmem_base, kTmemCols);
  }
}

}  // namespace attn_narrow
}  // namespace tsm100
