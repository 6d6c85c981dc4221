// Fused attention forward for f32 tensors on the 5th-generation tensor cores (tcgen05, kind::f16), f32-grade results.
//
// Semantics as attention_tf32x3.cuh (__tile_attention_f32, crates/tile_std/src/tile.rs:218-224;
// crates/rustc_codegen_tile/src/mlir_to_linalg.rs:1781-1902, :1191-1244; grouped heads
// crates/rustc_codegen_tile/src/mlir_to_gpu.rs:1657-1673).  Every operand, Q, K, V and the probabilities, is split into three bf16 numbers, 24 bits
// together, and six of the nine products are taken.
//
// One streaming launch writes the parts of K and of V, each as planes [3][heads][keys][D]; V is read MN-major as it lies.  Then one CTA owns 128
// query rows of one head and walks the keys in steps of 64:
//   warp 8       TMA producer: K_0, K_1, V_0, K_2, V_1, ... (three parts together, 384 * D bytes a unit) through a ring.  No multicast.
//   warp 9       S = Q K^T, the parts of Q in tensor memory for the CTA's life.
//   warp 10      O = P V of one step, from zero: the tensor core rounds its accumulator toward zero, and what that costs grows with what it holds.
//   warps 0..3   softmax, one thread per query row; the parts of the probabilities take the place of the scores they were made from.
//   warps 4..7   drain: the O of a step is added, round to nearest, to running sums in registers (D per thread), scaled by how far the
//                step's maximum has grown.
// Tensor memory at D = 128: 3 * 64 columns of Q, two buffers of 96 for scores (64) and then probabilities (3 * 32), 128 of O: all 512.  A step's softmax
// runs during the scores of the next, and the drain too, so one O is enough.
// Bound: the tensor pipe, 3072 cycles a step (48 products of 128 x 64 x 16, 24 of 128 x 128 x 16), and the board's power: 16 heads of 4096 x 128, causal,
// 297 us at 1.6 GHz, 475 K cycles of which 350 K are products, and 26 us for the parts of K and V; 363 us a call in a row (189 TFLOP/s), 2.2e-7 off the
// 64-bit result.  The form before this one took three products of two TF32 numbers in steps of 32 keys, whose scores spend most of a product on
// reading Q, and wrote a third more for the parts, V transposed: 450 us, 9e-7; 2 heads of 1283 70 us, 48 here, 256 heads of 530 242 / 182.
// Tiny operands and probabilities keep their bits (split2): V of 1e-36 2.9e-7 off, of 1e-37 1.5e-6, of 1e-38 1.5e-5 (two TF32 numbers 3.4e-6, 3.3e-5 and
// 3.4e-4, three bf16 numbers as they are 2.7e-5, 2.7e-4 and 2.7e-3).  That takes 0.1 % of the cycles, 2 % with heads of 32, where the softmax is the longer part.
#pragma once

#include "attention_simt.cuh"    // Params
#include "attention_tc.cuh"      // pack16x2
#include "ptx.cuh"

namespace tsm100 {
namespace attn_f32_tc {

constexpr int kBQ = 128;           // query rows per CTA
constexpr int kBKV = 64;           // keys per step
constexpr int kThreads = 384;
constexpr int kRegsOther = 56, kRegsSoftmax = 200, kRegsDrain = 224;
static_assert(128 * (kRegsOther + kRegsSoftmax + kRegsDrain) <= kThreads * 168, "setmaxnreg draws on the launch's registers");
constexpr int kTmemCols = 512;
constexpr int kTmemQ = 0, kQPart = 64, kTmemS = 192, kBuffer = 96, kPPart = 32, kTmemO = 384;
// its bounded waits report sites 71 .. 83

template <int D>
struct Shape {
  static constexpr int kGroup = D % 64 == 0 ? 64 : 32;   // columns of a swizzled row
  static constexpr int kRow = kGroup * 2;                // bytes: the swizzle
  static constexpr int kGroups = D / kGroup;
  static constexpr int kGroupBytes = kBKV * kRow;
  static constexpr int kPart = kBKV * D * 2;             // one part of 64 rows of K or V
  static constexpr int kUnitBytes = 3 * kPart;
  static constexpr int kRing = D == 128 ? 4 : D == 96 ? 5 : 8;
  static constexpr int kRowsOff = kRing * kUnitBytes;    // float [3][128]: per step, the maximum it is scaled by
  static constexpr int kBarsOff = kRowsOff + 3 * kBQ * 4;
};
constexpr int kMaxRing = 8;
struct alignas(8) Barriers {
  uint64_t q_ready;
  uint64_t kv_full[kMaxRing], kv_empty[kMaxRing];
  uint64_t s_full[2];     // the scores of a step are in its buffer
  uint64_t p_ready[2];    // its probabilities have taken their place
  uint64_t buf_free[2];   // its product has read them
  uint64_t o_full, o_empty;
  uint64_t m_ready[3];    // the maximum of a step is in its row slot
  uint64_t l_ready;       // the row sums are in the slot after the last step's
  uint32_t tmem_base;
  uint32_t abort_flag;
};
template <int D>
constexpr int smem_bytes() {
  return Shape<D>::kBarsOff + static_cast<int>(sizeof(Barriers)) + 1024;
}
static_assert(smem_bytes<128>() <= 227 * 1024 && smem_bytes<96>() <= 227 * 1024 && smem_bytes<64>() <= 227 * 1024, "shared memory budget of one CTA");

struct Params {
  attn_simt::Params a;      // shapes, and the strides of Q and O
  uint32_t* status;
};

// Two values as three pairs of bf16 numbers: hi truncated (the largest f32 numbers would round up to infinity), mid what is left of them rounded to nearest,
// lo 2^kLoShift times the rest, which has 8 bits or less.  Unscaled, it would end below the last bit that a bf16 number has, 2^-133, for values below
// 1e-34; this way bits from 2^-142 on are kept.  lo stays smaller than hi, and sums of products with it than those of hi.
// kPairs: lo by packed instructions.  The attention kernel spends 0.8 % more cycles without them (16 heads of 4096 x 128, the probabilities), the split pass 3 % more with.
constexpr int kLoShift = 10;
template <bool kPairs>
__device__ __forceinline__ void split2(float x0, float x1, uint32_t& hi, uint32_t& mid, uint32_t& lo) {
  constexpr float kUp = 1 << kLoShift;
  const uint32_t b0 = __float_as_uint(x0), b1 = __float_as_uint(x1);
  hi = __byte_perm(b0, b1, 0x7632);
  const float r0 = x0 - __uint_as_float(b0 & 0xffff0000u), r1 = x1 - __uint_as_float(b1 & 0xffff0000u);
  mid = attn::pack16x2<true>(r0, r1);
  float l0, l1;
  if constexpr (kPairs) {
    const ptx::f32x2_t m = ptx::pack_f32x2(attn::unpack16_lo<true>(mid), attn::unpack16_hi<true>(mid));
    const ptx::f32x2_t l = ptx::fma_f32x2(m, ptx::pack_f32x2(-1.0f, -1.0f), ptx::pack_f32x2(r0, r1));
    ptx::unpack_f32x2(ptx::mul_f32x2(l, ptx::pack_f32x2(kUp, kUp)), l0, l1);
  } else {
    l0 = (r0 - attn::unpack16_lo<true>(mid)) * kUp, l1 = (r1 - attn::unpack16_hi<true>(mid)) * kUp;
  }
  lo = __byte_perm(__float_as_uint(l0), __float_as_uint(l1), 0x7632);
}

// The parts of K and of V, bf16 [3][heads][rows * D]: grid (blocks, heads, 2), a thread per eight values.
struct SplitParams {
  const float* src[2];
  uint16_t* dst[2];
  int64_t head_stride;      // of src, in elements
  int64_t head_vecs;        // rows * D / 8
};
__global__ void __launch_bounds__(256)
split_kv_kernel(const SplitParams p) {
  ptx::launch_dependents_if_few();
  const int which = static_cast<int>(blockIdx.z);
  const int64_t head = blockIdx.y, part = p.head_vecs * gridDim.y;
  const float4* src = reinterpret_cast<const float4*>(ptx::wait_prior_grid((which ? p.src[1] : p.src[0]) + head * p.head_stride));
  uint4* dst = reinterpret_cast<uint4*>(which ? p.dst[1] : p.dst[0]) + head * p.head_vecs;
  const int64_t step = static_cast<int64_t>(gridDim.x) * blockDim.x;
  for (int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < p.head_vecs; i += step) {
    const float4 x = __ldcs(src + 2 * i), y = __ldcs(src + 2 * i + 1);
    uint32_t hi[4], mid[4], lo[4];
    split2<false>(x.x, x.y, hi[0], mid[0], lo[0]);
    split2<false>(x.z, x.w, hi[1], mid[1], lo[1]);
    split2<false>(y.x, y.y, hi[2], mid[2], lo[2]);
    split2<false>(y.z, y.w, hi[3], mid[3], lo[3]);
    dst[i] = make_uint4(hi[0], hi[1], hi[2], hi[3]);
    dst[i + part] = make_uint4(mid[0], mid[1], mid[2], mid[3]);
    dst[i + 2 * part] = make_uint4(lo[0], lo[1], lo[2], lo[3]);
  }
}

// What a product does with the accumulator: overwrites it, adds to it, or adds to it after bringing it down from the scale of lo.
enum Start { kFresh, kAdd, kDown };
__device__ __forceinline__ void product(uint32_t d, uint32_t a, uint64_t b_desc, uint32_t idesc, Start start) {
  if (start == kDown) ptx::tcgen05_mma_f16_ts_scaled<kLoShift>(d, a, b_desc, idesc);
  else ptx::tcgen05_mma_f16_ts(d, a, b_desc, idesc, start == kFresh ? 0u : 1u);
}
// The six products of the parts, the small ones first: the accumulator cuts every term off at its own last place.
template <typename F>
__device__ __forceinline__ void all_products(F products) {
  products(2, 0, kFresh);
  products(0, 2, kAdd);
  products(1, 1, kDown);
  products(1, 0, kAdd);
  products(0, 1, kAdd);
  products(0, 0, kAdd);
}

template <int D>
__global__ void __launch_bounds__(kThreads, 1)
attention_f32_tc_kernel(const __grid_constant__ CUtensorMap tmap_k, const __grid_constant__ CUtensorMap tmap_v, const float* __restrict__ q,
                        float* __restrict__ o, const Params pp) {
  using Sh = Shape<D>;
  constexpr int kRing = Sh::kRing;
  const attn_simt::Params& p = pp.a;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
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
  const int all_kv = p.batch * p.heads_kv;
  const int n_all = (p.seq_kv + kBKV - 1) / kBKV;
  const int n = p.causal ? min(n_all, (min(q0 + kBQ, p.seq) - 1 + p.q_offset) / kBKV + 1) : n_all;  // steps, >= 1

  if (threadIdx.x == 0) {
    ptx::mbar_init(&bars->q_ready, 128);
    for (int s = 0; s < kRing; ++s) {
      ptx::mbar_init(&bars->kv_full[s], 1);
      ptx::mbar_init(&bars->kv_empty[s], 1);
    }
    for (int i = 0; i < 2; ++i) {
      ptx::mbar_init(&bars->s_full[i], 1);
      ptx::mbar_init(&bars->p_ready[i], 128);
      ptx::mbar_init(&bars->buf_free[i], 1);
    }
    ptx::mbar_init(&bars->o_full, 1);
    ptx::mbar_init(&bars->o_empty, 128);
    for (int i = 0; i < 3; ++i) ptx::mbar_init(&bars->m_ready[i], 128);
    ptx::mbar_init(&bars->l_ready, 128);
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
  const uint32_t tmem = bars->tmem_base;
  ptx::wait_prior_grid();
  // ring positions: K_0, K_1, V_0, K_2, V_1, ..., K_{n-1}, V_{n-2}, V_{n-1}
  auto k_pos = [&](int j) { return j == 0 ? 0 : 2 * j - 1; };
  auto v_pos = [&](int j) { return j == n - 1 ? 2 * n - 1 : 2 * j + 2; };

  // Q, split, to tensor memory (warps 0..3, one row each)
  if (warp < 4) {
    const int r = warp * 32 + lane;
    const bool valid = q0 + r < p.seq;
    const float4* qr = reinterpret_cast<const float4*>(q + bh * p.q_head_stride + (q0 + r) * p.q_row_stride);
    const uint32_t tq = tmem + (static_cast<uint32_t>(warp * 32) << 16) + kTmemQ;
#pragma unroll
    for (int c = 0; c < D / 32; ++c) {
      uint32_t hi[16], mid[16], lo[16];
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        const float4 x = valid ? qr[c * 8 + u] : make_float4(0.f, 0.f, 0.f, 0.f);
        split2<true>(x.x, x.y, hi[2 * u], mid[2 * u], lo[2 * u]);
        split2<true>(x.z, x.w, hi[2 * u + 1], mid[2 * u + 1], lo[2 * u + 1]);
      }
      __syncwarp();
      ptx::tmem_st_32x32b_x16(tq + c * 16, hi);
      ptx::tmem_st_32x32b_x16(tq + kQPart + c * 16, mid);
      ptx::tmem_st_32x32b_x16(tq + 2 * kQPart + c * 16, lo);
    }
    ptx::tmem_st_wait();
    ptx::tcgen05_fence_before_thread_sync();
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
        uint8_t* dst = smem + slot * Sh::kUnitBytes;
        const CUtensorMap* map = is_v ? &tmap_v : &tmap_k;
#pragma unroll
        for (int part = 0; part < 3; ++part)
#pragma unroll
          for (int c = 0; c < Sh::kGroups; ++c)
            ptx::tma_load_3d(dst + part * Sh::kPart + c * Sh::kGroupBytes, map, &bars->kv_full[slot], c * Sh::kGroup, step * kBKV, part * all_kv + kvh);
      }
    }
  } else if (warp == 9 || warp == 10) {
    // ------------------------------ MMA issuers --------------------------------
    ptx::setmaxnreg_dec<kRegsOther>();
    constexpr uint64_t swizzle = Sh::kRow == 128 ? ptx::kSwizzle128B : ptx::kSwizzle64B;
    constexpr uint64_t k_base = ptx::make_smem_desc_base(16, 8 * Sh::kRow, swizzle);
    constexpr uint64_t v_base = ptx::make_smem_desc_base(Sh::kGroupBytes, 8 * Sh::kRow, swizzle);
    auto wait_kv = [&](int idx) -> bool {
      const bool r = ptx::mbar_wait_relaxed(&bars->kv_full[idx % kRing], (idx / kRing) & 1u, abort_flag, status, 72);
      return __all_sync(0xffffffffu, r);
    };
    auto desc = [](uint64_t base, uint32_t lo) -> uint64_t { return (base & 0xffffffff00000000ull) | lo; };
    const uint32_t ring16 = ptx::smem_u32(smem) >> 4;
    constexpr uint32_t kPart16 = Sh::kPart >> 4;
    bool ok = true;
    if (warp == 9) {
      constexpr uint32_t idesc = ptx::make_idesc_f16(kBQ, kBKV, false, false, true);
      ok = __all_sync(0xffffffffu, ptx::mbar_wait(&bars->q_ready, 0, abort_flag, status, 73));
      for (int j = 0; j < n && ok; ++j) {
        const int b = j & 1;
        if (!(ok = wait_kv(k_pos(j)))) break;
        // the product of step j - 2 has read the probabilities in this buffer
        if (j >= 2 && !(ok = __all_sync(0xffffffffu, ptx::mbar_wait_relaxed(&bars->buf_free[b], ((j - 2) >> 1) & 1u, abort_flag, status, 74)))) break;
        ptx::tcgen05_fence_after_thread_sync();
        const uint32_t d = tmem + kTmemS + b * kBuffer, a = tmem + kTmemQ;
        const uint32_t k_lo = static_cast<uint32_t>(k_base) | (ring16 + (k_pos(j) % kRing) * (Sh::kUnitBytes >> 4));
        if (ptx::elect_one_sync()) {
          auto products = [&](int x, int y, Start start) {
#pragma unroll
            for (int kk = 0; kk < D / 16; ++kk) {
              constexpr int kPerGroup = Sh::kGroup / 16;
              const uint32_t off = y * kPart16 + (kk / kPerGroup) * (Sh::kGroupBytes >> 4) + (kk % kPerGroup) * 2;
              product(d, a + x * kQPart + kk * 8, desc(k_base, k_lo + off), idesc, kk == 0 ? start : kAdd);
            }
          };
          all_products(products);
          ptx::tcgen05_commit(&bars->s_full[b]);
          ptx::tcgen05_commit(&bars->kv_empty[k_pos(j) % kRing]);
        }
        __syncwarp();
      }
    } else {
      constexpr uint32_t idesc = ptx::make_idesc_f16(kBQ, D, false, true, true);
      for (int j = 0; j < n && ok; ++j) {
        const int b = j & 1;
        if (!(ok = wait_kv(v_pos(j)))) break;
        if (j >= 1 && !(ok = __all_sync(0xffffffffu, ptx::mbar_wait_relaxed(&bars->o_empty, (j - 1) & 1u, abort_flag, status, 76)))) break;
        if (!(ok = __all_sync(0xffffffffu, ptx::mbar_wait(&bars->p_ready[b], (j >> 1) & 1u, abort_flag, status, 77)))) break;
        ptx::tcgen05_fence_after_thread_sync();
        const uint32_t d = tmem + kTmemO, a = tmem + kTmemS + b * kBuffer;
        const uint32_t v_lo = static_cast<uint32_t>(v_base) | (ring16 + (v_pos(j) % kRing) * (Sh::kUnitBytes >> 4));
        if (ptx::elect_one_sync()) {
          auto products = [&](int x, int y, Start start) {
#pragma unroll
            for (int kk = 0; kk < kBKV / 16; ++kk)
              product(d, a + x * kPPart + kk * 8, desc(v_base, v_lo + y * kPart16 + kk * (16 * Sh::kRow >> 4)), idesc, kk == 0 ? start : kAdd);
          };
          all_products(products);
          ptx::tcgen05_commit(&bars->buf_free[b]);
          ptx::tcgen05_commit(&bars->o_full);
          ptx::tcgen05_commit(&bars->kv_empty[v_pos(j) % kRing]);
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
      const uint32_t ts = lane_base + kTmemS + b * kBuffer;
      if (!__all_sync(0xffffffffu, ptx::mbar_wait(&bars->s_full[b], (j >> 1) & 1u, abort_flag, status, 78))) {
        alive = false;
        break;
      }
      ptx::tcgen05_fence_after_thread_sync();
      uint32_t v[2][32];
      ptx::tmem_ld_32x32b_x32(ts, v[0]);
      ptx::tmem_ld_32x32b_x32(ts + 32, v[1]);
      ptx::tmem_ld_wait();
      const int key0 = j * kBKV;
      if (key0 + kBKV - 1 > limit) {
#pragma unroll
        for (int h = 0; h < 2; ++h)
#pragma unroll
          for (int i = 0; i < 32; ++i)
            if (key0 + h * 32 + i > limit) v[h][i] = 0xff800000u;  // -inf
      }
      float mx4[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
      for (int i = 0; i < 64; i += 2)
        mx4[(i >> 1) & 3] = ptx::fmax3(mx4[(i >> 1) & 3], __uint_as_float(v[i >> 5][i & 31]), __uint_as_float(v[i >> 5][(i & 31) + 1]));
      const float m_new = fmaxf(m_used, fmaxf(fmaxf(mx4[0], mx4[1]), fmaxf(mx4[2], mx4[3])));
      // nothing of this step is in tensor memory yet; the drain warps rescale their sums
      if (m_new != m_used) {
        l *= ptx::ex2_approx((m_used - m_new) * sl2);  // l = 0 while m_used = -inf
        m_used = m_new;
      }
      // a row that has seen nothing but -inf so far: probabilities 0, not NaN
      const float nms = m_used == -INFINITY ? 0.f : -m_used * sl2;
      const ptx::f32x2_t sl2x2 = ptx::pack_f32x2(sl2, sl2), nmsx2 = ptx::pack_f32x2(nms, nms);
      ptx::f32x2_t ls[2] = {0ull, 0ull};
      // The parts of the probabilities take the place of the scores.
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        uint32_t hi[16], mid[16], lo[16];
#pragma unroll
        for (int i = 0; i < 16; ++i) {
          float t0, t1;
          ptx::unpack_f32x2(ptx::fma_f32x2(ptx::pack_f32x2(__uint_as_float(v[h][2 * i]), __uint_as_float(v[h][2 * i + 1])), sl2x2, nmsx2), t0, t1);
          const float e0 = ptx::ex2_approx(t0), e1 = ptx::ex2_approx(t1);
          ls[i & 1] = ptx::add_f32x2(ls[i & 1], ptx::pack_f32x2(e0, e1));
          split2<true>(e0, e1, hi[i], mid[i], lo[i]);
        }
        ptx::tmem_st_32x32b_x16(ts + h * 16, hi);
        ptx::tmem_st_32x32b_x16(ts + kPPart + h * 16, mid);
        ptx::tmem_st_32x32b_x16(ts + 2 * kPPart + h * 16, lo);
      }
      float l4[4];
      ptx::unpack_f32x2(ls[0], l4[0], l4[1]);
      ptx::unpack_f32x2(ls[1], l4[2], l4[3]);
      l += (l4[0] + l4[1]) + (l4[2] + l4[3]);
      ptx::tmem_st_wait();
      ptx::tcgen05_fence_before_thread_sync();
      ptx::mbar_arrive(&bars->p_ready[b]);
      // slot j % 3: the scores of step j were issued after the product of step j - 2 had retired, which was issued after step j - 3 was drained
      row_slot[j % 3 * kBQ + r] = m_used;
      ptx::mbar_arrive(&bars->m_ready[j % 3]);
    }
    // the row sum takes the slot after the last step's, once the last product has retired: by then step n - 3, which had it, is drained
    // (the product of step n - 1 was issued after step n - 2 was)
    if (alive && __all_sync(0xffffffffu, ptx::mbar_wait(&bars->buf_free[(n - 1) & 1], ((n - 1) >> 1) & 1u, abort_flag, status, 79))) {
      row_slot[n % 3 * kBQ + r] = l;
      ptx::mbar_arrive(&bars->l_ready);
    }
  } else {
    // ------------------------------ drain and output ---------------------------
    ptx::setmaxnreg_inc<kRegsDrain>();
    const int quad = warp & 3;
    const int r = quad * 32 + lane;
    const uint32_t to = tmem + (static_cast<uint32_t>(quad * 32) << 16) + kTmemO;
    const float sl2 = p.scale * 1.4426950408889634f;
    float sum[D];
#pragma unroll
    for (int i = 0; i < D; ++i) sum[i] = 0.f;
    float m_prev = -INFINITY;
    bool alive = true;
    for (int j = 0; j < n; ++j) {
      bool ready = ptx::mbar_wait(&bars->m_ready[j % 3], (j / 3) & 1u, abort_flag, status, 80);
      ready = ready && ptx::mbar_wait(&bars->o_full, j & 1u, abort_flag, status, 81);
      if (!__all_sync(0xffffffffu, ready)) {
        alive = false;
        break;
      }
      ptx::tcgen05_fence_after_thread_sync();
      const float m_j = row_slot[j % 3 * kBQ + r];
      const float alpha = m_j == m_prev ? 1.0f : ptx::ex2_approx((m_prev - m_j) * sl2);  // 0 before the first step
      m_prev = m_j;
#pragma unroll
      for (int cc = 0; cc < D / 32; ++cc) {
        uint32_t ov[32];
        ptx::tmem_ld_32x32b_x32(to + cc * 32, ov);
        ptx::tmem_ld_wait();
#pragma unroll
        for (int i = 0; i < 32; ++i) sum[cc * 32 + i] = fmaf(sum[cc * 32 + i], alpha, __uint_as_float(ov[i]));
      }
      ptx::tcgen05_fence_before_thread_sync();
      ptx::mbar_arrive(&bars->o_empty);
    }
    if (alive && __all_sync(0xffffffffu, ptx::mbar_wait(&bars->l_ready, 0, abort_flag, status, 82))) {
      const float inv = 1.0f / row_slot[n % 3 * kBQ + r];
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
