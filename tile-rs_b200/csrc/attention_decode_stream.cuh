// Decode attention on 16-bit caches, up to eight query heads per (batch, KV head): the caches as one stream of tiles, dealt out evenly.
//
// Semantics as attention_decode.cuh.  That kernel gives every cache to a cluster, or to a number of CTAs, so that a launch takes whole waves of them:
// 136 caches of 1729 positions are 544 CTAs for 444 places.  Here the tiles of all caches, 8 KiB of K and of V each, are numbered
// through and one CTA per SM takes an equal, contiguous share, which may begin and end inside a cache.  A cache that lies in one share is
// finished there; the records of the others, two per CTA at most, are merged by a second kernel.
//
// A CTA has eight warps.  Each takes every eighth tile of the share's part of a cache, loads K and V tiles by TMA (64-column groups, 128-byte swizzle, no
// multicast) into three slots of its own, a load ahead of the next one's use across caches, and keeps (maximum, sum, O) of the heads as the rows
// of mma.sync m16n8k16 tiles; rows 8 to 15 of those are zero and have no registers.  At the end of a cache the warps' records are merged
// through shared memory while the first tiles of the next are on their way.
// Bound: HBM.  134 MB by one CTA per SM take 20.8 us with bulk copies in flight of 128 KiB, 25 with a cp.async ring (the plain kernel's).
#pragma once

#include "attention_decode.cuh"
#include "ptx.cuh"

namespace tsm100 {
namespace attn_decode {
namespace stream {

constexpr int kWarps = 8, kThreads = kWarps * 32;
constexpr int kRows = 8;              // query heads
constexpr int kSlots = 3;             // per warp
constexpr int kTileBytes = 8192;      // of K or of V
constexpr int kMaxCtas = 256;
template <int D>
constexpr int tile_rows() { return kTileBytes / (D * 2); }
struct alignas(8) Barriers {
  uint64_t full[kWarps * kSlots];
  uint32_t abort_flag;
};
template <int D>
constexpr int kRec = D + 4;           // floats of a head's record: O, maximum, sum; 16-byte rows
template <int D>
constexpr int record_floats() { return kRows * kRec<D>; }
template <int D>
constexpr int smem_bytes() {
  return kWarps * kSlots * kTileBytes + kWarps * record_floats<D>() * 4 + static_cast<int>(sizeof(Barriers)) + 1024;
}
static_assert(smem_bytes<128>() <= 227 * 1024, "shared memory budget of one CTA");
// its bounded waits report sites 121 and 122

struct Params {
  int32_t heads_q, heads_kv, group;
  int32_t head_base, heads_here;   // of a group, this launch
  int32_t seq_len;
  int64_t max_seq;
  int32_t tiles;                   // per cache
  int32_t grain;                   // shares are whole multiples of so many tiles
  int64_t grains;
  float scale_log2;
  float* part;                     // [CTA][2][8][D + 4]: of a cache that began in an earlier share, of one that goes on in the next
  uint32_t* status;
};
__device__ __forceinline__ int64_t share_begin(const Params& p, int64_t cta, int64_t ctas) { return cta * p.grains / ctas * p.grain; }

__device__ __forceinline__ void tma_load_4d(uint32_t dst, const CUtensorMap* map, uint64_t* bar, int32_t y, int32_t w) {
  asm volatile(
      "cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %3, %5}], [%2];" ::"r"(dst),
      "l"(reinterpret_cast<uint64_t>(map)), "r"(ptx::smem_u32(bar)), "r"(0), "r"(y), "r"(w)
      : "memory");
}
// Rows 0 to 7 of a 16 x 8 tile; the others are zero.
template <bool kIsBf16>
__device__ __forceinline__ void mma_upper(float (&d)[2], uint32_t a0, uint32_t a2, uint32_t b0, uint32_t b1) {
  float unused0, unused1;
  if (kIsBf16)
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %6, %5, %6}, {%7, %8}, {%0, %1, %9, %9};"
                 : "+f"(d[0]), "+f"(d[1]), "=f"(unused0), "=f"(unused1) : "r"(a0), "r"(a2), "r"(0u), "r"(b0), "r"(b1), "f"(0.f));
  else
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %6, %5, %6}, {%7, %8}, {%0, %1, %9, %9};"
                 : "+f"(d[0]), "+f"(d[1]), "=f"(unused0), "=f"(unused1) : "r"(a0), "r"(a2), "r"(0u), "r"(b0), "r"(b1), "f"(0.f));
}

template <typename T, int D>
__global__ void __launch_bounds__(kThreads, 1)
attention_decode_stream_kernel(const __grid_constant__ CUtensorMap tmap_k, const __grid_constant__ CUtensorMap tmap_v, const T* __restrict__ q,
                               const uint8_t* __restrict__ kc, const uint8_t* __restrict__ vc, T* __restrict__ o, const __grid_constant__ Params p) {
  constexpr bool kIsBf16 = !std::is_same<T, __half>::value;
  constexpr int TP = tile_rows<D>(), N8 = TP / 8, KSTEPS = D / 16, REC = kRec<D>, kGroupBytes = TP * 128;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  float* records = reinterpret_cast<float*>(smem + kWarps * kSlots * kTileBytes);
  Barriers* bars = reinterpret_cast<Barriers*>(records + kWarps * record_floats<D>());
  volatile uint32_t* abort_flag = &bars->abort_flag;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, gr = lane >> 2, tq = lane & 3;
  const int64_t t0 = share_begin(p, blockIdx.x, gridDim.x), t1 = share_begin(p, blockIdx.x + 1, gridDim.x);
  if (tid == 0) {
    for (int i = 0; i < kWarps * kSlots; ++i) ptx::mbar_init(&bars->full[i], 1);
    bars->abort_flag = 0;
    ptx::fence_mbar_init();
  }
  __syncthreads();
  ptx::launch_dependents();

  // This warp's tiles: every eighth of each part of the share that lies in one cache.
  struct Cursor {
    int unit, tile, end;  // end: of the part
  };
  auto settle = [&](Cursor& c) {  // on to the first part that has a tile for this warp
    while (c.tile >= c.end) {
      const int64_t next = static_cast<int64_t>(++c.unit) * p.tiles;
      if (next >= t1) return false;
      c.tile = warp;
      c.end = static_cast<int>(min(static_cast<int64_t>(p.tiles), t1 - next));
    }
    return true;
  };
  const int unit0 = static_cast<int>(t0 / p.tiles), begin0 = static_cast<int>(t0 - static_cast<int64_t>(unit0) * p.tiles);
  const int end0 = static_cast<int>(min(static_cast<int64_t>(p.tiles), t1 - static_cast<int64_t>(unit0) * p.tiles));
  Cursor ahead{unit0, begin0 + warp, end0};
  bool more = t0 < t1 && settle(ahead);
  if (more && lane == 0) {
    // while the kernel before this one runs: the warp's first tiles into the L2
    const int64_t row = ahead.unit * p.max_seq + static_cast<int64_t>(ahead.tile) * TP;
    const uint32_t bytes = static_cast<uint32_t>(min(TP, p.seq_len - ahead.tile * TP)) * (D * 2);
    ptx::prefetch_l2(kc + row * (D * 2), bytes);
    ptx::prefetch_l2(vc + row * (D * 2), bytes);
    ptx::prefetch_tensormap(&tmap_k);
    ptx::prefetch_tensormap(&tmap_v);
  }
  q = ptx::wait_prior_grid(q);

  const uint32_t slots = ptx::smem_u32(smem) + warp * (kSlots * kTileBytes);
  uint64_t* full = &bars->full[warp * kSlots];
  int load_slot = 0;
  bool load_v = false;
  auto issue = [&]() {  // the warp's next load, K and V of a tile in turn
    if (!more) return;
    if (lane == 0) {
      ptx::mbar_arrive_expect_tx(&full[load_slot], kTileBytes);
      tma_load_4d(slots + load_slot * kTileBytes, load_v ? &tmap_v : &tmap_k, &full[load_slot], ahead.tile * TP, ahead.unit);
    }
    if (load_v) {
      ahead.tile += kWarps;
      more = settle(ahead);
    }
    load_v = !load_v;
    load_slot = load_slot + 1 == kSlots ? 0 : load_slot + 1;
  };
#pragma unroll
  for (int i = 0; i < kSlots; ++i) issue();

  int slot = 0;
  uint32_t phase = 0;
  bool alive = true;
  auto arrived = [&](int site) {
    alive = alive && __all_sync(0xffffffffu, ptx::mbar_wait(&full[slot], phase, abort_flag, p.status, site));
    return alive;
  };
  auto release = [&]() {  // every lane has read the slot: it is filled again
    __syncwarp();
    if (++slot == kSlots) slot = 0, phase ^= 1u;
    issue();
  };
  const int swizzle = lane & 7;
  uint32_t qa[KSTEPS][2];  // the heads' rows of Q, loaded while the cache before is merged
  auto load_q = [&](int unit) {
    const int64_t head = static_cast<int64_t>(unit / p.heads_kv) * p.heads_q + unit % p.heads_kv * p.group + p.head_base + gr;
    const uint32_t* row = reinterpret_cast<const uint32_t*>(q + head * D);
    const bool ok = gr < p.heads_here;
#pragma unroll
    for (int kk = 0; kk < KSTEPS; ++kk) {
      qa[kk][0] = ok ? __ldg(row + kk * 8 + tq) : 0u;
      qa[kk][1] = ok ? __ldg(row + kk * 8 + tq + 4) : 0u;
    }
  };
  load_q(unit0);
  for (int unit = unit0; static_cast<int64_t>(unit) * p.tiles < t1; ++unit) {
    const int begin = unit == unit0 ? begin0 : 0;
    const int end = static_cast<int>(min(static_cast<int64_t>(p.tiles), t1 - static_cast<int64_t>(unit) * p.tiles));
    const int b = unit / p.heads_kv, h0 = unit % p.heads_kv * p.group + p.head_base;
    float oacc[2 * KSTEPS][2];
#pragma unroll
    for (int j = 0; j < 2 * KSTEPS; ++j) oacc[j][0] = oacc[j][1] = 0.f;
    float m = -INFINITY, l = 0.f;  // of head gr; this thread's share of the sum
    for (int tile = begin + warp; tile < end; tile += kWarps) {
      if (!arrived(121)) break;
      const uint32_t ks = slots + slot * kTileBytes;
      float s[N8][2];
#pragma unroll
      for (int j = 0; j < N8; ++j) s[j][0] = s[j][1] = 0.f;
#pragma unroll
      for (int kk = 0; kk < KSTEPS; ++kk)
#pragma unroll
        for (int j = 0; j < N8 / 2; ++j) {
          uint32_t kb[4];  // (positions 0-7, k lo), (0-7, k hi), (8-15, k lo), (8-15, k hi)
          mma::ldmatrix_x4(ks + (kk >> 2) * kGroupBytes + (j * 16 + (lane & 7) + ((lane >> 4) & 1) * 8) * 128 + ((((kk & 3) * 2 + ((lane >> 3) & 1)) ^ swizzle) << 4), kb);
          mma_upper<kIsBf16>(s[2 * j], qa[kk][0], qa[kk][1], kb[0], kb[1]);
          mma_upper<kIsBf16>(s[2 * j + 1], qa[kk][0], qa[kk][1], kb[2], kb[3]);
        }
      release();
      // to log2 units; positions past the end carry no weight
      const int pos = tile * TP + 2 * tq;
      const bool ragged = (tile + 1) * TP > p.seq_len;
      float t = -INFINITY;
#pragma unroll
      for (int j = 0; j < N8; ++j)
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          s[j][e] = ragged && pos + j * 8 + e >= p.seq_len ? -INFINITY : s[j][e] * p.scale_log2;
          t = fmaxf(t, s[j][e]);
        }
      t = fmaxf(t, __shfl_xor_sync(0xffffffffu, t, 1));
      t = fmaxf(t, __shfl_xor_sync(0xffffffffu, t, 2));
      const float n = fmaxf(m, t), a = ptx::ex2_approx(m - n);  // a tile has at least one position; first tile: 2^(-inf) = 0
      m = n;
      uint32_t pa[N8];
      float sum = 0.f;
#pragma unroll
      for (int j = 0; j < N8; ++j) {
        const float p0 = ptx::ex2_approx(s[j][0] - n), p1 = ptx::ex2_approx(s[j][1] - n);
        sum += p0 + p1;
        pa[j] = mma::pack2<kIsBf16>(p0, p1);
      }
      l = fmaf(l, a, sum);
#pragma unroll
      for (int j = 0; j < 2 * KSTEPS; ++j) oacc[j][0] *= a, oacc[j][1] *= a;
      if (!arrived(122)) break;
      const uint32_t vs = slots + slot * kTileBytes;
      if (ragged) {
        // what lies behind the last position weighs nothing, but may be anything
        for (int i = lane; i < TP * (D / 8); i += 32) {
          const int row = i / (D / 8), c = i % (D / 8);
          if (tile * TP + row >= p.seq_len) ptx::st_shared_v4(vs + (c >> 3) * kGroupBytes + row * 128 + ((c & 7) << 4), 0u, 0u, 0u, 0u);
        }
        __syncwarp();
      }
#pragma unroll
      for (int jj = 0; jj < KSTEPS; ++jj)
#pragma unroll
        for (int j = 0; j < N8 / 2; ++j) {
          uint32_t vb[4];  // (positions 0-7, d lo), (8-15, d lo), (0-7, d hi), (8-15, d hi), transposed on load
          mma::ldmatrix_x4_trans(vs + (jj >> 2) * kGroupBytes + (j * 16 + (lane & 7) + ((lane >> 3) & 1) * 8) * 128 + ((((jj & 3) * 2 + ((lane >> 4) & 1)) ^ swizzle) << 4), vb);
          mma_upper<kIsBf16>(oacc[2 * jj], pa[2 * j], pa[2 * j + 1], vb[0], vb[1]);
          mma_upper<kIsBf16>(oacc[2 * jj + 1], pa[2 * j], pa[2 * j + 1], vb[2], vb[3]);
        }
      if (ragged) ptx::fence_proxy_async_smem();  // the zeros before the slot's next copy
      release();
    }
    l += __shfl_xor_sync(0xffffffffu, l, 1);
    l += __shfl_xor_sync(0xffffffffu, l, 2);

    if (static_cast<int64_t>(unit + 1) * p.tiles < t1) load_q(unit + 1);
    __syncthreads();  // the records of the cache before have been read
    {
      float* rec = records + warp * record_floats<D>() + gr * REC;
#pragma unroll
      for (int j = 0; j < 2 * KSTEPS; ++j) *reinterpret_cast<float2*>(rec + j * 8 + 2 * tq) = make_float2(oacc[j][0], oacc[j][1]);
      if (tq == 0) *reinterpret_cast<float2*>(rec + D) = make_float2(m, l);
    }
    __syncthreads();
    const bool whole = begin == 0 && end == p.tiles;
    for (int i = tid; i < p.heads_here * (D / 4); i += kThreads) {
      const int hh = i / (D / 4), dd = i % (D / 4) * 4;
      const float* rec = records + hh * REC;
      float2 ml[kWarps];
      float mm = -INFINITY;
#pragma unroll
      for (int w = 0; w < kWarps; ++w) {
        ml[w] = *reinterpret_cast<const float2*>(rec + w * record_floats<D>() + D);
        mm = fmaxf(mm, ml[w].x);
      }
      float ll = 0.f;
      float4 oo = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
      for (int w = 0; w < kWarps; ++w) {
        const float wgt = ml[w].x == -INFINITY ? 0.f : ptx::ex2_approx(ml[w].x - mm);  // a warp without tiles carries no weight
        const float4 x = *reinterpret_cast<const float4*>(rec + w * record_floats<D>() + dd);
        ll = fmaf(ml[w].y, wgt, ll);
        oo.x = fmaf(x.x, wgt, oo.x), oo.y = fmaf(x.y, wgt, oo.y), oo.z = fmaf(x.z, wgt, oo.z), oo.w = fmaf(x.w, wgt, oo.w);
      }
      if (whole) {
        const uint2 packed = make_uint2(mma::pack2<kIsBf16>(oo.x / ll, oo.y / ll), mma::pack2<kIsBf16>(oo.z / ll, oo.w / ll));
        *reinterpret_cast<uint2*>(o + (static_cast<int64_t>(b) * p.heads_q + h0 + hh) * D + dd) = packed;
      } else {
        float* out = p.part + ((static_cast<int64_t>(blockIdx.x) * 2 + (begin == 0 ? 1 : 0)) * kRows + hh) * REC;
        *reinterpret_cast<float4*>(out + dd) = oo;
        if (dd == 0) *reinterpret_cast<float2*>(out + D) = make_float2(mm, ll);
      }
    }
  }
  if (*abort_flag != 0u) {
    // a wait gave up: copies in flight land before the shared memory is released
    const unsigned long long since = ptx::globaltimer_ns();
    while (ptx::globaltimer_ns() - since < 1000000ull) {
    }
    __syncthreads();
  }
}

// The records of a cache that several shares have a part of, in order; one CTA of D threads per (cache, head).
template <typename T, int D>
__global__ void __launch_bounds__(D)
attention_decode_stream_merge_kernel(T* __restrict__ o, const Params p, int32_t ctas) {
  constexpr int REC = kRec<D>;
  __shared__ float w[kMaxCtas];
  const int unit = blockIdx.x / p.heads_here, hh = blockIdx.x % p.heads_here;
  const int64_t first_tile = static_cast<int64_t>(unit) * p.tiles;
  auto owner = [&](int64_t tile) {  // the CTA whose share has it
    int64_t c = tile / p.grain * ctas / p.grains;
    while (c + 1 < ctas && share_begin(p, c + 1, ctas) <= tile) ++c;
    while (share_begin(p, c, ctas) > tile) --c;
    return static_cast<int>(c);
  };
  const int first = owner(first_tile), n = owner(first_tile + p.tiles - 1) - first + 1;
  ptx::launch_dependents();
  const float* part = ptx::wait_prior_grid(p.part);
  if (n == 1) return;
  auto record = [&](int i) { return part + ((static_cast<int64_t>(first + i) * 2 + (i == 0 ? 1 : 0)) * kRows + hh) * REC; };
  // this thread's column of the first records, on its way while the weights are worked out
  constexpr int kFirst = 20;
  float early[kFirst];
#pragma unroll
  for (int i = 0; i < kFirst; ++i) early[i] = i < n ? record(i)[threadIdx.x] : 0.f;
  float mm = -INFINITY;
  for (int i = threadIdx.x & 31; i < n; i += 32) mm = fmaxf(mm, record(i)[D]);
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) mm = fmaxf(mm, __shfl_xor_sync(0xffffffffu, mm, off));
  float ll = 0.f;
  for (int i = threadIdx.x & 31; i < n; i += 32) {
    const float* r = record(i);
    const float x = r[D] == -INFINITY ? 0.f : ptx::ex2_approx(r[D] - mm);
    if (threadIdx.x < 32) w[i] = x;
    ll = fmaf(r[D + 1], x, ll);
  }
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) ll += __shfl_xor_sync(0xffffffffu, ll, off);
  __syncthreads();
  float oo = 0.f;
#pragma unroll
  for (int i = 0; i < kFirst; ++i)
    if (i < n) oo = fmaf(early[i], w[i], oo);
#pragma unroll 8
  for (int i = kFirst; i < n; ++i) oo = fmaf(record(i)[threadIdx.x], w[i], oo);
  softmax::Elem<T>::store1(o + (static_cast<int64_t>(unit / p.heads_kv) * p.heads_q + unit % p.heads_kv * p.group + p.head_base + hh) * D + threadIdx.x, oo / ll);
}

}  // namespace stream
}  // namespace attn_decode
}  // namespace tsm100
