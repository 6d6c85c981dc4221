// Which kernel a problem runs on, where that depends on its size: host arithmetic only, so that the rules can be looked at
// without a GPU (tests/test_routes.py).  The figures beside a rule are device times in microseconds as graph replays, the
// other side first.
#pragma once

#include <algorithm>
#include <cstdint>

namespace tsm100 {
namespace route {

constexpr int64_t div_up(int64_t a, int64_t b) { return (a + b - 1) / b; }

// 16-bit attention with heads of 32 or 64: the tcgen05 kernel (attention_narrow.cuh, 256 query rows and 128 keys at a time) or the
// warp-level one (64 query rows).  Up to 64 keys a tcgen05 tile is mostly padding, and its start alone is longer than the
// warp-level kernel's whole work: causal, 2048 heads of 64 keys x 64 61 warp-level, 97 tcgen05, 1 head 6.7 / 7.7; from 65 keys on it
// leads (98.4 / 97.3, 1 head 9.6 / 7.7).  Heads of 32 fill half of its width: there it leads from 129 keys on when it has query
// blocks for all SMs (256 heads of 160 19.1 / 17.7), from 449 on when there are fewer (8 heads of 300 10.0 / 11.8, of 400 13.1 / 13.8, of
// 512 15.6 / 14.1); 2048 heads of 64 keys x 32 31 / 96.
inline bool attention_narrow_on_tcgen05(int32_t head_dim, int64_t seq_kv, int64_t query_blocks, int sms) {
  if (head_dim == 64) return seq_kv > 64;
  return seq_kv > (query_blocks > sms ? 128 : 448);
}

// f32 attention: the tcgen05 kernel (attention_f32_tc.cuh, 128 query rows and 64 keys at a time, behind a launch that splits K and V), or the
// warp-level one (128 rows, 64 keys).  A step of 64 keys takes the one 1.9 us and the other 3 (heads of 32) to 11 us, the second launch 3.5 us of a
// call in a row and 1.5 as graph replays.  Calls in a row, causal, warp level / tcgen05: 2 heads of 16 x 128 11.6 / 10.3, of 64 x 128 13.2 / 10.5, of 200
// x 128 40.9 / 14.6, 128 heads of 128 x 128 25.9 / 19.2; heads of 96 16 of 64 11.0 / 10.4, of 128 19.8 / 12.3; of 64 16 of 64 7.9 / 10.4, of 65 12.6 /
// 10.4, 128 of 128 13.8 / 12.1; of 32 16 of 128 8.1 / 10.4, of 200 12.9 / 10.6, 128 of 200 24.8 / 16.1.
inline bool attention_f32_on_tcgen05(int32_t head_dim, int64_t seq_kv) { return head_dim == 128 || seq_kv > (head_dim == 32 ? 160 : 64); }

// 16-bit attention on tcgen05, unsplit: query rows of a block, 256 (two tiles) or 128.  Two tiles share K and V, and a step of both takes the SM
// 3240 cycles, of one 2060; but blocks of one tile are twice as many, and the longest chain of steps is shorter.  `rows` per head, which see
// `offset` keys before their own where `causal`, all `keys` otherwise; a block's start and end take 9000 cycles, once more where there is a second wave, and a
// wave as long as its lightest block at least.
// 256 rows / 128: causal 8 heads of 2482 37.3 / 27.7 us, 16 of 838 15.6 / 12.6, 32 of 938 18.4 / 19.8; all keys 16 of 640 13.7 / 10.8; heads of 64 8 of 764 13.9 /
// 10.7; with rotation and appends 131 tokens on 3677, 16 heads, 62.9 / 49.1, 581 on 11, 32 heads, 26.4 / 28.1.
inline int attention_block_rows(int64_t rows, int64_t heads, int64_t keys, int64_t offset, bool causal, int sms) {
  if (rows <= 128) return 128;
  if (div_up(rows, 256) * heads > 4 * sms) return 256;
  int64_t best = 0, best_cost = INT64_MAX;
  for (int64_t block = 256; block >= 128; block -= 128) {
    const int64_t blocks = div_up(rows, block);
    auto time = [&](int64_t i) {  // of the block that is i-th from the end, the heaviest first
      const int64_t r = (blocks - 1 - i) * block, end = std::min(rows, r + block);
      return 9000 + div_up(causal ? std::min(keys, end + offset) : keys, 128) * (end - r > 128 ? 3240 : 2060);
    };
    int64_t longest = 0, all = 0, waves = 0;
    for (int64_t i = 0; i < blocks; ++i) longest = std::max(longest, time(i)), all += time(i) * heads;
    for (int64_t done = 0; done < blocks * heads; done += sms) waves += time((std::min(blocks * heads, done + sms) - 1) / heads);  // the lightest of each
    const int64_t cost = blocks * heads <= sms ? longest : std::max({longest, waves, all / sms + 9000});
    if (cost < best_cost) best_cost = cost, best = block;
  }
  return static_cast<int>(best);
}

// 16-bit attention on tcgen05: how many CTAs share the KV steps of a query block.  One CTA fills an SM, so the steps are dealt out when
// there are blocks for at most half of the SMs: 512 keys or more to each CTA from 4096 keys on, 1024 or more from 8192 on, where the merge of more records
// takes what the shorter chains save.  With rotation and appends, 2048 keys to a CTA / 1024 / 512: 30 tokens on 5000, 4 heads, 47 / 32 / 26 us, 19 on 5342, 8 heads,
// 51 / - / 27, 512 on 7000, 8 heads, 50 / 38 / 39, 30 on 9000, 4 heads, 45 / 32 / 30, on 16000 48 / 37 / 39, 200 on 16000, 8 heads, 51 / 43 / 46; 512 on 15872, 32 heads (64
// blocks), 212 unsplit, 122 split.  Below 4096 keys a call is never split, so that a prompt in chunks gives the bits of the whole one.
inline int attention_split_ctas(int64_t blocks, int64_t keys, int sms) {
  if (keys < 4096) return 1;
  return static_cast<int>(std::max<int64_t>(1, std::min<int64_t>(sms / blocks, keys / (keys < 8192 ? 512 : 1024))));
}

// 16-bit GEMM on the tensor cores: CTA pairs (256 x 256 tiles, gemm_tc2.cuh), single CTAs (128 x 256 tiles, gemm_tc.cuh; both
// persistent) or the few-tiles kernel (128 columns x `rows` rows of C per CTA, K over `splits` CTAs of a cluster, gemm_skinny.cuh).
struct Gemm16 {
  enum Kind { kPairs, kSingles, kFewTiles } kind;
  int rows;             // few tiles: rows of C per CTA
  int splits;
  int64_t k_blocks_per_cta;  // 64 of K each
};
constexpr int kMaxGemmSplit = 8;

inline Gemm16 gemm16(int64_t m, int64_t n, int64_t k, int64_t batch, int sms) {
  Gemm16 r{Gemm16::kFewTiles, m <= 16 ? 16 : m <= 32 ? 32 : m <= 64 ? 64 : 128, 1, 0};
  const bool wide = r.rows == 128;
  const int64_t tiles = div_up(m, r.rows) * div_up(n, 128) * batch, kb = div_up(k, 64);
  // K over a cluster while every CTA keeps four k-blocks and all clusters fit the GPU at once, two CTAs per SM (clusters of 8 leave a
  // fifth of the SMs' places empty, of 4 a sixteenth; with 128 k-blocks or more a second wave pays all the same).  Two CTAs alone do
  // not earn a cluster's launch while K is short.
  while (r.splits < kMaxGemmSplit) {
    const int to = 2 * r.splits;
    const int64_t room = to == 2 || kb >= 128 ? 2 * sms : to == 4 ? sms * 15 / 8 : sms * 8 / 5;
    if (tiles * to > room || kb / to < 4) break;
    r.splits = to;
  }
  if (r.splits == 2 && kb < (tiles * 2 > sms ? 48 : wide ? 16 : r.rows == 64 ? 12 : 9)) r.splits = 1;
  r.k_blocks_per_cta = div_up(kb, r.splits);
  // Unsplit, the few-tiles kernel starts a CTA per tile and hides nothing of its start and end but behind a second CTA; the persistent
  // kernels load the next tile meanwhile.  So it pays for tiles that are all there at once, and beyond that for a long K where 256-wide
  // tiles would leave SMs idle or be half empty.  Weights from HBM, persistent / few tiles: 1 x 20480 x 5120 54 / 37, 65 x 6144 x
  // 1536 15 / 11, 20 x 4096 x 64 of a batch of 256 35 / 88.  Over 3038 sizes 0.6 % from the best choice of each, 7 more than 5 % slower
  // than the persistent kernels alone.
  bool few;
  if (r.splits > 1) few = true;
  else if (m > 128 && n > 128) few = tiles <= sms;
  else if (m <= 16) few = tiles <= 2 * sms || (n <= 128 && kb >= 8);
  else if (m <= 64) few = 2 * tiles <= 3 * sms || (kb >= 64 && tiles <= 2 * sms) || (n <= 128 && kb >= 8 && (tiles <= 2 * sms || kb >= 16));
  else if (n > 128) few = tiles <= sms;
  else few = (n % 32 != 0 && n > 32 && tiles <= sms) || (tiles > sms && kb >= 40) || (n <= 32 && tiles >= 2 * sms && kb >= 4);
  if (!few) r.kind = m > 128 && n > 128 ? Gemm16::kPairs : Gemm16::kSingles;
  // one CTA per tile has to fit one launch
  if (few && tiles * r.splits > 0x7fffffff) r.kind = m > 128 && n > 128 ? Gemm16::kPairs : Gemm16::kSingles;
  return r;
}

// CTA pairs: does C leave through shared memory, in whole boxes, or from the lanes that hold its rows?  The boxes are out in a sixth of the time, which
// counts where a tile's products take no longer than its end (K below 2048) or where the last wave's end is a part of the whole; in a
// long row of long tiles the board's power decides, and the slower way is 1 to 5 % cheaper.  Rows / boxes: 4096 x 4096 x 512 of a batch of 2 39.6 / 30.0 us, x
// 1024 53.7 / 51.2, x 2048 105.3 / 107.2, x 4096 198 / 203; 8192^3 803 / 833; 2048 x 2048 x 4096 (64 tiles) 26.1 / 25.6, 2048 x 4608 x 2048 (144) 28.4 / 26.2.
inline bool gemm16_pairs_store_boxes(int64_t k, int64_t tiles, int sms) { return k < 2048 || (k <= 4096 && tiles <= sms); }

// 16-bit products whose rows start anywhere: operands copied to rows that tensor maps can describe and the tensor cores (gemm_pad.cuh), or the FP32 pipe.  The
// copies cost one launch and traffic per row and column, whatever K is; a CTA of the FP32 pipe walks through K alone, 0.12 us for each step of it.  FP32 pipe /
// copies, calls in a row: 3 x 123 x 3313 275 / 10.3, 1 x 77 x 97 12.3 / 10.4, x 65 9.2 / 10.4, 64 x 301 x 57 11.6 / 10.4, x 41 8.9 / 10.3, 500 x 501 x 41 10.2 / 10.3, x 33 8.2 /
// 10.4, 2000 x 3001 x 33 30.8 / 19.8, x 17 22.6 / 19.8, 8001 x 5001 x 17 118 / 73.
// Fewer than 512 outputs with a long K keep the FP32 pipe's rounding to nearest, up to 2^26 products.  Where the line lies: the tensor core's sums, which round toward
// zero, move all-positive f16 results by less than 2^-24 (norm) from the 64-bit result up to K = 6144 (rounding error 2.2e-4, times 2e-6 more at 127, 5e-5 at 3313,
// 1.7e-4 at 5999, 3.3e-4 at 8191, 1.4e-3 at 16383, 2 % at 60001; FP32 pipe 3e-5 at most), bf16 ones by 4e-6 of theirs at 16383; normally distributed data is nearer
// than on the FP32 pipe.
inline bool gemm16_copies_pay(int64_t m, int64_t n, int64_t k, int64_t batch, bool bf16) {
  const double outputs = static_cast<double>(m) * n * batch;
  if (outputs < 512.0 && k > (bf16 ? 16384 : 6144) && outputs * k < 67108864.0) return false;
  return k >= (outputs >= 6000000.0 ? 16 : outputs >= 262144.0 ? 33 : outputs >= 16384.0 ? 48 : 72);
}

// f32 GEMM: operand planes and CTA pairs (gemm_tf32_tc.cuh), operands split on the way in (gemm_f32_fused.cuh), the warp-level kernel
// (gemm_tf32x3.cuh; `aligned`: rows start on 16-byte boundaries, the only ones it takes) or the FP32 pipe.
constexpr int kMaxWarpF32Split = 4, kMaxF32FusedSplit = 8;
inline int gemm_f32_warp_splits(int64_t tiles64, int64_t k, int sms) {
  // fewer 64 x 64 tiles than SMs: a cluster splits K while all CTAs still fit the GPU at once (two per SM) and every CTA keeps at least
  // four 32-deep slices
  int splits = 1;
  while (splits < kMaxWarpF32Split && tiles64 * splits * 2 <= 2 * sms && k / (2 * splits) >= 128) splits *= 2;
  return splits;
}
struct GemmF32 {
  enum Kind { kPlanes, kFused, kWarp, kFp32 } kind;
  int bn, splits;   // fused: columns per tile, CTAs that share K
};
inline GemmF32 gemm_f32(int64_t m, int64_t n, int64_t k, int64_t batch, bool aligned, int sms, bool b_transposed = false) {
  GemmF32 r{aligned ? GemmF32::kWarp : GemmF32::kFp32, 0, 1};
  // The fused kernel moves 32 KiB of operands from the L2 for every 128 x 128 x 32 products, the planes' 256 x 256 tiles half of that:
  // planes / fused 1552 x 2281 x 1827 82 / 141, 1533 x 1448 x 968 (72 tiles of 128 x 256) 31 / 36, 1500 x 1036 x 1723 (60) 43 / 41.
  if (div_up(m, 128) * div_up(n, 256) * batch >= 64 && k >= 256) {
    r.kind = GemmF32::kPlanes;
    return r;
  }
  const int64_t tiles64 = div_up(m, 64) * div_up(n, 64) * batch, kb = div_up(k, 32);
  if (!aligned && k < 64) return r;
  if (aligned) {
    // What is small in every way: warp level / fused 3.9 / 5.3 (650 x 80 x 64), 5.1 / 6.3 (1670 x 124 x 68), 6.4 / 6.9 (1268 x 228 x 100); but
    // 7.1 / 6.4 (878 x 984 x 68) and 9.5 / 8.4 (1523 x 120 x 220).
    if (k < 160 && tiles64 <= sms) return r;
    // Many tiles of 64 rows or less: the fused kernel's are half empty.  300 problems of 64 x 64 x 128 13.8 / 15.3, 1000 of 32 x 32 x 200
    // 39 / 50 (of 33 x 33 x 201, FP32 pipe, 110 / 64).
    if (m <= 64 && tiles64 > sms) return r;
    // A K of one block: a tile is little more than its start and its stores, and smaller ones overlap better, unless there are very many and
    // the fused kernel's are full: 1000 x 1000 x 32 3.8 / 4.9, 2000 x 2000 8.0 / 8.8, 40 of 1029 x 140 14.8 / 20.9, but 4000 x 4000 27.2 / 24.6.
    if (k <= 32 && (tiles64 <= 10 * sms || 2 * tiles64 <= 7 * div_up(m, 128) * div_up(n, 128) * batch)) return r;
    // One column of tiles: 60 of 931 x 16 x 64 12.4 / 15.8, x 96 17.3 / 18.7, x 128 22.4 / 21.8; 20 of 2000 x 64 x 64 10.0 / 11.2, x 96 13.5 / 13.6;
    // 400 of 128 x 64 x 64 11.7 / 11.5, x 96 16.0 / 13.8.
    if (k <= 64 && n <= 64) return r;
  }
  if (div_up(m, 128) * div_up(n, 64) * batch >= 0x7fffffff) return r;
  // Tile width and split by the time they take, in nanoseconds (fitted to 200 sizes between 64 and 2600, 8 % off in the mean): a launch costs
  // 4.4 us on 64 columns, 5.5 on 128, a further wave 1.4 and 2.3, a k-block what stands below: rows that start anywhere are loaded value by
  // value, B stored [K][N] in columns, and both cost more where a CTA loads 128 columns.  All clusters have to fit the GPU at
  // once, one CTA per SM (1419 x 372 x 680 as 36 clusters of four 23 us, in two waves, of two 16); of clusters of 2, 3, ... 8 a B200
  // holds 74, 45, 33, 26, 22, 15 and 15.  Any size of cluster, not powers of two alone: 2410 x 108 x 2256 27.5 -> 21.2, 549 x 1064 x 900 24.0 -> 20.9,
  // 1900 x 261 x 2591 62 -> 54, 267 x 724 x 792 14.8 -> 12.6.
  const int64_t kb64 = aligned ? 810 : 880, kb128 = aligned ? (b_transposed ? 1020 : 1170) : (b_transposed ? 1200 : 1270);
  int64_t best = INT64_MAX;
  for (int bn = 64; bn <= 128; bn += 64)
    for (int s = 1; s <= kMaxF32FusedSplit; ++s) {
      const int64_t tiles = div_up(m, 128) * div_up(n, bn) * batch, per = div_up(kb, s);
      const int64_t room = s == 2 ? sms / 2 : s == 3 ? sms * 9 / 29 : s == 4 ? sms * 9 / 40 : s == 5 ? sms * 7 / 40 : s == 6 ? sms * 3 / 20 : sms / 10;
      if (s > 1 && (tiles > room || per < 2 || (s - 1) * per >= kb)) continue;
      const int64_t waves = s > 1 ? 1 : div_up(tiles, sms);
      const int64_t ns = bn == 64 ? 4350 + waves * per * kb64 + (waves > 1 ? waves * 1400 : 0) + (s > 1 ? 860 + 80 * s : 0)
                                  : 5550 + waves * per * kb128 + (waves > 1 ? waves * 2300 : 0) + (s > 1 ? 440 + 110 * s : 0);
      if (ns < best) best = ns, r.bn = bn, r.splits = s;
    }
  r.kind = GemmF32::kFused;
  return r;
}

// The tiles of the planes' kernel over SM pairs: columns of a tile (256 or 128, of 256 rows), how many tiles are worked on whole, and how
// many pairs share each of the rest.
struct PairTiles {
  int bn;
  int64_t whole_tiles;
  int splits;
};
inline PairTiles gemm_f32_pair_tiles(int64_t m, int64_t n, int64_t k, int64_t batch, int sms) {
  const int64_t pairs = sms / 2 > 0 ? sms / 2 : 1, kb = div_up(k, 32);
  PairTiles best{256, 0, 1};
  int64_t best_cost = INT64_MAX;
  for (int bn = 256; bn >= 128; bn -= 128) {
    const int64_t tiles = div_up(m, 256) * div_up(n, bn) * batch, rest = tiles % pairs;
    // A 128-wide tile costs two thirds of a 256-wide one, not half (its operand traffic per product is 4/3 and a chunk's drain overlaps
    // half the products): 4096^3 655 us in 4 wide waves, 757 in 7 narrow ones; 1536^3 79 us in one wide wave, 56 in one narrow.
    const int64_t per_kb = bn == 256 ? 100 : 67;
    int64_t cost = div_up(tiles, pairs) * kb * per_kb;
    int splits = 1;
    for (int s = 2; rest > 0 && s <= 4 && rest * s <= pairs && kb / s >= 8; ++s) {
      // partial sums on their way through the L2 and back cost what 14 k-blocks do, and two for each of them
      const int64_t shared = (tiles / pairs * kb + div_up(kb, s) + 14 + 2 * s) * per_kb;
      if (shared < cost) cost = shared, splits = s;
    }
    if (cost < best_cost) best_cost = cost, best = PairTiles{bn, splits > 1 ? tiles - rest : tiles, splits};
  }
  // the last share has to have k-blocks of its own
  while (best.splits > 1 && (best.splits - 1) * div_up(kb, best.splits) >= kb) --best.splits;
  if (best.splits == 1) best.whole_tiles = div_up(m, 256) * div_up(n, best.bn) * batch;
  return best;
}

// Decode attention on 16-bit caches as one stream (attention_decode_stream.cuh): CTAs (0: another kernel), tiles per cache, and shares in multiples of
// `grain` tiles, one or those of a whole cache.  Clusters / one stream, calls in a row with two appends, eight KV heads, four query heads each: 17 caches of 1729
// x 128 41.9 / 30.2 us, 29 of 1312 54.2 / 35.7, 64 of 600 53.4 / 37.6, 64 of 6000 262 / 242, 2 of 8060 25.9 / 20.3, 1 of 32768 x 64 26.0 / 17.9, 17 of 1729 x 64 21.9 /
// 18.6.  Whole caches need no merge (18 of 200 13.0 / 13.4, as graph replays 10.3 / 6.9; 37 of 300 19.9 / 17.4); shares that part caches need a second
// launch, which 50 MB pay for (46 MB, 10 of 1120 x 128, 20.9 / 18.4 and 19.7 / 19.2 as replays; 36 MB, 29 of 600 x 64, 17.2 / 17.3 and 15.6 / 18.2; 26 MB 14.4 / 18.2).
// A few caches of heads of 128 have their own CTAs already (1 of 32768 30.7 / 32.6).
struct DecodeStream {
  int64_t ctas;
  int32_t tiles, grain;
  int64_t grains;
};
constexpr int kDecodeTileBytes = 8192;  // of K or of V
inline DecodeStream decode_stream(int64_t units, int64_t seq_len, int head_dim, int sms) {
  const int64_t tiles = div_up(seq_len, kDecodeTileBytes / (2 * head_dim)), total = units * tiles;
  if (total == 0 || tiles > 0x7fffffff) return {0, 0, 0, 0};
  if (div_up(units, sms) * sms * 100 <= 108 * units) return {std::min<int64_t>(units, sms), static_cast<int32_t>(tiles), static_cast<int32_t>(tiles), units};
  if (units * seq_len * head_dim * 4 < 50ll << 20 || (head_dim == 128 && units <= 12)) return {0, 0, 0, 0};
  return {sms, static_cast<int32_t>(tiles), 1, total};
}

// Decode attention in clusters, as a programmatic dependent of the kernel before it?  That is worth 1.5 to 2.5 us of a call (not replayed from a
// graph), but with one CTA on some SMs and two on others an uneven placement beside the last CTAs of that kernel may cost the time of a CTA:
// in a row of calls, plain / chained, 10 caches of 18800 x 128 with 2 KV heads (160 CTAs) 42.7 / 48.3 us, 4 of 8000 with 8 (256) 28.9 / 33.0, 60 of
// 1000 with 2 (240, 250 KB each) 19.3 / 21.3; but one cache of 1000 with its rotation and appends (16) 17.4 / 14.1, 55 of 182 with 8 (440) 16.6 /
// 14.6, 5 of 8000 with 8 (320) 40.8 / 37.6, 10 of 3000 with 2 (160, 184 KB each) 16.5 / 13.8.
inline bool decode_is_chained(int64_t ctas, int64_t bytes_per_cta, int sms) {
  return ctas <= sms || ctas > 2 * sms || bytes_per_cta < 200 * 1024;
}

// Few-rows GEMM: is the next kernel placed from the start, or after the main loop?  From the start its first tiles follow at once where B is
// larger than the L2 and the CTAs leave few of the places of two to an SM; with more places free the next grid piles up on them.  MLP,
// off / on, where all three products are such (256 CTAs): 4096 x 16384 (128 MB) 1 token 71.8 / 73.6 us, 4 73.9 / 76.8, 16 80.3 / 78.0, 32 83.1 / 80.4,
// 8192 x 16384 137.2 / 135.0, 138.8 / 136.9, 141.8 / 139.6, 143.8 / 142.5; 3072 x 16384 (96 MB) 57.3 / 57.9, 62.2 / 62.6 (16 tokens).  With 160 CTAs 5120 x
// 20480 106 / 126 and, 16 tokens, 110 / 119, with 192 8192 x 12288 102 / 108 and 4096 x 12288 57 / 60.
inline bool skinny_places_early(uint64_t b_bytes, int64_t ctas, int sms) { return b_bytes >= (126ull << 20) && 10 * ctas >= 17 * sms; }

// Row softmax whose rows start anywhere or are too wide for one CTA's registers (softmax.cuh); `span`: the most 16-byte vectors a row
// can touch.
// 129 .. 256 vectors: a warp per row while there are rows for all warps, else a CTA.  1111 bf16, 200 rows 3.7 a warp, 2.9 a CTA, 600
// 3.7 / 3.6, 4000 8.1 / 14; 513 f32, 200 rows 2.5 / 2.4, 600 2.6 / 3.1.
inline bool softmax_row_per_warp(int64_t span, int64_t rows, int sms) { return span <= 128 || (span <= 256 && rows > 2 * sms); }

// More than 1024 vectors: how many CTAs of a cluster share a row, or 0 for one CTA per row that reads it twice.  CTAs of 256 threads
// and 1024 vectors (four of which fit an SM) while eight of them hold a row, of 512 threads and 4096 vectors beyond.  A cluster
// reads a row once, but has to fit the GPU with all others: a second wave costs more than the second read.  Cluster / twice: f32 74 rows of
// 30001 6.1 / 7.6, 130 of 28000 9.4 / 8.0, 148 of 32776 19 / 8.6, 32 of 128000 16.5 / 23; bf16 74 of 50001 5.7 / 7.5, 148 of 65536 20 / 9.0.
// Two or three CTAs for a hundred rows and more do not earn the exchange between them (f32 130 of 4099 4.0 / 3.5).
inline int softmax_cluster(int64_t span, int64_t rows, int sms) {
  if (rows > sms || span > 8 * 4096) return 0;
  if (span <= 8 * 1024) {
    const int64_t ctas = div_up(span, 1024);
    const bool fits = 3 * rows <= 2 * sms ? rows * ctas <= 4 * sms : ctas >= 4 && rows * ctas < 4 * sms;
    return fits ? static_cast<int>(ctas) : 0;
  }
  // a wave of such CTAs takes 5.3 us, reading rows twice 4.5 us and 1 us for 2048 vectors
  const int64_t ctas = div_up(span, 4096), waves = div_up(rows * ctas, sms);
  return 53 * waves < 45 + 10 * span / 2048 ? static_cast<int>(ctas) : 0;
}

// Threads of a CTA that reads its rows twice, 1024 of them per SM in all: as many CTAs as keep their rows within half of the L2 (126
// MB), but not more than there are rows.  f32 149 rows of 16400 8.3 in CTAs of 256, 7.7 in CTAs of 512; bf16 149 of 50001 10.6 / 9.9.
inline int softmax_twice_threads(int64_t row_bytes, int64_t rows, int sms) {
  const int64_t fit = (64ll << 20) / (row_bytes * sms);
  if (fit >= 4 && rows > 2 * sms) return 256;
  return fit >= 2 && rows > sms ? 512 : 1024;
}
// Whether such CTAs stay for several rows, or a CTA goes after one.  A long row outweighs a CTA's start, and the places left by rows that end first are taken
// at once: stay / go 1000 rows of 50001 bf16 48.5 / 44.2 us, 1016 of 35816 35.6 / 33.4, 5000 of 100000 425 / 397, 4000 of 14001 f32 89.3 / 87.1; but 3112 of 10848 f32
// 56.3 / 57.3, 700 of 70000 bf16 (two CTAs to an SM) 43.5 / 44.5, 1000 of 60000 f32 102.8 / 104.5.
inline bool softmax_twice_stays(int64_t row_bytes, int64_t rows, int threads, int sms) { return row_bytes < 48 * 1024 || (threads > 256 && rows < 12 * sms); }
// Whether more than an eighth of the row's work would fall behind its end if every thread took whole steps of `unroll` vectors.  f32 1000
// rows of 9000 18.7 with whole steps, 16.0 without; bf16 1000 of 65536 57 / 61.
inline bool softmax_twice_skip(int64_t vectors, int threads, int unroll) {
  const int64_t step = static_cast<int64_t>(threads) * unroll;
  return (div_up(vectors, step) * step - vectors) * 8 > vectors;
}

// Rotary embedding: how many heads a thread walks through (`blocks` blocks of 256 threads for one head group).  Few tokens: groups of four
// heads or more, as many as make two blocks per SM; the angles are computed once per group.  With a block for every second SM that
// pays for any number of heads (128 tokens of 32 x 128 bf16 6.3 in one group, 3.1 in eight), with one for nearly every SM only for many (2048 of
// 64 x 128 10.2 / 9.4, of 12 x 128 4.3 / 4.5), with more not at all (4096 of 8 x 128 4.6 / 5.3).
inline int rope_heads_per_thread(int64_t blocks, int heads, int sms) {
  if (2 * blocks > sms && (blocks > sms || heads < 24)) return heads;
  const int64_t groups = std::max<int64_t>(1, std::min<int64_t>(div_up(2 * sms, blocks), heads / 4));
  return static_cast<int>(div_up(div_up(heads, groups), 4) * 4);
}
// Little work: one or two rounds of loads to a thread, and room for all blocks at once beside those of the kernel before (rowops.cuh: kFew).
inline bool rope_few(int64_t blocks, int heads_per, int sms) { return heads_per <= 8 && blocks <= 2 * sms; }

}  // namespace route
}  // namespace tsm100
