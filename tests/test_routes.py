"""Which kernel a problem runs on: the host rules of csrc/route.hpp, compiled with g++ and called here."""
import ctypes as C
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "tile-rs_b200" / "csrc"
SMS = 148
SOURCE = """
#include "route.hpp"
using namespace tsm100::route;
extern "C" int attention_narrow(int d, long long kv, long long blocks, int sms) { return attention_narrow_on_tcgen05(d, kv, blocks, sms); }
extern "C" void gemm16_plan(long long m, long long n, long long k, long long batch, int sms, long long* out) {
  const Gemm16 r = gemm16(m, n, k, batch, sms);
  out[0] = r.kind, out[1] = r.rows, out[2] = r.splits, out[3] = r.k_blocks_per_cta;
}
extern "C" void gemm_f32_plan(long long m, long long n, long long k, long long batch, int aligned, int sms, long long* out) {
  const GemmF32 r = gemm_f32(m, n, k, batch, aligned != 0, sms);
  out[0] = r.kind, out[1] = r.bn, out[2] = r.splits;
}
extern "C" void pair_tiles(long long m, long long n, long long k, long long batch, int sms, long long* out) {
  const PairTiles r = gemm_f32_pair_tiles(m, n, k, batch, sms);
  out[0] = r.bn, out[1] = r.whole_tiles, out[2] = r.splits;
}
extern "C" int rope_is_few(long long blocks, int heads_per, int sms) { return rope_few(blocks, heads_per, sms); }
extern "C" int decode_chained(long long ctas, long long bytes, int sms) { return decode_is_chained(ctas, bytes, sms); }
extern "C" int early(long long b_bytes, long long ctas, int sms) { return skinny_places_early(b_bytes, ctas, sms); }
extern "C" int row_per_warp(long long span, long long rows, int sms) { return softmax_row_per_warp(span, rows, sms); }
extern "C" int cluster(long long span, long long rows, int sms) { return softmax_cluster(span, rows, sms); }
extern "C" void stream_plan(long long units, long long seq, int d, int sms, long long* out) {
  const DecodeStream r = decode_stream(units, seq, d, sms);
  out[0] = r.ctas, out[1] = r.tiles, out[2] = r.grain, out[3] = r.grains;
}
extern "C" int twice_stays(long long bytes, long long rows, int threads, int sms) { return softmax_twice_stays(bytes, rows, threads, sms); }
extern "C" int copies_pay(long long m, long long n, long long k, long long batch, int bf16) { return gemm16_copies_pay(m, n, k, batch, bf16 != 0); }
extern "C" int split_ctas(long long blocks, long long keys, int sms) { return attention_split_ctas(blocks, keys, sms); }
extern "C" int boxes(long long k, long long tiles, int sms) { return gemm16_pairs_store_boxes(k, tiles, sms); }
extern "C" int block_rows(long long rows, long long heads, long long keys, long long offset, int causal, int sms) { return attention_block_rows(rows, heads, keys, offset, causal != 0, sms); }
extern "C" int attention_f32(int d, long long keys) { return attention_f32_on_tcgen05(d, keys); }
extern "C" int rope_heads(long long blocks, int heads, int sms) { return rope_heads_per_thread(blocks, heads, sms); }
extern "C" int twice_skip(long long vectors, int threads) { return softmax_twice_skip(vectors, threads, 4); }
extern "C" int twice_threads(long long bytes, long long rows, int sms) { return softmax_twice_threads(bytes, rows, sms); }
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    out = tmp_path_factory.mktemp("routes") / "libroute.so"
    src = out.with_suffix(".cpp")
    src.write_text(SOURCE)
    subprocess.run(["/usr/bin/g++", "-std=c++17", "-O1", "-Wall", "-Werror", "-shared", "-fPIC", f"-I{CSRC}", str(src), "-o", str(out)], check=True)
    return C.CDLL(str(out))


# keys, query blocks of 256 rows -> tcgen05?  (short sequences were up to three times slower there)
@pytest.mark.parametrize("d,kv,blocks,tcgen05", [
    (64, 1, 1, False), (64, 64, 4096, False), (64, 65, 1, True), (64, 2000, 1024, True),
    (32, 64, 4096, False), (32, 128, 4096, False), (32, 129, 149, True), (32, 129, 148, False), (32, 448, 148, False), (32, 449, 1, True)])
def test_short_sequences_of_narrow_heads_stay_on_the_warp_level_kernel(lib, d, kv, blocks, tcgen05):
    assert lib.attention_narrow(d, C.c_longlong(kv), C.c_longlong(blocks), SMS) == tcgen05


PAIRS, SINGLES, FEW = 0, 1, 2


def gemm16(lib, m, n, k, batch):
    out = (C.c_longlong * 4)()
    lib.gemm16_plan(C.c_longlong(m), C.c_longlong(n), C.c_longlong(k), C.c_longlong(batch), SMS, out)
    return tuple(out)


# the few-tiles kernel, and how far it splits K
@pytest.mark.parametrize("m,n,k,batch,kind,splits", [
    (16, 16384, 4096, 1, FEW, 2), (16, 4096, 16384, 1, FEW, 8), (1, 20480, 5120, 1, FEW, 1), (1, 24576, 8192, 1, FEW, 1),
    (65, 6144, 1536, 1, FEW, 4), (192, 64, 512, 1, SINGLES, 1), (192, 64, 4096, 1, FEW, 8), (4096, 4096, 64, 1, PAIRS, 1),
    (1, 4096, 128, 1024, SINGLES, 1), (16, 4096, 64, 64, SINGLES, 1), (32, 512, 64, 1024, SINGLES, 1), (128, 64, 64, 1024, SINGLES, 1),
    (256, 256, 256, 128, PAIRS, 1), (65536, 64, 64, 1, SINGLES, 1), (65536, 64, 4096, 1, FEW, 1), (8192, 8192, 8192, 1, PAIRS, 1)])
def test_16_bit_products(lib, m, n, k, batch, kind, splits):
    plan = gemm16(lib, m, n, k, batch)
    assert plan[0] == kind and (kind != FEW or plan[2] == splits), plan


def test_16_bit_plans_fit_a_launch(lib):
    """Every CTA of a split has work, and no problem that the persistent kernels take is refused for its number of tiles."""
    import random
    rng = random.Random(5)
    size = lambda top: int(2 ** rng.uniform(0, top))  # noqa: E731
    for _ in range(20000):
        m, n, k, batch = size(20), 8 * size(17), 8 * size(14), size(31 - 0.01)
        kind, rows, splits, per = gemm16(lib, m, n, k, batch)
        tiles, kb = -(-m // rows) * -(-n // 128) * batch, -(-k // 64)
        if kind == FEW:
            assert tiles * splits <= 0x7fffffff and (splits == 1 or tiles * splits <= 2 * SMS) and (-(-kb // per) - 1) * per < kb
            assert rows == (16 if m <= 16 else 32 if m <= 32 else 64 if m <= 64 else 128)
        assert (kind == PAIRS) <= (m > 128 and n > 128)
    assert gemm16(lib, 1 << 20, 128, 8192, 1 << 20)[0] == SINGLES  # 2^33 tiles of 128 x 128


@pytest.mark.parametrize("m,n,k,batch,pays", [
    (2000, 3001, 2501, 1, True), (500, 1001, 999, 1, True), (28, 3134, 4883, 1, True),
    (2000, 3001, 17, 1, True), (8001, 10001, 7, 1, False), (2000, 3001, 33, 1, True), (8001, 1001, 33, 1, True), (2000, 3001, 65, 1, True),
    (100, 101, 103, 1, True), (64, 64, 65, 500, True), (64, 64, 65, 64, True), (64, 64, 65, 3, False),
    (1, 3001, 50001, 1, True), (30, 101, 1003, 64, True), (1, 501, 4001, 1, True), ((1 << 31) - 1, (1 << 31) - 1, (1 << 31) - 1, 1, True)])
def test_16_bit_products_of_odd_sizes(lib, m, n, k, batch, pays):
    assert lib.copies_pay(C.c_longlong(m), C.c_longlong(n), C.c_longlong(k), C.c_longlong(batch), 1) == pays


@pytest.mark.parametrize("span,rows,warp", [(10, 1, True), (128, 1, True), (129, 1, False), (256, 296, False), (256, 297, True), (257, 5000, False)])
def test_softmax_of_rows_that_start_anywhere(lib, span, rows, warp):
    assert lib.row_per_warp(C.c_longlong(span), C.c_longlong(rows), SMS) == warp


# vectors of a row, rows -> CTAs of a cluster, or 0: one CTA that reads the row twice
@pytest.mark.parametrize("span,rows,ctas", [
    (1026, 1, 2), (1026, 98, 2), (1026, 99, 0), (7501, 74, 8), (7501, 75, 0), (4098, 100, 5), (4098, 148, 0), (8192, 1, 8),
    (8193, 32, 3), (8193, 74, 0), (16384, 32, 4), (16384, 148, 0), (32000, 32, 8), (32768, 1, 8), (32769, 1, 0), (2000, 149, 0)])
def test_softmax_of_a_few_wide_rows(lib, span, rows, ctas):
    assert lib.cluster(C.c_longlong(span), C.c_longlong(rows), SMS) == ctas


@pytest.mark.parametrize("row_bytes,rows,threads", [
    (100002, 1000, 256), (100002, 296, 512), (100002, 148, 1024), (200004, 1000, 512), (600000, 1000, 1024), (1 << 32, 1000, 1024)])
def test_softmax_of_rows_read_twice(lib, row_bytes, rows, threads):
    assert lib.twice_threads(C.c_longlong(row_bytes), C.c_longlong(rows), SMS) == threads


@pytest.mark.parametrize("vectors,threads,skip", [(8192, 512, False), (8193, 512, True), (2250, 256, True), (3000, 256, False), (1026, 1024, True)])
def test_softmax_steps_behind_the_row(lib, vectors, threads, skip):
    assert lib.twice_skip(C.c_longlong(vectors), threads) == skip


@pytest.mark.parametrize("blocks,heads,per", [
    (1, 32, 4), (1, 3, 4), (1, 5, 8), (8, 32, 4), (74, 64, 16), (75, 12, 12), (75, 24, 8), (148, 64, 32), (149, 64, 64), (1184, 32, 32)])
def test_rotary_head_groups(lib, blocks, heads, per):
    assert lib.rope_heads(C.c_longlong(blocks), heads, SMS) == per


@pytest.mark.parametrize("blocks,keys,ctas", [
    (1, 1, 1), (1, 3969, 1), (1, 4095, 1), (1, 4096, 8), (64, 16384, 2), (74, 1 << 20, 2), (75, 1 << 20, 1), (9, 34000, 16), (1, 1 << 20, 148), (1 << 20, 8192, 1)])
def test_attention_steps_over_several_ctas(lib, blocks, keys, ctas):
    assert lib.split_ctas(C.c_longlong(blocks), C.c_longlong(keys), SMS) == ctas


@pytest.mark.parametrize("blocks,keys,ctas", [(1, 8191, 15), (1, 8192, 8), (4, 9030, 8), (16, 10200, 9), (64, 16384, 2), (75, 16384, 1)])
def test_attention_steps_of_long_caches(lib, blocks, keys, ctas):
    assert lib.split_ctas(C.c_longlong(blocks), C.c_longlong(keys), SMS) == ctas


@pytest.mark.parametrize("m,n,k,batch,pays", [
    (20, 320, 693, 4, True), (3, 1001, 5003, 1, True), (64, 301, 129, 1, True), (2, 4097, 129, 1, True), (64, 301, 127, 1, True), (25, 99, 501, 1, True),
    (3, 171, 8001, 1, True), (1, 511, 100001, 1, False), (10, 60, 1001, 1, True)])
def test_16_bit_products_of_odd_sizes_and_a_longer_k(lib, m, n, k, batch, pays):
    assert lib.copies_pay(C.c_longlong(m), C.c_longlong(n), C.c_longlong(k), C.c_longlong(batch), 1) == pays


@pytest.mark.parametrize("blocks,heads_per,few", [(1, 4, True), (296, 8, True), (297, 4, False), (250, 9, False), (1, 32, False)])
def test_little_rotary_work(lib, blocks, heads_per, few):
    assert lib.rope_is_few(C.c_longlong(blocks), heads_per, SMS) == few


@pytest.mark.parametrize("ctas,kib,chained", [(1, 500, True), (148, 500, True), (149, 500, False), (296, 200, False), (296, 199, True), (297, 500, True)])
def test_decode_is_placed_early_unless_some_sms_have_two_long_ctas(lib, ctas, kib, chained):
    assert lib.decode_chained(C.c_longlong(ctas), C.c_longlong(kib * 1024), SMS) == chained


@pytest.mark.parametrize("mib,ctas,early", [(128, 256, True), (256, 256, True), (126, 252, True), (125, 256, False), (256, 251, False), (200, 160, False), (64, 256, False)])
def test_few_rows_products_that_place_the_next_kernel_early(lib, mib, ctas, early):
    assert lib.early(C.c_longlong(mib << 20), C.c_longlong(ctas), SMS) == early


PLANES, FUSED, WARP, FP32 = 0, 1, 2, 3


@pytest.mark.parametrize("m,n,k,batch,aligned,kind,splits", [
    (4096, 4096, 4096, 1, 1, PLANES, None), (1999, 3001, 1501, 1, 0, PLANES, None), (1999, 3001, 255, 1, 0, FUSED, 1),
    (512, 512, 512, 1, 1, FUSED, 4), (512, 512, 512, 1, 0, FUSED, 4), (64, 64, 64, 1, 1, WARP, None), (64, 64, 63, 1, 0, FP32, None),
    (64, 64, 64, 1, 0, FUSED, 1), (1024, 1024, 156, 1, 1, FUSED, 1), (300, 300, 156, 1, 1, WARP, None),
    (1024, 1024, 1024, 1, 1, FUSED, 2), (1000, 1000, 4096, 1, 1, FUSED, 2), (900, 900, 20000, 1, 1, FUSED, 2), (64, 64, 100000, 1, 1, FUSED, 8),
    (1024, 1024, 1024, 1, 0, FUSED, 2), (64, 64, 100000, 1, 0, FUSED, 8),
    # one block of K, and one column of tiles
    (1000, 1000, 32, 1, 1, WARP, None), (1000, 1000, 36, 1, 1, FUSED, 1), (2000, 2000, 20, 1, 1, WARP, None), (4000, 4000, 32, 1, 1, FUSED, 1),
    (1029, 140, 20, 300, 1, WARP, None), (931, 16, 64, 60, 1, WARP, None), (931, 16, 68, 60, 1, FUSED, 1), (931, 68, 64, 60, 1, FUSED, 1), (931, 17, 65, 60, 0, FUSED, 1),
    (1419, 372, 680, 1, 1, FUSED, 2), (64, 64, 200, 149, 1, WARP, None), (64, 64, 200, 148, 1, FUSED, 1), (65, 64, 200, 149, 1, FUSED, 1)])
def test_f32_products(lib, m, n, k, batch, aligned, kind, splits):
    out = (C.c_longlong * 3)()
    lib.gemm_f32_plan(C.c_longlong(m), C.c_longlong(n), C.c_longlong(k), C.c_longlong(batch), aligned, SMS, out)
    assert out[0] == kind
    if kind == FUSED:
        assert out[1] in (64, 128) and out[2] == splits
        # every CTA of a cluster has work, and all clusters fit the GPU at once
        tiles = -(-m // 128) * -(-n // out[1]) * batch
        assert out[2] == 1 or tiles * out[2] <= SMS


# columns of a tile, whole tiles, pairs to each of the rest
@pytest.mark.parametrize("m,n,k,batch,want", [
    (1999, 3001, 1501, 1, (256, 74, 3)), (2048, 2048, 2048, 1, (256, 64, 1)), (512, 10880, 999, 1, (256, 74, 4)), (4096, 4096, 4096, 1, (256, 222, 2)),
    (1536, 1536, 1536, 1, (128, 72, 1)), (512, 9472, 1500, 1, (256, 74, 1)), (1999, 3001, 256, 1, (256, 96, 1)), (256, 256, 100000, 75, (256, 74, 4))])
def test_shared_tiles(lib, m, n, k, batch, want):
    out = (C.c_longlong * 3)()
    lib.pair_tiles(C.c_longlong(m), C.c_longlong(n), C.c_longlong(k), C.c_longlong(batch), SMS, out)
    assert tuple(out) == want
    kb, splits = -(-k // 32), out[2]
    assert (splits - 1) * -(-kb // splits) < kb  # every share has k-blocks
    tiles = -(-m // 256) * -(-n // out[0]) * batch
    assert (tiles - out[1]) * splits <= SMS // 2


# clusters of any size: tiles x CTAs at once, and every share has k-blocks
@pytest.mark.parametrize("m,n,k,aligned,splits", [(1900, 261, 2591, 0, 3), (549, 1064, 900, 1, 3), (341, 412, 796, 1, 5), (234, 2177, 1525, 0, 2), (330, 180, 388, 1, 7)])
def test_f32_shares_of_k(lib, m, n, k, aligned, splits):
    out = (C.c_longlong * 3)()
    lib.gemm_f32_plan(C.c_longlong(m), C.c_longlong(n), C.c_longlong(k), C.c_longlong(1), aligned, SMS, out)
    kb, tiles = -(-k // 32), -(-m // 128) * -(-n // out[1])
    assert out[0] == FUSED and out[2] == splits and tiles * splits <= SMS and (splits - 1) * -(-kb // splits) < kb


@pytest.mark.parametrize("d,keys,tc", [(128, 1, True), (96, 64, False), (96, 65, True), (64, 64, False), (64, 65, True), (32, 160, False), (32, 161, True)])
def test_f32_attention(lib, d, keys, tc):
    assert lib.attention_f32(d, C.c_longlong(keys)) == tc


# query rows of a block: one tile where all blocks of 128 rows find an SM, or the longest chain of a causal call is what counts
@pytest.mark.parametrize("rows,heads,keys,offset,causal,want", [
    (1, 1, 1, 0, 1, 128), (128, 1000, 128, 0, 1, 128), (129, 1, 129, 0, 1, 128), (256, 74, 256, 0, 0, 128), (256, 75, 256, 0, 0, 256), (838, 16, 838, 0, 1, 128),
    (512, 32, 4000, 3488, 1, 128), (2048, 12, 2048, 0, 1, 128), (4096, 256, 4096, 0, 1, 256), (300, 64, 300, 0, 0, 256), (2777, 8, 2777, 0, 0, 256), (1430, 16, 8206, 6776, 1, 256), (2482, 8, 2482, 0, 1, 128), (938, 32, 938, 0, 1, 256), (0x7fffffff, 1, 0x7fffffff, 0, 1, 256)])
def test_attention_block_rows(lib, rows, heads, keys, offset, causal, want):
    assert lib.block_rows(C.c_longlong(rows), C.c_longlong(heads), C.c_longlong(keys), C.c_longlong(offset), causal, SMS) == want


@pytest.mark.parametrize("k,tiles,want", [(8, 100000, True), (2047, 1024, True), (2048, 148, True), (2048, 149, False), (4096, 64, True), (4097, 64, False), (8192, 1024, False)])
def test_results_of_pairs_in_boxes(lib, k, tiles, want):
    assert lib.boxes(C.c_longlong(k), C.c_longlong(tiles), SMS) == want


@pytest.mark.parametrize("m,n,k,batch,pays", [(760, 144, 124, 1, True), (64, 1000, 81, 1, True), (64, 1000, 71, 1, True), (64, 1000, 47, 1, False), (74, 304, 106, 1, True), (500, 117, 72, 1, True), (100, 5, 9001, 1, True), (100, 5, 71, 1, False)])
def test_16_bit_products_of_odd_sizes_and_a_shorter_k(lib, m, n, k, batch, pays):
    assert lib.copies_pay(C.c_longlong(m), C.c_longlong(n), C.c_longlong(k), C.c_longlong(batch), 1) == pays


# caches, positions, head_dim -> CTAs, and whether a cache may be parted
@pytest.mark.parametrize("units,seq,d,ctas,parted", [
    (136, 1729, 128, 148, True), (144, 200, 128, 144, False), (296, 300, 128, 148, False), (8, 32768, 128, 0, False), (8, 32768, 64, 148, True), (64, 1, 64, 0, False), (148, 1, 64, 148, False),
    (80, 1120, 128, 0, False), (512, 600, 64, 148, True), (500, 0, 128, 0, False), (512, 100, 128, 0, False), (1 << 20, 77, 64, 148, False)])
def test_decode_as_one_stream(lib, units, seq, d, ctas, parted):
    out = (C.c_longlong * 4)()
    lib.stream_plan(C.c_longlong(units), C.c_longlong(seq), d, SMS, out)
    assert out[0] == ctas
    if ctas:
        tiles = -(-seq // (4096 // d))
        assert out[1] == tiles and out[2] == (1 if parted else tiles) and out[2] * out[3] == units * tiles and out[3] >= ctas


@pytest.mark.parametrize("kib,rows,threads,stays", [(47, 100000, 256, True), (48, 1000, 256, False), (98, 1000, 256, False), (137, 700, 512, True), (195, 5000, 512, False), (195, 1776, 512, False), (195, 1775, 1024, True)])
def test_softmax_ctas_that_stay(lib, kib, rows, threads, stays):
    assert lib.twice_stays(C.c_longlong(kib * 1024), C.c_longlong(rows), threads, SMS) == stays


@pytest.mark.parametrize("m,n,k,batch,pays", [
    (3, 123, 3313, 1, True), (1, 77, 72, 1, True), (1, 77, 71, 1, False), (1, 1, 16384, 1, True), (1, 1, 16385, 1, False), (64, 256, 48, 1, True), (64, 255, 48, 1, False), (500, 525, 33, 1, True),
    (500, 524, 33, 1, False), (2000, 3000, 16, 1, True), (2000, 3000, 15, 1, False), (1, 511, 100001, 1, False), (3, 171, 100001, 1, True)])
def test_16_bit_products_of_odd_sizes_with_one_copy(lib, m, n, k, batch, pays):
    assert lib.copies_pay(C.c_longlong(m), C.c_longlong(n), C.c_longlong(k), C.c_longlong(batch), 1) == pays


# f16 with few outputs: K only as long as sums that round toward zero do not show beside the result's own rounding
@pytest.mark.parametrize("m,n,k,batch,pays", [(3, 123, 6144, 1, True), (3, 123, 6145, 1, False), (1, 511, 16384, 1, False), (1, 512, 16384, 1, True), (3, 171, 100001, 1, True), (1, 77, 72, 1, True), (1, 511, 100001, 1, False)])
def test_f16_products_of_few_outputs(lib, m, n, k, batch, pays):
    assert lib.copies_pay(C.c_longlong(m), C.c_longlong(n), C.c_longlong(k), C.c_longlong(batch), 0) == pays


@pytest.mark.parametrize("blocks,keys,ctas", [(1, 4095, 1), (1, 4096, 8), (8, 5361, 10), (64, 7512, 2), (74, 8191, 2), (75, 8191, 1), (30, 4100, 4), (1, 8191, 15), (1, 8192, 8), (64, 16384, 2)])
def test_attention_steps_of_middling_caches(lib, blocks, keys, ctas):
    assert lib.split_ctas(C.c_longlong(blocks), C.c_longlong(keys), SMS) == ctas
