"""store_rows of csrc/gemm_tc.cuh, compiled with g++ against a model of the TMA store's groups: no box is written while a store may still read it, whatever
the number of boxes of the tile before and whether this tile has rows of C."""
import ctypes as C
import re
import subprocess
from pathlib import Path

import pytest

SOURCE = Path(__file__).resolve().parent.parent / "tile-rs_b200" / "csrc" / "gemm_tc.cuh"
# What lane 0 sees: it issues and waits for all stores, and its row is in every box.  A store reads until a wait says that it has done so.
MODEL = r"""
#include <algorithm>
#include <cstdint>
#include <deque>
#define __device__
#define __forceinline__ inline
using std::min;
struct CUtensorMap {};
constexpr int kBN = 256, kBoxBytes = 32 * 128;
template <typename OutT> uint32_t narrow2(uint32_t lo, uint32_t) { return lo; }
template <typename OutT> constexpr int kBoxCols = 128 / static_cast<int>(sizeof(OutT));
static uint8_t* base;
static std::deque<int> reading, open_group;   // boxes of committed stores, of the group that is not committed yet
static long long overwritten, stores, empty_groups;
inline void __syncwarp() {}
namespace ptx {
inline uint32_t smem_u32(const void* p) { return static_cast<uint32_t>(static_cast<const uint8_t*>(p) - base); }
inline void tmem_ld_32x32b_x32(uint32_t, uint32_t (&)[32]) {}
inline void tmem_ld_wait() {}
inline void st_shared_v4(uint32_t at, uint32_t, uint32_t, uint32_t, uint32_t) {
  const int box = static_cast<int>(at / kBoxBytes);
  for (const auto* q : {&reading, &open_group})
    for (int r : *q) overwritten += r == box;
}
inline void fence_proxy_async_smem() {}
inline void tma_store_3d(const CUtensorMap*, const void* src, int, int, int) { open_group.push_back(static_cast<int>(smem_u32(src) / kBoxBytes)), ++stores; }
inline void tma_store_commit() {
  if (open_group.empty()) ++empty_groups;
  reading.insert(reading.end(), open_group.begin(), open_group.end()), open_group.clear();
}
template <int N> inline void tma_store_wait_read() { while (reading.size() > N) reading.pop_front(); }
}
"""
CALLER = r"""
template <typename OutT>
static void walk(const int* row0, const int* col0, int tiles, int m, int n) {
  static uint8_t staging[2 * kBoxBytes];
  base = staging;
  reading.clear(), open_group.clear(), overwritten = stores = empty_groups = 0;
  uint32_t boxes = 0;
  for (int t = 0; t < tiles; ++t) store_rows<OutT, false>(nullptr, static_cast<OutT*>(nullptr), 0, 0u, staging, boxes, row0[t], col0[t], m, n, 0, 0);
}
extern "C" void run(int bytes, const int* row0, const int* col0, int tiles, int m, int n, long long* out) {
  if (bytes == 4) walk<float>(row0, col0, tiles, m, n);
  else walk<uint16_t>(row0, col0, tiles, m, n);
  out[0] = overwritten, out[1] = stores, out[2] = empty_groups;
}
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    body = re.search(r"template <typename OutT, bool kLoose>\n__device__ __forceinline__ void store_rows.*?\n}\n", SOURCE.read_text(), re.S).group(0)
    out = tmp_path_factory.mktemp("boxes") / "libboxes.so"
    src = out.with_suffix(".cpp")
    src.write_text(MODEL + body + CALLER)
    subprocess.run(["/usr/bin/g++", "-std=c++17", "-O1", "-w", "-shared", "-fPIC", str(src), "-o", str(out)], check=True)
    return C.CDLL(str(out))


# columns of C: one, two, three and four boxes in its last tile, f32 one to eight; rows: tiles with no row for this warp between others
@pytest.mark.parametrize("n", [8, 64, 72, 128, 136, 192, 200, 256, 264, 320, 392, 448, 512, 520])
@pytest.mark.parametrize("m", [1, 33, 129, 161, 300])
@pytest.mark.parametrize("bytes_", [2, 4])
def test_no_box_is_written_while_it_is_read(lib, bytes_, m, n):
    cols = 128 // bytes_
    for quad in range(4):
        for turn in range(4):
            # the tiles of one persistent CTA, in launch order from different starts and strides
            grid = [(r, c) for r in range(0, max(m, 513), 128) for c in range(0, n, 256)] * 3
            tiles = (grid[turn:] + grid[:turn])[::turn + 1]
            row0 = (C.c_int * len(tiles))(*[r + 32 * quad for r, _ in tiles])
            col0 = (C.c_int * len(tiles))(*[c for _, c in tiles])
            out = (C.c_longlong * 3)()
            lib.run(bytes_, row0, col0, len(tiles), m, n, out)
            want = sum(-(-min(256, n - c) // cols) for r, c in tiles if r + 32 * quad < m)
            assert list(out) == [0, want, 0], (quad, turn)
