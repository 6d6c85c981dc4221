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
