"""A status word 0x1000|site says which kernel gave up a bounded wait: no two kernel files may use one site number."""
import re
from pathlib import Path

CSRC = Path(__file__).resolve().parent.parent / "tile-rs_b200" / "csrc"
WAIT = re.compile(r"(?:mbar_wait\w*|wait_counter_ge)\([^;]*?status, (\d+|kSite)( \+ \w+)?[,)]")


def sites(text):
    for base, plus in WAIT.findall(text):
        first = 63 if base == "kSite" else int(base)
        if plus.strip(" +") == "g":  # one of two query tiles
            yield from (first, first + 1)
        else:
            yield first + (int(plus.strip(" +")) if plus else 0)


def test_a_site_belongs_to_one_file():
    owner = {}
    for path in sorted(CSRC.glob("*.cuh")):
        if path.name == "ptx.cuh":
            continue
        for site in sites(path.read_text()):
            assert owner.setdefault(site, path.name) == path.name, (site, owner[site], path.name)
    assert {"attention_f32_tc.cuh", "attention_tc.cuh", "gemm_skinny.cuh", "gemm_tc.cuh", "gemm_tc2.cuh", "gemm_tf32_tc.cuh",
            "selftest.cuh"} <= set(owner.values())
    assert all(0 < site < 0x1000 for site in owner)
