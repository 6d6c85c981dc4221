"""barrier.cluster.*.aligned is undefined for a warp whose lanes arrive one after the other: where it stands, lanes are
brought together first, and it stands in one place."""
import re
from pathlib import Path

CSRC = Path(__file__).resolve().parent.parent / "tile-rs_b200" / "csrc"


def test_aligned_cluster_barriers_follow_a_syncwarp():
    found = []
    for path in sorted([*CSRC.glob("*.cuh"), *CSRC.glob("*.cu")]):
        for m in re.finditer(r"asm volatile\(\s*\"barrier\.cluster", path.read_text()):
            found.append((path.name, path.read_text()[:m.start()].rstrip().endswith("__syncwarp();")))
    assert found == [("ptx.cuh", True)]
