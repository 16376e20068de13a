"""What a relaxed mbarrier arrival may hand over (csrc/cuda): tensor memory that tcgen05.wait::ld has emptied, nothing else.  A buffer
that loads or bulk copies fill again needs the release of a plain arrival behind the reads."""
import glob
import os
import re

CUDA = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "fastface_b200", "csrc", "cuda")


def test_relaxed_arrivals_are_for_accumulators():
    uses = []
    for path in sorted(glob.glob(os.path.join(CUDA, "*.cu*"))):
        for line in open(path):
            for m in re.finditer(r"\bmbar_arrive_(?:relaxed|cluster)\((?!uint32_t)(.*)", line):
                uses.append((os.path.basename(path), m.group(1)))
    assert len(uses) >= 3
    assert all("acc_empty" in what for _, what in uses), uses
