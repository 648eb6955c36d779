"""Barriers in their aligned form want every lane of a warp together, which code after a branch does not promise: read from the
sources, no GPU needed, they are issued by helpers that bring the lanes together first."""

import glob
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "decentrik_prime_b200", "csrc")
ALIGNED = r"bar\.sync|bar\.arrive|barrier\.cluster\.\w+(?:\.\w+)*\.aligned"


def test_aligned_barriers_follow_a_warp_barrier():
    seen = 0
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu*"))):
        lines = [line.split("//")[0].strip() for line in open(path)]
        for i, line in enumerate(lines):
            if "asm" in line and re.search(ALIGNED, line):
                seen += 1
                assert lines[i - 1] in ("__syncwarp();", "cluster_arrive();"), f"{os.path.basename(path)}:{i + 1}"
                assert os.path.basename(path) == "nf4ll_common.cuh"
    assert seen == 4
