"""Barriers in their aligned form want every lane of a warp together, which code after a branch does not promise: read from the
sources, no GPU needed, they are issued by helpers that bring the lanes together first."""

import glob
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "decentrik_prime_b200", "csrc")
ALIGNED = r"bar\.sync|bar\.arrive|barrier\.cluster\.\w+(?:\.\w+)*\.aligned"


BARRIER = r"__syncthreads\(\);|__syncwarp\(\);|named_barrier\(.*\);"


def sources():
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu*"))):
        yield os.path.basename(path), [line.split("//")[0].strip() for line in open(path)]


def test_aligned_barriers_follow_a_warp_barrier():
    seen = 0
    for name, lines in sources():
        for i, line in enumerate(lines):
            if "asm" in line and re.search(ALIGNED, line):
                seen += 1
                assert name == "nf4ll_common.cuh", f"{name}:{i + 1}"
                assert lines[i - 1] in ("__syncwarp();", "cluster_arrive();") or "_together() {" in line, f"{name}:{i + 1}"
    assert seen == 6


def test_the_form_without_one_is_used_where_lanes_are_together():
    """Right behind a barrier, or with nothing but what a whole warp does alike between: waiting for the kernel in front, a condition on the
    warp's number or the cluster's size, declarations."""
    calls = 0
    for name, lines in sources():
        for i, line in enumerate(lines):
            if name == "nf4ll_common.cuh" or not re.search(r"cluster_(arrive|wait)_together\(\);", line):
                continue
            calls += 1
            assert re.fullmatch(r"if \(cl > 1( && warp < \w+)?\) cluster_(arrive|wait)_together\(\);", line), f"{name}:{i + 1}"
            before = next(b for b in reversed([text for text in lines[:i] if text]) if b != "if (p.early) pdl_wait();")
            assert re.search(BARRIER, before) or re.fullmatch(r"if \(warp >= \w+\) \{", before), f"{name}:{i + 1}: {before}"
    assert calls == 3
