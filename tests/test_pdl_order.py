"""Kernels launched as programmatic dependents may start before the kernel in front of them on the stream has finished: only
after griddepcontrol.wait are its writes visible. Read from the sources, no GPU needed: a kernel that waits unconditionally
touches no global pointer before it."""

import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "decentrik_prime_b200", "csrc")


def kernels():
    """(file, kernel, parameter list, body) of every __global__ function."""
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu"))):
        text = re.sub(r"//[^\n]*", "", open(path).read())
        for m in re.finditer(r"__global__\s+void\s+(?:__launch_bounds__\([^;{]*?\)\s+)?(\w+)\s*\(([^{;]*)\)\s*\{", text):
            end = text.index("\n}", m.end())
            yield os.path.basename(path), m.group(1), m.group(2), text[m.end():end]


def body_of(name):
    return next(k[3] for k in kernels() if k[1] == name)


def waiting():
    return [k for k in kernels() if re.search(r"^  pdl_wait\(\);", k[3], re.M)]


def test_the_sources_are_understood():
    names = {k[1] for k in waiting()}
    assert {"dequant_kernel", "lora_down_kernel", "lora_shadow_kernel", "rope_kernel", "attn_fwd_kernel", "nf4_gemm_kernel"} <= names


@pytest.mark.parametrize("file,name,params,body", waiting(), ids=lambda v: v if re.fullmatch(r"\w+", v) else "")
def test_wait_comes_before_global_memory(file, name, params, body):
    before = body[:re.search(r"^  pdl_wait\(\);", body, re.M).start()]
    pointers = re.findall(r"\*\s*(?:__restrict__\s+)?(\w+)", params)
    structs = re.findall(r"(?:Params|Problem|Side)&?\s+(\w+)", params)
    for p in pointers:
        assert not re.search(rf"\b{p}\s*(\[|\+)|\*\s*{p}\b|__ldg\(\s*{p}\b", before), f"{file}: {name} reads {p} before pdl_wait()"
    for s in structs:
        assert not re.search(rf"\b{s}\.\w+\s*\[", before), f"{file}: {name} reads through {s} before pdl_wait()"


def test_the_kernel_for_middling_batches_reads_early_only_what_its_projection_does_not_write():
    """Behind a projection of the same call (p.early) its producers, tables and decoding warps go on at once and the epilogue warps
    wait before they touch the rank-16 product or an output; otherwise every warp waits before anything is read."""
    body = body_of("nf4_mid_kernel")
    roles = body.index("if (warp == 0) {")
    prologue, rest = body[:roles], body[roles:]
    waits = [m.start() for m in re.finditer(r"if \(!p\.early\)( \{\n)?\s+pdl_wait\(\);", prologue)]
    assert len(waits) == 2                                      # the table warps' and the two producers'
    assert not re.search(r"p\.(qabs|scale2|offset2|code2|mask|seg_left|seg_right|bias|out)\w*\s*(\[|\+)|tma_load", prologue[:waits[0]])
    assert prologue.index("p.code2[") > waits[0]
    late = rest.index("if (p.early) pdl_wait();")
    assert rest[:late].rstrip().endswith("if (warp >= kMidEpiWarp) {")
    assert not re.search(r"p\.(seg_left|seg_right|bias|out|out_u|out_h)\b|p\.mask\s*[+\[]", rest[:late])      # the epilogue's, all behind its wait
    # and the host says "early" only behind a projection of the same call that it has just launched
    host = open(os.path.join(CSRC, "nf4ll_gemm.cu")).read()
    assert "mid_launch(c, mp, projected && !ev0, status, stream)" in host
