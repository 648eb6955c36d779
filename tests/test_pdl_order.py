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
