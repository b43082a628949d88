"""Programmatic dependent launch and TMEM: a kernel that allocates TMEM columns must own them before it lets its dependents
start.  A dependent's CTA on the same SM could otherwise take the columns first and hold them while it waits for this kernel
to complete, which waits for the columns: tcgen05.alloc has no time limit.  Read off the sources, because nothing of the
kind may be tried on a GPU."""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "rtp_b200", "csrc")
SOURCES = sorted(f for pat in ("*.cu", "*.cuh") for f in glob.glob(os.path.join(CSRC, pat)))


def bodies(text):
    """(name, body) of every __device__ / __global__ function."""
    text = re.sub(r"//[^\n]*|/\*.*?\*/", lambda m: " " * len(m.group()), text, flags=re.S)
    for m in re.finditer(r"__(?:device|global)__(?:\s+__launch_bounds__\([^)]*\))?[^;{]*?(\w+)\s*\([^;{]*\)\s*\{", text):
        depth, i = 1, m.end()
        while depth:
            depth += {"{": 1, "}": -1}.get(text[i], 0)
            i += 1
        yield m.group(1), text[m.end():i]


ALLOCATORS = [(os.path.basename(f), name, body) for f in SOURCES for name, body in bodies(open(f).read())
              if re.search(r"\btmem_alloc(_pair)?\(&", body)]


def test_found():
    assert {f for f, _, _ in ALLOCATORS} == {"attn_tc.cu", "flash_attn.cu", "gemm_kernel.cuh", "gemm_local.cu"}


@pytest.mark.parametrize("file,name,body", ALLOCATORS, ids=[f"{f}:{n}" for f, n, _ in ALLOCATORS])
def test_columns_are_owned_before_dependents_start(file, name, body):
    alloc = max(m.end() for m in re.finditer(r"\btmem_alloc(_pair)?\(&", body))
    triggers = [m.start() for m in re.finditer(r"\bpdl_(launch_dependents|prologue)\(", body)]
    assert triggers
    for t in triggers:
        assert alloc < t and "__syncthreads()" in body[alloc:t], f"{file}: {name} starts its dependents before it owns its TMEM"
