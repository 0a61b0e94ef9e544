"""CPU: kernels that start before their predecessor has ended.  What they read may still be being written until they have waited,
so every kernel waits, and none reads through the read-only path: its loads assume memory that nobody writes while the kernel
runs, and the compiler may move them over the wait."""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "causal-flare_b200", "csrc")
SOURCES = sorted(glob.glob(os.path.join(CSRC, "*.cu")) + glob.glob(os.path.join(CSRC, "*.cuh")))


def code(path):
    text = open(path).read()
    return re.sub(r"//[^\n]*|/\*.*?\*/", "", text, flags=re.S)


@pytest.mark.parametrize("path", SOURCES, ids=os.path.basename)
def test_no_load_assumes_read_only_memory(path):
    found = re.findall(r"__restrict__|__ldg\b|__ldc[sgav]\b|__ldlu\b|ld\.global\.nc\b", code(path))
    assert not found, found


@pytest.mark.parametrize("path", [p for p in SOURCES if p.endswith(".cu")], ids=os.path.basename)
def test_every_kernel_waits_before_it_reads(path):
    for part in code(path).split("__global__")[1:]:
        head, _, body = part.partition("{")
        before, wait, _ = re.split(r"\b(pdl_wait|pdl_begin)\(\)", body, maxsplit=1) if "pdl_" in body else (body, None, "")
        assert wait, head
        assert not re.search(r"\bp\.\w+\[|\*p\.|load\w*\(|load8|tma_", before), f"{head}: reads before it waits"
