"""Rules that every tensor-core kernel's source keeps and that no run on a GPU can show to be broken for certain."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "vkml_b200", "csrc")
SOURCES = sorted(f for f in os.listdir(CSRC) if f.endswith((".cu", ".cuh")))


def read(name):
    with open(os.path.join(CSRC, name)) as f:
        return f.read()


@pytest.mark.parametrize("name", SOURCES)
def test_warps_meet_before_aligned_instructions(name):
    """Each .aligned instruction has the whole warp: a __syncwarp() opens the function that wraps it, or the one
    aligned instruction before it in the same function did."""
    text = read(name)
    assert not re.search(r"barrier\.cluster\.\w+(\.\w+)*\.aligned", text)
    for at in re.finditer(r'asm volatile\(\s*"tcgen05\.[^"]*\.sync\.aligned', text):
        body = text[text.rfind("__device__ __forceinline__", 0, at.start()):at.start()]
        inline = "tcgen05.wait::st" in text[at.start():at.start() + 60]  # (behind the stores that it waits for, tmem_st8)
        assert "__syncwarp();" in body or (inline and "tmem_st8(" in body), text[at.start():at.start() + 80]


@pytest.mark.parametrize("name", SOURCES)
def test_no_commit_outlives_its_cta(name):
    """A producer that fills a ring whose stages tcgen05.commit releases waits for the last of these releases too."""
    text = read(name)
    kernels = re.split(r"\n__global__ ", text)
    for kernel in kernels[1:]:
        if re.search(r"(umma_commit|commit_all<CG>)\(empty_bar\(", kernel):
            assert "drain_commits<STAGES>(empty_bar, it," in kernel, kernel[:200]
