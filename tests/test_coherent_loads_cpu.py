"""Kernels that start while the grid before them still runs (launch() in common.cuh) must not read global
memory as read-only for their lifetime: neither __ldg nor const __restrict__ kernel parameters, which the
compiler turns into the same non-coherent load."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "kmeans_gb300", "csrc")
OVERLAPPED = [f for f in sorted(os.listdir(CSRC)) if f.endswith(".cu")
              and re.search(r"[^\w]launch\(", open(os.path.join(CSRC, f)).read())]


@pytest.mark.parametrize("name", OVERLAPPED + ["common.cuh"])
def test_overlapped_kernels_load_coherently(name):
    src = re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, name)).read())
    assert "__ldg" not in src and "ld.global.nc" not in src
    kernels = re.findall(r"__global__[^{;]*?\{", src)
    assert kernels or name == "common.cuh"
    for k in kernels:
        assert not re.search(r"const\s[^,()]*\*\s*__restrict__", k), k


def test_every_overlapped_kernel_waits_first():
    for name in OVERLAPPED:
        src = re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, name)).read())
        for k in re.finditer(r"__global__[^{;]*?\{(.{0,80})", src, re.S):
            assert k.group(1).lstrip().startswith("if (grid_enter()) return;"), (name, k.group(0))


def test_sources_are_found():
    assert {"update.cu", "rerank.cu", "kmeanspp.cu", "assign_bf16.cu"} <= set(OVERLAPPED)
