"""Kernels launched as programmatic dependents read global memory with ordinary loads.

Such a kernel is alive while the kernels ahead of it still write its inputs, so the read-only path (__ldg, ld.global.nc, or a
const __restrict__ pointer, which the compiler may load through it) is not defined for them.  A stale line there
would depend on timing, so the sources are held to the rule here instead.
"""
import re

import pytest

from sharq_b200._build import CSRC

READ_ONLY = re.compile(r"__ldg\s*\(|ld\.global\.nc|__restrict__")


def _block(text, at):
    """text[at:] up to the brace that closes the first one."""
    depth = 0
    for i in range(text.index("{", at), len(text)):
        depth += {"{": 1, "}": -1}.get(text[i], 0)
        if depth == 0:
            return text[at:i + 1]
    raise AssertionError("unbalanced braces")


def _code(path):
    return re.sub(r"//[^\n]*|/\*.*?\*/", "", path.read_text(), flags=re.S)


def _functions(text):
    """The __global__ and __device__ functions with a body."""
    for m in re.finditer(r"__(?:global|device)__[^;{}]*\{", text):
        yield _block(text, m.start())


# a helper's loads run in its callers: in these files every function belongs to a kernel that waits
@pytest.mark.parametrize("name", ["prepare.cu", "prepare_device.cuh", "gemm.cu"])
def test_files_of_dependent_kernels(name):
    assert [f.split("{")[0] for f in _functions(_code(CSRC / name)) if READ_ONLY.search(f)] == []


def test_kernels_that_wait():
    seen = 0
    for path in sorted(CSRC.glob("*.cu")):
        for f in _functions(_code(path)):
            if "grid_dependency_wait" in f:
                seen += 1
                assert not READ_ONLY.search(f), (path.name, f.split("{")[0])
    assert seen >= 8  # abs / rms statistics, two prepares, the GEMM, SwiGLU, absmax partials and scaled quantisation
