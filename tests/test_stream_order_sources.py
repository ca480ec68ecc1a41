"""Kernels are launched before their predecessors on the stream have ended and wait at their top, or, for an SpMM's weights
with launch overlap on, not at all.  That is only sound for ordinary loads: the read-only path (ld.global.nc, __ldg, and what
the compiler makes of const __restrict__ kernel parameters) is for data that nobody writes during the kernel's lifetime.  A
violation is a race that hardly ever shows, so the sources are checked."""
import glob
import os
import re

import pytest

from conftest import ROOT

SOURCES = sorted(glob.glob(os.path.join(ROOT, "flash-llm_b200", "csrc", "*.cu*")))


def _code(path):
    with open(path) as f:
        text = f.read()
    return re.sub(r"//[^\n]*|/\*.*?\*/", "", text, flags=re.S)


@pytest.mark.parametrize("path", SOURCES, ids=[os.path.basename(p) for p in SOURCES])
def test_no_load_takes_the_read_only_path(path):
    code = _code(path)
    assert not re.search(r"\bld\.global\.nc\b|__ldg\s*\(", code)
    for kernel in re.finditer(r"__global__[^;{]*\{", code):
        assert "__restrict__" not in kernel.group(0), kernel.group(0)


def test_every_kernel_waits_for_its_predecessors():
    kernels = 0
    for path in SOURCES:
        code = _code(path)
        for kernel in re.finditer(r"__global__[^;{]*\{", code):
            end = code.index("\n}\n", kernel.end())
            assert "grid_dependency_wait()" in code[kernel.end():end], kernel.group(0)
            kernels += 1
    assert kernels >= 12


def test_the_streaming_epilogue_reads_bias_and_residual_behind_an_accumulator():
    """Earlier work in the stream may be writing them, and with launch overlap on the epilogue warps have not waited for it at
    the kernel's top.  A full accumulator holds products of a B that was loaded after the wait."""
    code = _code(os.path.join(ROOT, "flash-llm_b200", "csrc", "spmm_kernel_stream_sm100.cuh"))
    body = code[code.index("spmm_tcgen05_stream_kernel("):]
    epilogue = body[re.search(r"else if \(warp < kStreamFirstEpi\).*?else \{", body, re.S).end():]
    assert re.search(r"bias_of|p\.residual|load_residual|finish_columns", epilogue)
    segment = epilogue[epilogue.index("for (int row = row0"):]
    before = epilogue[:epilogue.index("for (int row = row0")] + segment[:segment.index("wait_bounded_converged(acc_full")]
    assert not re.search(r"bias_of|p\.bias|p\.residual|load_residual|finish_columns", before)
    assert re.search(r"=\s*ok \? bias_of", segment)
