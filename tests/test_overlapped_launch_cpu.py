"""Kernels that start before the kernel in front of them has ended (common.cuh, launch_overlapped) read memory that is being
written while they run: their sources use no load that promises otherwise, and every one of them waits first."""
import re
from pathlib import Path

import pytest

KERNELS = Path(__file__).resolve().parent.parent / "ryft_b200" / "csrc" / "kernels"
SOURCES = sorted(list(KERNELS.glob("*.cu")) + list(KERNELS.glob("*.cuh")))
IN_TURN = ("gemm_simt.cu", "wide.cu")      # launched without the attribute


def code(path):
    return re.sub(r"//[^\n]*", "", path.read_text())


@pytest.mark.parametrize("path", SOURCES, ids=lambda p: p.name)
def test_no_read_only_loads(path):
    text = code(path)
    if path.name in IN_TURN:
        assert "launch_overlapped" not in text and "ProgrammaticStreamSerialization" not in text
        return
    found = re.findall(r"__ldg\b|ld\.global\.nc|__restrict__", text)
    assert not found, found


@pytest.mark.parametrize("path", [p for p in SOURCES if p.name not in IN_TURN], ids=lambda p: p.name)
def test_every_kernel_waits(path):
    for kernel in re.split(r"__global__", code(path))[1:]:
        body = kernel[kernel.index("{"):]
        wait = body.find("pdl_wait()")
        assert wait >= 0, kernel[:120]
        # nothing leaves the kernel before the wait: the kernel behind it counts on this one having waited
        assert not re.search(r"\breturn\s*;", body[:wait]), kernel[:120]
