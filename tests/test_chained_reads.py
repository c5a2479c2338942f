"""Kernels whose launches overlap read what the kernel in front writes, after a wait
on the device.  The compiler may load through a const __restrict__ pointer on a path
that is not coherent with another kernel's writes, and ahead of the wait, so in the
sources of these kernels the qualifier stands on twiddle tables alone: the copy in
shared memory (tw), and the tables of the two-factor passes (twg), which nothing
writes after a context's creation.  The Stockham passes' tables may be filled on the
same stream and carry none.  (CPU)"""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "wavedm.jl_gb300", "csrc")
STOCKHAM = ("passes.cuh", "xpass_warp.cuh", "xpass_staged.cuh", "fft_engine.cuh", "instantiate.cuh")
FACTOR = ("fft_factor.cuh", "factor_lines.cuh", "factor_rows.cuh", "factor_planes.cuh", "factor_instantiate.cuh")


@pytest.mark.parametrize("name,tables", [(f, ("tw",)) for f in STOCKHAM] + [(f, ("tw", "twg")) for f in FACTOR])
def test_only_tables_are_restrict(name, tables):
    with open(os.path.join(CSRC, name), encoding="utf-8") as f:
        text = re.sub(r"//[^\n]*", "", f.read())
    found = re.findall(r"([\w ]+)\*\s*__restrict__\s+(\w+)", text)
    assert text.count("__restrict__") == len(found)
    assert [(t, v) for t, v in found if v not in tables or t.split() != ["const", "float4"]] == []


def test_tables_go_up_on_the_stream_that_reads_them():
    """A copy on the default stream is not in front of work on the context's non-blocking stream."""
    with open(os.path.join(CSRC, "wdm_api.cu"), encoding="utf-8") as f:
        text = re.sub(r"//[^\n]*", "", f.read())
    assert re.findall(r"cudaMemcpy\([^;]*HostToDevice", text) == []
