"""Registers and spills of kernels whose resident CTAs, or whose inner loops, depend on them: as the compiler reports them
(`-Xptxas -v`) when it compiles the sources for sm_100a.  No GPU is needed."""

import os
import re
import shutil
import subprocess

import pytest

from mlstm_kernels_b200 import build

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "mlstm_kernels_b200", "csrc")

pytestmark = pytest.mark.skipif(shutil.which("nvcc") is None and not os.path.exists("/usr/local/cuda/bin/nvcc"), reason="no CUDA compiler")


def report(source):
    """{kernel with its template arguments: (registers, bytes of spill stores and loads)}"""
    flags = [f for f in build.NVCC_FLAGS if f != "--use_fast_math=false"]
    text = subprocess.run([build._nvcc(), *flags, "-Xptxas=-v", "-c", os.path.join(CSRC, source), "-o", os.devnull], capture_output=True,
                          text=True, check=True).stderr
    text = subprocess.run(["c++filt"], input=text, capture_output=True, text=True, check=True).stdout
    found = re.findall(r"Compiling entry function '(?:void )?mlstm::(?:\(anonymous namespace\)::)?(\w+(?:<[^(]*>)?)\(.*?"
                       r"(\d+) bytes spill stores, (\d+) bytes spill loads.*?Used (\d+) registers", text, re.S)
    return {name: (int(regs), int(stores) + int(loads)) for name, stores, loads, regs in found}


@pytest.mark.parametrize("source,least", [("chunkwise_sm100.cu", 16), ("chunkwise_bw_sm100.cu", 2)])
def test_tcgen05_kernels_do_not_spill(source, least):
    """(A local-memory access is a trip to L2 here: nearly all of L1 is shared memory.)"""
    kernels = report(source)
    assert len(kernels) >= least
    assert {name: x for name, x in kernels.items() if x[1] > 0} == {}


def test_portable_recurrence_without_score_blocks_keeps_its_resident_ctas():
    """Four CTAs of 256 threads, and twelve of 128 in the scan, to an SM of 65536 registers."""
    kernels = report("chunkwise_simt.cu")
    parts = {name: x[0] for name, x in kernels.items() if re.fullmatch(r"part_kernel<\w+, \w+, false>", name)}
    scans = {name: x[0] for name, x in kernels.items() if re.fullmatch(r"rec_scan_kernel<\d, (true, false|false, true)>", name)}
    assert len(parts) == 6 and len(scans) == 4
    assert max(parts.values()) <= 64 and max(scans.values()) <= 40
