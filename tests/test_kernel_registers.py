"""Registers of the general path's flux kernels: the batches of limiter quotients
(kFluxBatch, kRowBatch in e4c_cells.cuh) are as wide as keeps the resident
warps the kernels need, 4 CTAs of 128 threads per SM for the one-thread-per-face
kernel and 3 for the row walk (65,536 registers per SM, given out to warps in
units of 256), with no more than a few bytes of spills."""
import os
import re
import shutil
import subprocess

import pytest

from eilmer4_b200 import build

SOURCE = """
#include "e4c_internal.h"
#include "e4c_cells.cuh"
namespace e4c {
#define ROWS(F, M) template __global__ void k_flux_rows<1, F, 0, M, kRowBatch>(BlockView, const SimDev*, FluxOpts, int3);
ROWS(0, false) ROWS(1, true) ROWS(3, true)
template __global__ void k_flux<1, 1, 0>(BlockView, const SimDev*, FluxOpts, int);
template __global__ void k_flux<1, 3, 0>(BlockView, const SimDev*, FluxOpts, int);
}
"""


@pytest.mark.skipif(shutil.which(build.nvcc()) is None, reason="needs nvcc")
def test_flux_kernels_keep_their_resident_warps(tmp_path):
    src = tmp_path / "flux.cu"
    src.write_text(SOURCE)
    flags = dict(build.UNITS)["e4c_general.cu"]
    out = subprocess.run([build.nvcc(), *build.ARCH, *build.COMMON, *flags, "-Xptxas", "-v", "-c",
                          str(src), "-o", os.devnull], capture_output=True, text=True)
    assert out.returncode == 0, out.stderr
    found = re.findall(r"Compiling entry function '(\w+)'.*?(\d+) bytes spill stores.*?"
                       r"Used (\d+) registers", out.stderr, re.S)
    assert len(found) == 5, out.stderr
    for name, spill, regs in found:
        assert int(spill) <= 16, (name, spill)
        per_warp = -(-int(regs) * 32 // 256) * 256
        ctas = 65536 // (4 * per_warp)
        assert ctas >= (3 if "k_flux_rows" in name else 4), (name, regs, ctas)
