"""The kernels of the gated product and the gathered ones of pairs run at their register limit (168 a
thread with 352 threads, 128 with 512); a form of the epilogue that holds more than that is compiled
without complaint, into spills."""
import os
import re
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "grouped_gemm_b200", "csrc")
NVCC = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"

SOURCE = """
#include <cuda.h>
#include "gmm_kernel.cuh"
using namespace b200gmm;
const void* kernels[] = {(const void*)gmm_kernel<kNN, 1, false, true>, (const void*)gmm_kernel<kNT, 1, false, true>,
                         (const void*)gmm_kernel<kNN, 2, false, true>, (const void*)gmm_kernel<kNT, 2, false, true>,
                         (const void*)gmm_kernel<kNN, 2, false, true, false, true>,
                         (const void*)gmm_kernel<kNT, 2, false, true, false, true>,
                         (const void*)gmm_kernel<kTN, 2, true>, (const void*)gmm_kernel<kNN, 2, true>};
"""


@pytest.mark.skipif(not os.path.exists(NVCC), reason="needs nvcc")
def test_gated_and_gathered_kernels_do_not_spill(tmp_path):
    source = tmp_path / "gated.cu"
    source.write_text(SOURCE)
    done = subprocess.run([NVCC, "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17", "-lineinfo", "-Xptxas", "-v",
                           "-I", CSRC, "-c", "-o", str(tmp_path / "gated.o"), str(source)], capture_output=True, text=True)
    assert done.returncode == 0, done.stderr
    spills = re.findall(r"Compiling entry function '(\w*gmm_kernel\w*)'.*?(\d+) bytes spill stores, (\d+) bytes spill loads",
                        done.stderr, re.S)
    assert len(spills) == 8
    assert all(stores == loads == "0" for _, stores, loads in spills), spills
