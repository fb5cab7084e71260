"""The planes per thread that the launches choose (fit_xchunk of csrc/yee_common.cuh), compiled for the host."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

# blocks across a plane, planes, resident blocks, waves from which on it is 8 -> planes per thread
CASES = [((157, 200, 760, 6), 11),                           # 5.2 waves: the planes of fewest whole waves
         ((157, 200, 760, 3), 8),                            # S of 200^3 cells
         ((113, 170, 760, 3), 8),
         ((16, 64, 608, 6), 2),                              # one wave, as short as it can be
         ((821, 33, 608, 6), 8),
         ((1, 1, 608, 6), 1),
         ((57, 208, 608, 6), 10),
         ((1, 1, 0, 6), 8)]


def test_fit_xchunk(tmp_path):
    from opencl_fdtd_gb300 import build
    try:
        nvcc = build.nvcc()
    except RuntimeError:
        pytest.skip("nvcc not found")
    src, exe = tmp_path / "fit.cu", tmp_path / "fit"
    calls = "\n".join('printf("%%u\\n", fdtd::fit_xchunk(%d, %d, %d, %d));' % c for c, _ in CASES)
    src.write_text('#include <cstdio>\n#include "yee_common.cuh"\nint main() {\n%s\nreturn 0; }\n' % calls)
    subprocess.check_call([nvcc, "-std=c++17", "-gencode", "arch=compute_103a,code=sm_103a", "-I", build.CSRC, str(src),
                           "-o", str(exe)])
    got = [int(v) for v in subprocess.check_output([str(exe)], text=True).split()]
    assert got == [want for _, want in CASES]


def test_s_takes_eight_planes_from_three_waves_on():
    with open(os.path.join(ROOT, "opencl_fdtd_gb300", "csrc", "yee_kernels.cu")) as f:
        text = f.read()
    body = text[text.index("cudaError_t launch_poynting("):]
    assert "5ull * sm_count(), 3u)" in body[:body.index("\n}\n")]
