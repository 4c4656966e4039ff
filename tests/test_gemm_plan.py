"""Which kernel a GEMM shape takes, from the library's own host code (compiled here, no GPU)."""
import os
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "rvllm_b200", "csrc")
NVCC = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"


@pytest.mark.skipif(not os.path.exists(NVCC), reason="no nvcc")
def test_pair_kernel_up_to_32_rows_only_where_the_split_grid_is_not_resident(tmp_path):
    """223 to 240 weight tiles, split in two: more than the three CTAs per SM; the neighbours are one wave."""
    src = tmp_path / "plan.cu"
    src.write_text('#include <stdio.h>\n#include "host_util.h"\n#include "fp8_gemm_pair.cuh"\n'
                   "int main() {\n"
                   "    for (int t = 1; t <= 1100; t++)\n"
                   "        printf(\"%d %d %d %d\\n\", t, (int)rvpair::prefer_pair(32, t * 128, 5376),\n"
                   "               (int)rvpair::prefer_pair(1, t * 128 - 127, 5376), (int)rvpair::prefer_pair(33, t * 128, 5376));\n"
                   "}\n")
    exe = str(tmp_path / "plan")
    subprocess.run([NVCC, "-gencode", "arch=compute_100a,code=sm_100a", "-std=c++17", "--expt-relaxed-constexpr", "-I", CSRC,
                    "-ccbin", "/usr/bin/g++", "-o", exe, str(src)], check=True, capture_output=True)
    rows = [tuple(map(int, line.split())) for line in subprocess.run([exe], check=True, capture_output=True, text=True).stdout.splitlines()]
    assert [t for t, at32, _, _ in rows if at32] == list(range(223, 241))
    assert all(at32 == at1 and at33 for _, at32, at1, at33 in rows)


@pytest.mark.skipif(not os.path.exists(NVCC), reason="no nvcc")
def test_tile_widths_of_the_narrow_tile_tests(tmp_path):
    """The shapes that the GPU tests run for their narrow tiles have them."""
    from tests.test_gpu_pair_widths import SHAPES
    src = tmp_path / "plan.cu"
    src.write_text('#include <stdio.h>\n#include "host_util.h"\n#include "fp8_gemm_pair.cuh"\nint main() {\n' +
                   "".join(f'    {{ auto p = rvpair::pair_plan({M}, {N}, {K}, rvpair::pair_ranges({M}, {N}, {K}));\n'
                           f'      printf("{N} {K} {M} %d %d\\n", p.bn, p.splits); }}\n' for N, K, M, _, _ in SHAPES) + "}\n")
    exe = str(tmp_path / "plan")
    subprocess.run([NVCC, "-gencode", "arch=compute_100a,code=sm_100a", "-std=c++17", "--expt-relaxed-constexpr", "-I", CSRC,
                    "-ccbin", "/usr/bin/g++", "-o", exe, str(src)], check=True, capture_output=True)
    out = subprocess.run([exe], check=True, capture_output=True, text=True).stdout
    assert [tuple(map(int, line.split())) for line in out.splitlines()] == SHAPES
