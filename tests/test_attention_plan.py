"""Ring depth of the decode-attention kernels, from the library's own host code (compiled here, no GPU)."""
import os
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "rvllm_b200", "csrc")
NVCC = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"


@pytest.mark.skipif(not os.path.exists(NVCC), reason="no nvcc")
def test_ring_is_as_deep_as_the_ctas_that_registers_allow_permit(tmp_path):
    """Units, CTAs per SM that fit with them, CTAs that registers allow: no shallow ring for CTAs that cannot be resident."""
    src = tmp_path / "plan.cu"
    src.write_text('#include <stdio.h>\n#include "host_util.h"\n#include "paged_decode_fp8_items.cuh"\n'
                   "template <int HD, int GT, typename C> void show() {\n"
                   "    const int most = rvua::ctas_per_sm<HD, GT>();\n"
                   "    for (long long ctas = 1; ctas <= 8192; ctas++) {\n"
                   "        const int u = rvua::pick_units<C>(ctas, most);\n"
                   "        printf(\"%d %d %d %d %d\\n\", HD, GT, u, 228 * 1024 / (C::smem_bytes(u) + 1024), most);\n"
                   "    }\n}\n"
                   "template <int HD, int GT> void both() { show<HD, GT, rvua::Cfg<HD>>(); show<HD, GT, rvua::ItemCfg<HD>>(); }\n"
                   "int main() { both<128, 1>(); both<128, 4>(); both<128, 8>(); both<256, 1>(); both<256, 4>(); both<256, 8>(); both<512, 8>(); }\n")
    exe = str(tmp_path / "plan")
    subprocess.run([NVCC, "-gencode", "arch=compute_100a,code=sm_100a", "-std=c++17", "--expt-relaxed-constexpr", "-I", CSRC,
                    "-ccbin", "/usr/bin/g++", "-o", exe, str(src)], check=True, capture_output=True)
    rows = {tuple(map(int, line.split())) for line in subprocess.run([exe], check=True, capture_output=True, text=True).stdout.splitlines()}
    assert {r[:2] for r in rows} == {(128, 1), (128, 4), (128, 8), (256, 1), (256, 4), (256, 8), (512, 8)}
    assert all(fit <= most for _, _, _, fit, most in rows), sorted(rows)
    assert {u for hd, gt, u, _, _ in rows if (hd, gt) == (128, 8)} == {6}
