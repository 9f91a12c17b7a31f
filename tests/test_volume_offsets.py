"""The tiled volume's offsets on the host: vol_offset is a bijection onto the
volume with vol_row_offset as its step in d, and vol_row_offset takes any int,
as planes of any slope give any disparity, without signed overflow (built with
the compiler's check for it)."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

MAIN = r"""
#include <climits>
#include <cstdio>
#include <vector>
#include "engine.h"
using namespace hbp;
int main()
{
    const int W = 21, H = 10, D = 7, TX = ceil_div(W, VT_W);
    std::vector<int> hit(volume_bytes(W, H, D), 0);
    for (int y = 0; y < VT_H * ceil_div(H, VT_H); ++y)
        for (int x = 0; x < VT_W * TX; ++x)
            for (int d = 0; d < D; ++d)
            {
                const size_t o = vol_offset(x, y, d, TX, D);
                if (o >= hit.size() || hit[o]++ || o != vol_tile_base(x, y, TX, D) + vol_row_offset(d))
                    return 1;
            }
    volatile int any[] = {INT_MIN, INT_MIN + 1, -(1 << 27), -1, 0, 1 << 26, (1 << 26) + 1, INT_MAX};
    for (int d : any)
        if (vol_row_offset(d) != (unsigned)((unsigned long long)(long long)d * VT_BYTES))
            return 2;
    return 0;
}
"""


def test_volume_offsets(tmp_path):
    nvcc = "/usr/local/cuda/bin/nvcc" if os.path.exists("/usr/local/cuda/bin/nvcc") else shutil.which("nvcc")
    if not nvcc:
        pytest.skip("no nvcc")
    src, exe = tmp_path / "offsets.cu", tmp_path / "offsets"
    src.write_text(MAIN)
    subprocess.run([nvcc, "-std=c++17", "-gencode", "arch=compute_100a,code=sm_100a",
                    "-I" + os.path.join(ROOT, "hbp-isp_b200", "csrc"), "-I" + os.path.join(ROOT, "include"),
                    "-Xcompiler", "-fsanitize=signed-integer-overflow", "-Xcompiler", "-fno-sanitize-recover=all",
                    "-Xlinker", "-lubsan", "-o", str(exe), str(src)], check=True, capture_output=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
