"""The FP64 path's table of the buffer's rate never takes the memory that later
calls of the context need (the rule of csrc/runtime.cuh, on the CPU)."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = r"""
#include <cstdio>
#include "runtime.cuh"

int main()
{
    const size_t total = (size_t)284208 << 20;
    int kept = 0, left_out = 0;
    for (size_t nf = 3; nf <= 4; ++nf)
        for (size_t n = 64; n * n <= (size_t)1 << 31; n += 37) {
            // four slots, the background and a staging buffer; the transfers' four staging buffers
            const size_t zones = n * n, made = 6 * 8 * nf * zones, transfers = 4 * 8 * nf * zones, table = 8 * zones;
            if (made + transfers > total) continue;      // fits neither with a table nor without
            const bool keep = b2d::room_for_tables(total - made, total, table);
            (keep ? kept : left_out)++;
            if (keep && made + transfers + table > total) {
                printf("%zu^2, %zu fields: a table that leaves no room\n", n, nf);
                return 1;
            }
            if (!keep && 4 * (made + table) < total) {
                printf("%zu^2, %zu fields: left out with room to spare\n", n, nf);
                return 1;
            }
        }
    if (b2d::room_for_tables(8, 16, 9)) return 1;        // (no underflow)
    return kept && left_out ? 0 : 1;
}
"""


def test_tables_leave_room(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("nvcc not available")
    src, exe = tmp_path / "room.cu", tmp_path / "room"
    src.write_text(PROGRAM)
    subprocess.run([nvcc, "-std=c++17", "-O1", "-I", os.path.join(ROOT, "app-binary2d_gb300", "csrc"), "-I",
                    os.path.join(ROOT, "include"), str(src), "-o", str(exe)], check=True, capture_output=True, text=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
