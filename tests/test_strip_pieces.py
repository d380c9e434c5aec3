"""The ledger pieces of the FP32 kernel's strips: every piece of a block has a slot
of its own within what is allocated, and the pieces of a block cover its zones
once (the helpers of csrc/runtime.cuh, on the CPU, walked as the kernel walks)."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = r"""
#include <cstdio>
#include <set>
#include <vector>
#include "runtime.cuh"
using namespace b2d;

static int bad(const char* what, int nb, int bs, int C)
{
    printf("%s: nb %d bs %d chunks %d\n", what, nb, bs, C);
    return 1;
}

static int check(int nb, int bs, int C)
{
    const int N = nb * bs, most = most_strip_pieces(bs, nb, C);
    std::vector<std::set<int>> slots(nb * nb);
    std::vector<long long> zones(nb * nb, 0);
    for (int strip = 0; strip * STRIP_COLS < N; ++strip) {
        const int j0 = strip * STRIP_COLS, w = N - j0 < STRIP_COLS ? N - j0 : STRIP_COLS;
        for (int ti = 0; ti < C; ++ti) {
            const int i0 = chunk_start(ti, N, C), TH = chunk_start(ti + 1, N, C) - i0;
            if (TH < 1) return bad("empty chunk", nb, bs, C);
            // the kernel's sums: one per block row that the chunk meets, ended at the block's last row or its own
            int brow = i0 / bs, next = bs - i0 % bs, from = 0;
            for (int r = 0; r < TH; ++r) {
                if (r + 1 != next && r + 1 != TH) continue;
                const int nc = chunks_in_block_row(brow, bs, N, C), first = chunk_of_row(brow * bs, N, C);
                for (int b = j0 / bs; b <= (j0 + w - 1) / bs; ++b) {
                    const int piece = strip_piece(strip, ti, b, bs, nc, first);
                    if (piece < 0 || piece >= most) return bad("piece out of range", nb, bs, C);
                    if (!slots[brow * nb + b].insert(piece).second) return bad("slot written twice", nb, bs, C);
                    const int lo = b * bs > j0 ? b * bs : j0, hi = b * bs + bs < j0 + w ? b * bs + bs : j0 + w;
                    zones[brow * nb + b] += (long long)(r + 1 - from) * (hi - lo);
                }
                from = r + 1;
                ++brow;
                next += bs;
            }
        }
    }
    for (long long z : zones)
        if (z != (long long)bs * bs) return bad("zones missed", nb, bs, C);
    return 0;
}

int main()
{
    int rc = 0;
    const int shapes[][2] = {{1, 1}, {16, 1}, {1, 61}, {3, 5}, {5, 25}, {3, 50}, {2, 60}, {2, 64}, {4, 120}, {6, 64}, {1, 512}, {4, 128}, {7, 33}};
    for (const auto& s : shapes) {
        const int N = s[0] * s[1];
        for (int C = 1; C <= N; C += C < 40 ? 1 : 13) rc |= check(s[0], s[1], C);   // strip rows: any count
        for (int h = 1; h <= s[1]; ++h)
            if (s[1] % h == 0) rc |= check(s[0], s[1], N / h);                     // block-aligned heights
        rc |= check(s[0], s[1], N);
    }
    return rc;
}
"""


def test_every_piece_has_its_slot(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("nvcc not available")
    src, exe = tmp_path / "pieces.cu", tmp_path / "pieces"
    src.write_text(PROGRAM)
    subprocess.run([nvcc, "-std=c++17", "-O1", "-I", os.path.join(ROOT, "app-binary2d_gb300", "csrc"), "-I",
                    os.path.join(ROOT, "include"), str(src), "-o", str(exe)], check=True, capture_output=True, text=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
