"""The FP32 stage kernel puts its ledger sums over a consumed update row
(csrc/stagew.cuh).  Where a lane's sums cover words that another lane reads, the
warp has to meet before they are written."""
import os
import shutil
import subprocess

import numpy as np
import pytest

import binary2d as b2
from helpers import ledger_err, make_case
from test_gpu_strips import case

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "app-binary2d_gb300", "csrc")

PROGRAM = r"""
#include <cstdio>
#include "stagew.cuh"
using namespace b2d;

// Whether a lane's sums overlap a pair that another lane reads from the update row.
template <int NF, int STORE, int COPY> bool overlaps()
{
    using T = SWShape<NF, STORE, COPY>;
    const int word = STORE == 1 ? 4 : 8;
    for (int lane = 0; lane < 32; ++lane)
        for (int m = 0; m < T::SINKS_AT; ++m) {
            const int lo = (m * 64 + 2 * lane) * 4, hi = lo + 8;
            for (int plane = 0; plane < T::NU; ++plane)
                for (int other = 0; other < 32; ++other) {
                    const int at = (plane * T::U_PITCH + T::U_FIRST + 2 * other) * word;
                    if (other != lane && lo < at + 2 * word && at < hi) return true;
                }
        }
    return false;
}

template <int NF, int STORE, int COPY> int check()
{
    const bool own = SWShape<NF, STORE, COPY>::SUMS_OVER_OWN;
    if (own != overlaps<NF, STORE, COPY>()) return 0;
    printf("NF %d STORE %d COPY %d: sums over own words only: said %d\n", NF, STORE, COPY, own);
    return 1;
}

int main()
{
    int bad = 0;
    bad += check<3, 0, COPY_WORDS>() + check<3, 0, COPY_PAIRS>() + check<4, 0, COPY_WORDS>() + check<4, 0, COPY_PAIRS>();
    bad += check<3, 1, COPY_WORDS>() + check<3, 1, COPY_PAIRS>() + check<3, 1, COPY_QUADS>();
    bad += check<4, 1, COPY_WORDS>() + check<4, 1, COPY_PAIRS>() + check<4, 1, COPY_QUADS>();
    return bad;
}
"""


def test_sums_over_other_lanes_words_are_known(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("nvcc not available")
    src, exe = tmp_path / "sums.cu", tmp_path / "sums"
    src.write_text(PROGRAM)
    subprocess.run([nvcc, "-std=c++17", "-O1", "-gencode", "arch=compute_103a,code=sm_103a", "-I", CSRC, str(src), "-o", str(exe)],
                   check=True, capture_output=True, text=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout


@pytest.mark.gpu
@pytest.mark.parametrize("nb,bs", [(3, 5), (3, 50), (2, 64)])
@pytest.mark.parametrize("variant", ["plain", "alpha_rk3", "euler"])
def test_tilings_agree_on_the_fp64_state(nb, bs, variant):
    """Chunks of one row up (sums after every row) and whole blocks: the same
    states bit for bit and the same ledgers to FP32 summation order."""
    mesh, hydro, physics, model = case(nb, bs, variant)
    cons = make_case(mesh, hydro, physics, model)[0]
    out = []
    for th in [h for h in (1, 2, 5, 25, 64) if bs % h == 0]:
        with b2.Runtime([b2.Run(mesh, hydro, physics)], precision="fp32_state64") as rt:
            rt.set_tile(0, th)
            rt.upload(0, cons)
            dts = [rt.advance(3)[0] for _ in range(2)]
            out.append((rt.download(0)[0], dts, rt.ledger(0)))
    for s, dts, led in out[1:]:
        assert np.array_equal(s, out[0][0])
        assert dts == out[0][1]
        assert ledger_err(led, out[0][2]) <= 1e-5
