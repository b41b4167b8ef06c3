"""The row pass by the number of histogram bins: its blocks per SM (compiled for the host), and
searches against the FP64 oracle, the histogram bin by bin, up to the largest number."""
import os
import shutil
import subprocess

import pytest

from tests.search_cases import make_case
from tests.search_check import search_and_check

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "cistem_downstream_bah_b200", "csrc")

PROGRAM = r"""
#include "tm_kernels.cuh"
#include <cstdio>

// the grid's blocks fit an SM's 228 KB together, and one more per SM would not (or the registers allow no more)
template <int X>
static int check() {
    using PC = tmk::PassC<X>;
    const int widths[] = {4, 8, 16};
    for (int w : widths)
        for (int bins = 1; bins <= 1024; bins++) {
            const int XP = (X / 2 + 1 + w - 1) / w * w;
            const size_t block = PC::smem_bytes(XP, bins) + 1024;
            const int n = PC::resident(XP, bins);
            if (n < 1 || n * block > 233472 || (n < PC::MIN_BLOCKS && (n + 1) * block <= 233472)) {
                std::printf("FAIL width %d, %d bins: %d blocks of %zu bytes\n", X, bins, n, block);
                return 1;
            }
            const int heights[] = {256, 288, 512, 1024};
            for (int Y : heights)
                if (PC::parts(Y, n * 148) > 1 && Y / PC::ROWS * PC::parts(Y, n * 148) > n * 148) {
                    std::printf("FAIL width %d, height %d: a divided grid of more than are resident\n", X, Y);
                    return 1;
                }
        }
    return 0;
}

int main() {
    if (check<256>() || check<512>() || check<1024>() || check<2048>() || check<4096>()) return 1;
    std::printf("OK\n");
    return 0;
}
"""


def test_blocks_of_the_row_pass_are_resident_together(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("nvcc not found")
    src = tmp_path / "resident.cu"
    src.write_text(PROGRAM)
    exe = tmp_path / "resident"
    # the header's device code is compiled for sm_100a as in the library; only host code runs
    subprocess.run([nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-std=c++17", "--extended-lambda", "-I", CSRC,
                    "-o", str(exe), str(src)], check=True, capture_output=True, timeout=600)
    out = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert out.returncode == 0 and out.stdout.strip() == "OK", out.stdout


@pytest.mark.gpu
@pytest.mark.parametrize("T,X,Y,n,bins", [(32, 256, 256, 33, 1), (32, 256, 256, 33, 860), (32, 256, 256, 33, 1024),
                                          (64, 512, 512, 17, 863), (64, 512, 512, 17, 1024), (64, 1024, 1024, 5, 1024),
                                          (128, 2048, 2048, 3, 1024)])
def test_every_number_of_bins(T, X, Y, n, bins):
    search_and_check(make_case(T=T, X=X, Y=Y, n_particles=1, n_orient=n), bins=bins)
