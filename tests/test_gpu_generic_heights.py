"""Run-time heights where the column pass turns from column pairs with their rows of A staged in
shared memory to pairs without, and to one column: the choice (compiled for the host) and the
search against the FP64 oracle."""
import os
import subprocess

import pytest

from cistem_downstream_bah_b200.build import _cxx
from tests.search_cases import make_case
from tests.search_check import search_and_check

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "cistem_downstream_bah_b200", "csrc")

PROGRAM = r"""
#include "tm_generic_forms.h"
#include <cstdio>

int main() {
    // two columns per block for every height whose two lines of pairs fit a block's shared memory
    const int templates[] = {32, 48, 64, 128, 256, 384};
    for (int T : templates)
        for (int Y = 64; Y <= 8192; Y++) {
            const tmk::GenColForm p = tmk::gen_col_form(T, Y);
            if (p.smem > 232448) return printf("template %d, height %d: %zu bytes\n", T, Y, p.smem), 1;
            if (p.columns() < (32 * Y <= 232448 ? 2 : 1)) return printf("template %d, height %d: %d columns\n", T, Y, p.columns()), 1;
        }
    return 0;
}
"""


def test_heights_keep_two_columns_per_block(tmp_path):
    src = tmp_path / "heights.cpp"
    src.write_text(PROGRAM)
    exe = tmp_path / "heights"
    subprocess.run([_cxx(), "-std=c++17", "-I", CSRC, "-o", str(exe), str(src)], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True)
    assert out.returncode == 0, out.stdout


@pytest.mark.gpu
@pytest.mark.parametrize("T,X,Y,n", [(256, 300, 7128, 2), (256, 300, 7150, 3), (256, 300, 7200, 19), (256, 300, 7260, 2),
                                     (256, 300, 7280, 2), (384, 440, 7098, 2), (32, 66, 7260, 3)])
def test_heights_match_oracle(T, X, Y, n):
    search_and_check(make_case(T=T, X=X, Y=Y, n_particles=1, n_orient=n))
