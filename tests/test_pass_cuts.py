"""How the resize passes of a launch are cut into CTAs (csrc/kernels.h), without a GPU."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = """
#include <cstdio>
#include "%s/datago_b200/csrc/kernels.h"
int main() {
    for (int vertical = 0; vertical < 2; ++vertical) {
        dg::ConvPass p[8] = {};
        unsigned tiles = 0;
        for (auto& q : p) { q.out_w = 1600; q.out_h = 1200; q.channels = 3; q.fast = 2; }
        dg::cut_pass_tiles(p, 8, vertical != 0);
        for (auto& q : p) tiles += dg::conv_tiles(q, vertical != 0);
        std::printf("%%u ", tiles);
    }
}
"""


@pytest.mark.parametrize("per_sm", [2, 3])
def test_ctas_follow_the_resident_places(tmp_path, per_sm):
    (tmp_path / "cuts.cpp").write_text(PROGRAM % ROOT)
    cuda = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    exe = str(tmp_path / "cuts")
    subprocess.run(["g++", "-std=c++17", "-I", os.path.join(cuda, "include"), "-DDG_HMMA_CTAS=%d" % per_sm, str(tmp_path / "cuts.cpp"), "-o", exe], check=True)
    horizontal, vertical = map(int, subprocess.run([exe], capture_output=True, text=True, check=True).stdout.split())
    # 8 passes of 75 strips x 38 chunks and of 19 row groups x 75 chunks: about two CTAs per resident place (whole chunks: up to 2.75)
    assert 1.7 * 148 * per_sm <= horizontal <= 2.75 * 148 * per_sm
    assert 1.7 * 148 * 2 <= vertical <= 2.3 * 148 * 2
