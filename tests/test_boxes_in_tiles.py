"""boxes_in_tiles (csrc/types.cuh) against the boxes' own cells: the rule by which
FP32 sums of several tiles get FP64 accumulators.  No GPU."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CUDA = "/usr/local/cuda/include"

PROGRAM = r"""
#include "host_cuda.hpp"
#include <cstdio>
#include "types.cuh"
// n m t, the rule's answer, and whether a box holds cells of two tiles
int main() {
    for (int n = 1; n <= 48; ++n)
        for (int t = 1; t <= n; ++t) {
            if (n % t) continue;
            for (int m = 1; m <= n; ++m) {
                bool within = true;
                for (int b = 0; b < m; ++b)
                    within = within && pic::box_start(n, b, m) / t == (pic::box_start(n, b + 1, m) - 1) / t;
                std::printf("%d %d %d %d %d\n", n, m, t, (int)pic::boxes_in_tiles(n, m, t), (int)within);
            }
        }
}
"""


@pytest.fixture(scope="module")
def rows(tmp_path_factory):
    if shutil.which("g++") is None or not os.path.exists(os.path.join(CUDA, "cuda_runtime.h")):
        pytest.skip("needs g++ and the CUDA headers")
    d = tmp_path_factory.mktemp("boxes")
    (d / "boxes.cpp").write_text(PROGRAM)
    exe = str(d / "boxes")
    subprocess.run(["g++", "-std=c++20", "-w", "-pthread", "-I", os.path.join(ROOT, "tests", "cpp"), "-I", os.path.join(ROOT, "picpp_gb300", "csrc"), "-I", CUDA,
                    str(d / "boxes.cpp"), "-o", exe], check=True)
    out = subprocess.run([exe], check=True, capture_output=True, text=True).stdout
    return [tuple(int(v) for v in line.split()) for line in out.splitlines()]


def test_no_box_of_two_tiles_counts_as_within_one(rows):
    assert len(rows) > 1000
    assert not [r for r in rows if r[3] and not r[4]]
    # 15 cells in tiles of 5, cut into boxes of 3: the second box holds cells of two
    assert (15, 5, 5, 0, 0) in rows


def test_even_boxes_within_tiles_do_count(rows):
    assert all(r[3] for r in rows if r[4] and r[0] % r[1] == 0)
