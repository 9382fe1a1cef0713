"""The rules of csrc/explicit_split.hpp: the CTAs that share a tile of the fused
explicit kernel have enough particles each, and a step never takes more blocks of
current than a box has room for.  No GPU."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CUDA = "/usr/local/cuda/include"

PARTS = r"""
#include "host_cuda.hpp"
#include <cstdio>
#include "explicit_split.hpp"
// preal tiles particles parts most
int main() {
    const int tiles[] = {1, 2, 3, 7, 8, 27, 64, 75, 76, 77, 100, 151, 152, 153, 180, 228, 303, 304, 305, 320, 500, 512, 561, 729, 4096, 29155};
    const long long particles[] = {0, 1, 40, 1023, 1024, 5000, 16384, 100000, 1048576, 9000000, 67108864, 537000000, 4000000000ll};
    for (int preal = 0; preal < 2; ++preal)
        for (int n : tiles)
            for (long long p : particles) {
                const pic::TileGeom t{8, 8, 8, n, 1, 1, 3, 3, 3};
                std::printf("%d %d %lld %d %d\n", preal, n, p, pic::explicit_parts(t, preal, p), pic::explicit_parts(t, preal, LLONG_MAX));
            }
}
"""


def output(tmp_path, program):
    if shutil.which("g++") is None or not os.path.exists(os.path.join(CUDA, "cuda_runtime.h")):
        pytest.skip("needs g++ and the CUDA headers")
    (tmp_path / "split.cpp").write_text(program)
    exe = str(tmp_path / "split")
    subprocess.run(["g++", "-std=c++20", "-w", "-pthread", "-I", os.path.join(ROOT, "tests", "cpp"), "-I",
                    os.path.join(ROOT, "picpp_gb300", "csrc"), "-I", CUDA, str(tmp_path / "split.cpp"), "-o", exe], check=True)
    out = subprocess.run([exe], check=True, capture_output=True, text=True).stdout
    return [tuple(int(v) for v in line.split()) for line in out.splitlines()]


def test_parts_have_particles_and_room(tmp_path):
    rows = output(tmp_path, PARTS)
    assert len(rows) == 2 * 26 * 13
    for preal, tiles, particles, parts, most in rows:
        assert 1 <= parts <= most
        assert parts == 1 or particles >= 1024 * tiles * parts
        assert tiles >= (152 if preal else 304) or tiles * parts <= (152 if preal else 304)
    # enough particles: the CTAs that run at once all have some
    assert (0, 64, 1048576, 4, 4) in rows and (1, 64, 1048576, 2, 2) in rows
    assert (0, 1, 16384, 16, 64) in rows and (1, 1, 16384, 16, 152) in rows
