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
                std::printf("%d %d %lld %d %d\n", preal, n, p, pic::explicit_parts(t, preal, (double)p / n),
                            pic::explicit_parts(t, preal, HUGE_VAL));
            }
}
"""

WORK = r"""
#include "host_cuda.hpp"
#include <cstdio>
#include "explicit_split.hpp"
// preal nx ny nz particles, work tiles taken, CTAs per tile, numbers of the step's partial
// blocks, room for them
int main() {
    const int axes[] = {8, 9, 11, 12, 13, 15, 17, 20, 26, 30, 33, 44, 50, 60, 96, 100, 255};
    const long long particles[] = {0, 1, 300, 5000, 60000, 700000, 8000000, 100000000};
    for (int preal = 0; preal < 2; ++preal)
        for (int nx : axes) for (int ny : axes) for (int nz : axes) {
            pic_config c{};
            c.nx = nx; c.ny = ny; c.nz = nz;
            c.boundary_x = PIC_BOUNDARY_PERIODIC;
            const int n[3] = {nx, ny, nz};
            int e[3];
            for (int a = 0; a < 3; ++a) e[a] = n[a] % 8 == 0 ? 8 : (n[a] % 4 == 0 ? 4 : (n[a] % 2 == 0 ? 2 : 1));
            const pic::TileGeom t{e[0], e[1], e[2], nx / e[0], ny / e[1], nz / e[2], 0, 0, 0};
            pic::TileShape ts{}, ws{};
            ts.jcells = (long long)(e[0] + 4) * (e[1] + 4) * (e[2] + 4);
            pic::TileGeom w = t;
            ws = ts;
            pic::work_tiles(c, t, w, ws);
            for (long long p : particles) {
                const pic::ExplicitSplit x = pic::explicit_split(t, w, (long long)nx * ny * nz, preal, 2, p);
                std::printf("%d %d %d %d %lld %d %d %lld %lld\n", preal, nx, ny, nz, p, (int)x.work, x.parts,
                            3 * (x.work ? ws : ts).jcells * pic::tile_count(x.work ? w : t) * x.parts,
                            (long long)pic::partial_cells(t, ts, w, ws, preal));
            }
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
        assert parts == 1 or particles >= 1024 * tiles * (parts - preal)
        assert tiles >= (152 if preal else 304) or tiles * parts <= (152 if preal else 304)
    # enough particles: the CTAs that run at once all have some
    assert (0, 64, 1048576, 4, 4) in rows and (1, 64, 1048576, 2, 2) in rows
    assert (0, 1, 16384, 16, 304) in rows and (1, 1, 16384, 17, 152) in rows and (0, 1, 67108864, 304, 304) in rows


def test_work_tiles_where_they_pay_and_room_for_either(tmp_path):
    rows = output(tmp_path, WORK)
    assert len(rows) == 2 * 17 ** 3 * 8
    for preal, nx, ny, nz, particles, take, parts, numbers, room in rows:
        assert parts >= 1 and numbers <= room
        assert not (take and nx % 8 == ny % 8 == nz % 8 == 0)
        # the memory of single-cell tiles is bounded: as many numbers as 3,000 tiles take
        # whose blocks and CTAs are the largest, or three blocks of 12^3 for each 8^3 cells
        tiles = ((nx + 7) // 8) * ((ny + 7) // 8) * ((nz + 7) // 8)
        assert room <= 3 * 1728 * max(4 * tiles, 3000, 304)
    took = {r[:5]: r[5] for r in rows}
    # measured faster in work tiles, and in the sort's
    assert took[0, 33, 33, 33, 60000] and took[1, 33, 33, 33, 60000] and took[1, 60, 60, 60, 700000]
    assert not took[0, 20, 20, 20, 60000] and not took[1, 20, 20, 20, 60000] and not took[0, 9, 9, 9, 5000]
    assert took[0, 26, 26, 26, 5000] and not took[0, 26, 26, 26, 8000000]
