// explicit_split.hpp -- how the fused explicit kernel (boris_tile.cuh) cuts a box
// into CTAs: the sort's tiles or work tiles made of them, and the CTAs that
// share one.
#pragma once
#include <algorithm>
#include <climits>
#include <cmath>
#include "kernels.hpp"

namespace pic {

// CTAs that share one tile's particles, of which `slots` run at once.  A box with
// fewer tiles than that would leave SMs idle: its tiles are cut into as many parts
// as still run in one wave.  `even`: larger boxes are cut too where that fills the
// last wave (the FP64 kernel, milliseconds per tile: staging a tile again costs
// nothing beside them), by the fewest parts up to 4 that leave 6% of it idle.
// At most `most`; never fewer for a larger `most`.
inline int tile_parts(const TileGeom& t, int slots, bool even, int most) {
    const int n = t.ntx * t.nty * t.ntz;
    if (n < slots) return std::min(slots / n, most);
    int best = 1;
    double full = 0;
    for (int p = 1; even && p <= std::min(4, most) && full < 0.94; ++p) {
        const double waves = (double)n * p / slots, use = waves / std::ceil(waves);
        if (use > full + 0.02) { full = use; best = p; }
    }
    return best;
}

// Two CTAs per SM run at once with FP32 particles, one with FP64 ones.
inline int explicit_slots(int preal) { return preal ? kNumSM : 2 * kNumSM; }

// CTAs per tile for so many particles in the box (LLONG_MAX: the most there can
// be).  Every CTA stages the tile's fields and flushes a block of current that the
// assembly reads again, so each gets at least 1,024 particles of an even load (two
// chunks for each of its warps), and FP32 ones, quick to push, no more than 64
// share a tile.
// us per step of 8^3 cells, FP32, with 1 / 4 / 16 / 64 / 304 CTAs:
//   1,024 particles 38 / 40 / 46 / 74 / 211    16,384: 127 / 60 / 48 / 74 / 212
//   65,536: 408 / 132 / 67 / 75 / 212         262,144: 1,524 / 415 / 139 / 94 / 218
// FP64, 152 CTAs at most: 1,024: 142 / 144 / 153 / 192 / 257
//   16,384: 1,659 / 460 / 166 / 204 / 269     262,144: 26,460 / 6,800 / 1,780 / 565 / 417
inline int explicit_parts(const TileGeom& t, int preal, long long particles) {
    const long long each = particles / ((long long)t.ntx * t.nty * t.ntz) / 1024;
    return tile_parts(t, explicit_slots(preal), preal != 0,
                      (int)std::max(1LL, std::min<long long>(each, preal ? kNumSM : 64)));
}

}  // namespace pic
