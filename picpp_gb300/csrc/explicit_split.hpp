// explicit_split.hpp -- how the fused explicit kernel (boris_tile.cuh) cuts a box
// into CTAs: the sort's tiles or work tiles made of them, and the CTAs that
// share one.
#pragma once
#include <algorithm>
#include <cmath>
#include "../../include/picpp_gb300.h"
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

// CTAs per tile for so many particles in one (infinity: the most there can be).
// Every CTA stages the tile's fields and flushes a block of current that the assembly
// reads again, so each gets about 1,024 particles at least, two chunks for each of its
// warps (FP64, where a chunk more is 45 us: no more than that), and FP32 ones, quick
// to push, only so many that the assembly does not lose what the push gains.
// us per step of 8^3 cells, FP32, with 1 / 4 / 16 / 64 / 304 CTAs:
//   1,024 particles 38 / 40 / 46 / 74 / 211    16,384: 127 / 60 / 48 / 74 / 212
//   65,536: 408 / 132 / 67 / 75 / 212         262,144: 1,524 / 415 / 139 / 94 / 218
// FP64, 152 CTAs at most: 1,024: 142 / 144 / 153 / 192 / 257
//   16,384: 1,659 / 460 / 166 / 204 / 269     262,144: 26,460 / 6,800 / 1,780 / 565 / 417
inline int explicit_parts(const TileGeom& t, int preal, double in_tile) {
    const double most = preal ? std::floor(in_tile / 1024) + 1 : std::min(in_tile / 1024, std::sqrt(0.018 * in_tile));
    return tile_parts(t, explicit_slots(preal), preal != 0, (int)std::max(1.0, std::min(most, 2.0 * kNumSM)));
}

// Work tiles of 8^3 cells, several of the sort's tiles each, which a box may take
// where the caller left the tiles to the library and some axis is no multiple of 8
// (its default tile is then smaller).  Axes below 8 cells keep the sort's tiles: a
// work tile would wrap onto itself.  w and ws come as the sort's tiles.
inline void work_tiles(const pic_config& c, const TileGeom& t, TileGeom& w, TileShape& ws) {
    const int n[3] = {c.nx, c.ny, c.nz}, e[3] = {t.tx, t.ty, t.tz};
    bool small = false;
    for (int a = 0; a < 3; ++a) {
        if (c.tile[a] > 0 || n[a] < 8 || 8 % e[a] != 0) return;
        small = small || e[a] < 8;
    }
    if (!small || c.boundary_x != PIC_BOUNDARY_PERIODIC) return;
    w.tx = w.ty = w.tz = 8;
    w.ntx = (n[0] + 7) / 8; w.nty = (n[1] + 7) / 8; w.ntz = (n[2] + 7) / 8;
    w.lx = w.ly = w.lz = 3;
    ws.fx = ws.fy = ws.fz = ws.jx = ws.jy = ws.jz = 12;
    ws.jcells = 12 * 12 * 12;
}
inline bool has_work_tiles(const TileGeom& t, const TileGeom& w) { return w.tx != t.tx || w.ty != t.ty || w.tz != t.tz; }
inline long long tile_count(const TileGeom& t) { return (long long)t.ntx * t.nty * t.ntz; }

// Above this many of the sort's tiles (ten waves of FP32 CTAs) work tiles always are
// faster, and a partial block per tile of one or a few cells takes memory: 29,155
// tiles of 35x49x17 cells, 5 particles per species and cell, FP64: 15.3 ms for five
// steps, 4.7 ms in work tiles; 100x60x54, 9, FP32: 428 and 273 us a step.
constexpr long long kMostSmallTiles = 3000;

// How the fused kernel cuts a box for one step.
struct ExplicitSplit {
    bool work;   // work tiles rather than the sort's
    int parts;   // CTAs per tile
};

// The split for so many particles of ns species: tiles of the sort t, or work tiles w
// (the results are the same: FP32 bit for bit).  Small tiles cost their staging,
// wave after wave; work tiles cost the assembly, which finds them by a search, and
// the waves of their fullest one, since a ragged axis leaves the last ones part
// empty.  The estimates in us fit 93 boxes of 9^3 to 100x100x100 cells with 1, 6 and
// 32 particles per species and cell, each timed both ways (the better way in all but
// a few, which lose up to 14%, 13^3 FP32 with 32 37%).  us per step, tiles of
// the sort / work tiles:
//   FP32  12^3, 32: 65 / 107       20^3, 32: 92 / 129    26^3, 1: 114 / 84   26^3, 32: 150 / 203
//         44^3, 1: 101 / 81        44^3, 6: 126 / 147    60^3, 6: 252 / 233
//   FP64  20^3, 6: 164 / 329       32x32x36, 6: 433 / 755   44^3, 1: 392 / 301   60^3, 1: 897 / 553
// Axes of 9 to 12 cells, on which a work tile's block wraps onto itself: tiles of
// the sort (11^3, 6: FP32 130 / 229, FP64 402 / 893).
// CTAs per work tile: its chunks start at the sort's tiles (FP64: rows of them), so
// few particles make many chunks, and a chunk takes the FP64 pipe as long as a full
// one, FP32 ones three fifths of it and more with their particles.  The assembly reads
// every part of the tiles that may hold a cell: no more parts than the push gains
// (17^3, 1 per species and cell, FP32 with 1 / 2 / 4 / 8 / 11 CTAs: 210 / 172 / 164 / 183 /
// 207; FP64: 492 / 328 / 261 / 270 / 270).
// cells: those that may hold particles (not a wall box's columns beside them).
inline ExplicitSplit explicit_split(const TileGeom& t, const TileGeom& w, long long cells, int preal, int ns,
                                    long long particles) {
    const double in_small = (double)particles * t.tx * t.ty * t.tz / cells;
    const int pt = explicit_parts(t, preal, in_small);
    if (!has_work_tiles(t, w) || ns == 0) return {false, pt};
    const int n[3] = {t.tx * t.ntx, t.ty * t.nty, t.tz * t.ntz}, nw[3] = {w.ntx, w.nty, w.ntz};
    double cover = 1;   // work tiles whose blocks hold a cell
    bool wraps = false;
    for (int a = 0; a < 3; ++a) {
        wraps = wraps || (n[a] % 8 != 0 && n[a] < 13);
        cover *= 12.0 * nw[a] / n[a];
    }
    const double push = preal ? 0.11 : 0.0105, stage = preal ? 27 : 7;   // a CTA's us per particle and per tile
    const double search = preal ? 20 : 4, read = preal ? 0.7 : 0.5;      // the assembly's, and its per block read
    // a full work tile's particles, and what its chunks amount to in particles
    const int cut = preal ? 8 * t.ty * t.tz : t.tx * t.ty * t.tz;   // cells from which its chunks are cut
    const double full = 512.0 * particles / cells;
    const double chunks = ns * (512 / cut) * std::max(1.0, full / ns * cut / 512 / 32 + 0.5);
    const double load = std::max(full, preal ? 32 * chunks : 0.6 * 32 * chunks + 0.4 * full);
    const double most = std::min(load / (preal ? 512 : 1024), std::sqrt(push * load / (read * cover)));
    const int pw = tile_parts(w, explicit_slots(preal), preal != 0, std::max(1, (int)std::min(most, 152.0)));
    if (tile_count(t) > kMostSmallTiles) return {true, pw};
    if (wraps) return {false, pt};
    const double small = std::max(1.0, (double)tile_count(t) * pt / explicit_slots(preal)) * (stage + push * in_small / pt);
    // (the ragged tiles' FP32 CTAs run beside the others)
    const double ctas = (preal ? (double)tile_count(w) : (double)(n[0] / 8) * (n[1] / 8) * (n[2] / 8)) * pw;
    const double merged = search + read * cover * pw +
                          std::max(1.0, std::ceil(ctas / explicit_slots(preal))) * push * (preal ? load : full) / pw;
    return merged < small ? ExplicitSplit{true, pw} : ExplicitSplit{false, pt};
}

// FP64 numbers that the partial blocks of any step may take.
inline size_t partial_cells(const TileGeom& t, const TileShape& ts, const TileGeom& w, const TileShape& ws, int preal) {
    const int slots = explicit_slots(preal);
    const size_t merged = has_work_tiles(t, w) ? 3 * (size_t)ws.jcells * tile_count(w) * tile_parts(w, slots, preal != 0, 152) : 0;
    if (merged && tile_count(t) > kMostSmallTiles) return merged;
    return std::max<size_t>(merged, 3 * (size_t)ts.jcells * tile_count(t) * explicit_parts(t, preal, HUGE_VAL));
}

}  // namespace pic
