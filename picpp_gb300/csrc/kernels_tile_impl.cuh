// kernels_tile_impl.cuh -- launchers of the per-tile particle kernels (fused
// explicit step, tiled implicit deposit and mover) for one particle precision
// T; instantiated by kernels_f32.cu and kernels_f64_tile.cu.
#pragma once
#include <algorithm>
#include <cmath>
#include "boris_tile.cuh"
#include "implicit_tile.cuh"
#include "kernels.hpp"

namespace pic {

template <typename T>
size_t PK<T>::tile_smem_bytes(const TileShape& sh, bool merge) {
    size_t F = (size_t)sh.fx * sh.fy * sh.fz;
    // FP32: the current block is 64-bit fixed point in two 32-bit words,
    // followed by the warps' scratch for spreading the run heads' adds
    const size_t fixed_scratch = sizeof(T) == 4 ? (size_t)(kTileThreads / 32) * kSpreadBytes : 0;
    // and every warp's staged chunk of particles
    return ((6 * F * sizeof(T) + 15) & ~size_t(15)) + ((3 * (size_t)sh.jcells * 8 + 15) & ~size_t(15)) + fixed_scratch +
           (size_t)(kTileThreads / 32) * sizeof(ChunkBuf<T>) + (merge ? sizeof(MergeTable) : 0);
}

template <typename T>
void PK<T>::push_deposit_tiled(cudaStream_t s, const GridP& g, const TileGeom& t, const TileGeom& o, const TileShape& sh,
                               const SpeciesSet<T>& S, const void* E, const void* B, double* Jpart, int parts) {
    static bool attr_set = false;
    if (!attr_set) {
        for (auto* k : {k_push_deposit_tile<T, T, 8, false, false, false>, k_push_deposit_tile<T, T, 8, false, true, false>,
                        k_push_deposit_tile<T, T, 8, false, true, true>, k_push_deposit_tile<T, T, 0, false, false, false>,
                        k_push_deposit_tile<T, T, 0, false, true, false>, k_push_deposit_tile<T, T, 0, true, false, false>,
                        k_push_deposit_tile<T, T, 0, true, true, false>})
            cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, 208 * 1024);
        attr_set = true;
    }
    const bool merge = t.tx != o.tx || t.ty != o.ty || t.tz != o.tz;   // (work_tiles: 8^3 cells)
    const bool cube8 = t.tx == 8 && t.ty == 8 && t.tz == 8 && g.y3 && g.z3 && sh.fx == 12 && sh.fy == 12 &&
                       sh.fz == 12 && sh.jx == 12 && sh.jy == 12 && sh.jz == 12;
    const int grid = std::min(t.ntx * t.nty * t.ntz * parts, kNumSM * 8);
    PushSet<T> K{};
    K.fx_scale = fixed_scale(g, S);
    K.parts = parts;
    K.dt = T(g.dt);
    K.idt = T(1.0 / g.dt);
    const double d[3] = {g.dx, g.dy, g.dz}, id[3] = {g.idx, g.idy, g.idz};
    for (int a = 0; a < 3; ++a) {
        K.d[a] = T(d[a]);
        K.id[a] = T(id[a]);
        K.hid[a] = T(0.5) * K.id[a];
    }
    const T vol = K.d[0] * K.d[1] * K.d[2];
    for (int q = 0; q < S.ns; ++q) {
        K.q[q] = S.q[q];
        K.m[q] = S.m[q];
        K.beta[q] = S.q[q] * K.dt / (T(2) * S.m[q]);
        K.fcd[q] = S.q[q] * S.w[q] / vol;
    }
    // a wall box runs its own instantiation (run-time tile shape)
    auto* whole = g.wall ? k_push_deposit_tile<T, T, 0, true, false, false>
                         : cube8 ? k_push_deposit_tile<T, T, 8, false, false, false>
                                 : k_push_deposit_tile<T, T, 0, false, false, false>;
    auto* shared = g.wall ? k_push_deposit_tile<T, T, 0, true, true, false>
                          : cube8 ? k_push_deposit_tile<T, T, 8, false, true, false>
                                  : k_push_deposit_tile<T, T, 0, false, true, false>;
    auto* kernel = merge ? k_push_deposit_tile<T, T, 8, false, true, true> : (parts > 1 ? shared : whole);
    kernel<<<grid, kTileThreads, tile_smem_bytes(sh, merge), s>>>(g, t, o, sh, S, K, (const T*)E, (const T*)B, Jpart);
}

// Fixed-point scale of the FP32 current block: the power of two with
// max_species |q w / V| * scale <= 2^35 (every zigzag term is bounded by
// q w / V because |v| < c = 1, so a run total of up to 32 terms stays below
// 2^40; a tile entry takes at most two terms per particle of the tile, and
// a cell's sum of at most 27 tile partials stays below 2^63 up to about five
// million particles per tile).
template <typename T>
float PK<T>::fixed_scale(const GridP& g, const SpeciesSet<T>& S) {
    double fmax = 0;
    for (int q = 0; q < S.ns; ++q)
        fmax = std::max(fmax, std::fabs((double)S.q[q] * (double)S.w[q] / (g.dx * g.dy * g.dz)));
    return fmax > 0 ? (float)std::ldexp(1.0, 35 - (int)std::ceil(std::log2(fmax))) : 1.0f;
}

template <typename T>
void PK<T>::assemble_j(cudaStream_t s, const GridP& g, const TileGeom& t, const TileShape& sh, const double* Jpart,
                       const double* Jfix, double* J, double inv_scale, int parts) {
    // (an axis of one cell: one tile, no halo)
    auto whole_axis = [](int n, int te, int nt) { return n == 1 || (te >= 4 && te * nt == n); };
    const bool whole = whole_axis(g.nx, t.tx, t.ntx) && whole_axis(g.ny, t.ty, t.nty) && whole_axis(g.nz, t.tz, t.ntz);
    auto* kernel = parts > 1 ? (whole ? k_assemble_j<T, true, true> : k_assemble_j<T, true, false>)
                             : (whole ? k_assemble_j<T, false, true> : k_assemble_j<T, false, false>);
    kernel<<<dim3(grid_for(g.N, 256), whole ? 3 : 1), 256, 0, s>>>(g, t, sh, Jpart, Jfix, J, inv_scale, parts);
}

template <typename T>
ImpBlock PK<T>::implicit_block(const GridP& g, const TileGeom& t, int h, bool wide) {
    ImpBlock b{};
    b.h = h;
    b.areal = wide ? sizeof(double) : sizeof(T);
    b.field = sizeof(T) == sizeof(float) ? sizeof(float4) : 3 * sizeof(double);
    b.nbx = g.nx > 1 ? t.tx + 2 * h + 1 : 1;
    b.nby = g.y3 ? t.ty + 2 * h + 1 : 1;
    b.nbz = g.z3 ? t.tz + 2 * h + 1 : 1;
    b.cbx = g.nx > 1 ? t.tx + 2 * h + 2 : 1;
    b.cby = g.y3 ? t.ty + 2 * h + 2 : 1;
    b.cbz = g.z3 ? t.tz + 2 * h + 2 : 1;
    b.NB = b.nbx * b.nby * b.nbz;
    b.CB = b.cbx * b.cby * b.cbz;
    return b;
}

template <typename T>
size_t PK<T>::implicit_tile_smem(const ImpBlock& bk, int cells, int ns) {
    // FP32 accumulators: the per-warp rows of the tensor-core run sums and
    // their 32-entry lane table; staged: every warp's next chunk of particles
    // and the particle ranges of the box's cells, of every species
    size_t n = bk.scratch_at();
    if (sizeof(T) == sizeof(float))
        n += (size_t)(imp_threads<T>() / 32) * kScrParticles * kScrRow * sizeof(float) + 32 * sizeof(TcLane);
    if (bk.stage) n += (size_t)(imp_threads<T>() / 32) * sizeof(ChunkBuf<T>) + (size_t)ns * cells * sizeof(int2);
    return n;
}

template <typename T>
void PK<T>::implicit_deposit_tiled(cudaStream_t s, const GridP& g, const TileGeom& t, const TileGeom& o, const ImpBlock& bk,
                                   const ImpSpecies<T>& S, const T* E, const T* B, double* J, double* mu,
                                   double* rho, double* Pi) {
    constexpr bool kF64 = sizeof(T) == sizeof(double);   // its kernels for boxes of one cell along z
    static bool attr_set = false;
    if (!attr_set) {
        for (auto* k : {k_implicit_deposit_tile<T, T, true, false>, k_implicit_deposit_tile<T, double, true, false>,
                        k_implicit_deposit_tile<T, T, true, kF64>, k_implicit_deposit_tile<T, T, false, false>})
            cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);
        attr_set = true;
    }
    const size_t smem = implicit_tile_smem(bk, t.tx * t.ty * t.tz, S.ns);
    const int per_sm = (int)((227 * 1024) / (smem + 1024));
    const int ntiles = t.ntx * t.nty * t.ntz;
    const int grid = ntiles < kNumSM * (per_sm > 0 ? per_sm : 1) ? ntiles : kNumSM * (per_sm > 0 ? per_sm : 1);
    constexpr int nt = imp_threads<T>();
    const bool wide = bk.areal > (int)sizeof(T);
    auto* kernel = !bk.stage      ? k_implicit_deposit_tile<T, T, false, false>
                   : wide         ? k_implicit_deposit_tile<T, double, true, false>
                   : g.z3         ? k_implicit_deposit_tile<T, T, true, false> : k_implicit_deposit_tile<T, T, true, kF64>;
    const double PI_D = 3.14159265358979323846;
    const double ivol = 1.0 / (g.dx * g.dy * g.dz);
    DepositSet<T> K{};
    for (int q = 0; q < S.ns; ++q) {
        K.beta[q] = T(0.5 * S.q[q] * g.dt / S.m[q]);
        K.m[q] = T(S.m[q]);
        K.cq[q] = S.q[q] * S.w[q] * ivol;
        K.cm[q] = -(S.w[q] * g.theta * g.dt * g.dt * 2 * PI_D * S.q[q] * S.q[q] / S.m[q]) * ivol;
    }
    kernel<<<grid, nt, smem, s>>>(g, t, o, bk, S, K, E, B, J, mu, rho, Pi);
}

template <typename T>
bool PK<T>::implicit_push_tiled(cudaStream_t s, const GridP& g, const TileGeom& t, const TileGeom& o, const ImpSpecies<T>& S,
                                const double* E, const double* B, const double* Et) {
    constexpr bool kF64 = sizeof(T) == sizeof(double);   // its kernels for boxes of one cell along z
    MoverBlock mb{};
    const int H = kMoverHalo;
    mb.nbx = g.nx > 1 ? t.tx + 2 * H + 1 : 1;
    mb.nby = g.y3 ? t.ty + 2 * H + 1 : 1;
    mb.nbz = g.z3 ? t.tz + 2 * H + 1 : 1;
    mb.cbx = g.nx > 1 ? t.tx + 2 * H + 2 : 1;
    mb.cby = g.y3 ? t.ty + 2 * H + 2 : 1;
    mb.cbz = g.z3 ? t.tz + 2 * H + 2 : 1;
    mb.NB = mb.nbx * mb.nby * mb.nbz;
    mb.CB = mb.cbx * mb.cby * mb.cbz;
    // FP32: E^theta and B^n as float4 nodes / cells, E^n as three planes
    const size_t fld = sizeof(T) == sizeof(float)
                           ? ((size_t)mb.NB + (size_t)mb.CB) * 16 + 3 * (size_t)mb.NB * sizeof(float)
                           : (6 * (size_t)mb.NB + 3 * (size_t)mb.CB) * sizeof(T);
    // after the fields every thread's staged next particle (6 values and a cell),
    // and the rows of a work box
    const int nrows = S.ns * (t.ty / o.ty) * (t.tz / o.tz);
    const size_t whole = ((fld + 15) & ~size_t(15)) + (size_t)kMoverThreads * (6 * sizeof(T) + sizeof(int));
    const size_t most_smem = whole + (3 * (size_t)nrows + 1) * sizeof(int);
    if (most_smem > 227 * 1024) return false;
    // CTAs per box (p): at least as many as run at once, and so many that the last
    // wave of them is nearly full, as long as each has enough particles to pay
    // for staging the box.  FP64 particles, ten times as long in work, are cut as
    // fine as that allows (pairs of 61x43x1: 6 CTAs per box 511 us, 25 413 us);
    // FP32 as little (40x56x56: one CTA per box 806 us, five 760 us; 64x64x16: 2
    // 475 us, 7 435 us).  192 and 4,096 particles: what a CTA moves in the time that it
    // stages its box; p goes to four waves, and a dozen more where a box is one of few.
    // us of a call (with its launch) by p, (p) the choice:
    //   FP64 32x32x1, 32 per species and cell: 1 625, 4 175, 8 102, (19) 104, 64 116
    //        16x16x16, 8: 1 1,653, 8 239, 16 137, (38) 148, 64 166;  61x43x1, 32: 1 630, 8 254, (18) 229
    //        26x20x18, 16: 1 640, 8 489, (14) 444, 64 537
    //   FP32 26x20x18, 16: 1 153, (8) 59, 16 69, 64 144;  16x16x16, 8: 1 111, 8 48, 16 43, (38) 44, 64 57
    //        39x57x53, 20: (1) 302, 2 307, 8 390;  112x51x5, 24: 1 189, (3) 104, 4 148, 8 140
    const int n = t.ntx * t.nty * t.ntz, slots = (int)std::min<size_t>(2, 228 * 1024 / (most_smem + 1024)) * kNumSM;
    long long total = 0;
    for (int q = 0; q < S.ns; ++q) total += S.p[q].n;
    int parts = n < slots ? slots / n : 1;
    const long long least = sizeof(T) == 8 ? 192 : 4096;
    double most = 0;
    for (int p = parts, limit = 4 * parts + 12; p <= limit && (sizeof(T) == 8 || most < 0.94) && (most == 0 || total / least >= (long long)n * p); ++p) {
        const double waves = (double)n * p / slots, use = waves / std::ceil(waves);
        if (use > most + 0.02 || (sizeof(T) == 8 && use >= 0.94)) { most = use; parts = p; }
    }
    const bool rows = parts > 1 || t.tx != o.tx || t.ty != o.ty || t.tz != o.tz;
    const size_t smem = rows ? most_smem : whole;
    static bool attr_set = false;
    if (!attr_set) {
        for (auto* k : {k_implicit_push_tile<T, false, false, false>, k_implicit_push_tile<T, false, true, false>,
                        k_implicit_push_tile<T, false, false, kF64>, k_implicit_push_tile<T, false, true, kF64>,
                        k_implicit_push_tile<T, true, false, false>, k_implicit_push_tile<T, true, true, false>})
            cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);
        attr_set = true;
    }
    const int per_sm = (int)((228 * 1024) / (smem + 1024));
    const int cap = kNumSM * (per_sm > 0 ? per_sm : 1);
    const int nwork = n * parts;
    // the particles it left over: one thread per mask word
    long long words = 1;
    for (int q = 0; q < S.ns; ++q) words = std::max(words, (S.p[q].n + 31) / 32);
    // the wall rules are a separate instantiation: the periodic mover keeps
    // none of their code in its loop
    auto* kernel = g.wall ? (rows ? k_implicit_push_tile<T, true, true, false> : k_implicit_push_tile<T, true, false, false>)
                   : g.z3 ? (rows ? k_implicit_push_tile<T, false, true, false> : k_implicit_push_tile<T, false, false, false>)
                          : (rows ? k_implicit_push_tile<T, false, true, kF64> : k_implicit_push_tile<T, false, false, kF64>);
    MoverSet<T> K{};
    K.dt = T(g.dt); K.eta = T(g.eta); K.edt = T(g.eta * g.dt); K.redt = T((1.0 - g.eta) * g.dt);
    K.dx2 = T(g.dx) * T(g.dx);
    K.id[0] = T(g.idx); K.id[1] = T(g.idy); K.id[2] = T(g.idz);
    for (int q = 0; q < S.ns; ++q) {
        K.beta[q] = T(0.5 * S.q[q] * g.dt / S.m[q]);
        K.qdt[q] = T(S.q[q] * g.dt);
        K.m[q] = T(S.m[q]);
    }
    kernel<<<nwork < cap || rows ? nwork : cap, kMoverThreads, smem, s>>>(g, t, o, mb, S, K, E, B, Et, parts);
    if (g.wall) k_implicit_push_deferred<T, true><<<grid_for(words, 128), 128, 0, s>>>(g, S, E, B, Et);
    else k_implicit_push_deferred<T, false><<<grid_for(words, 128), 128, 0, s>>>(g, S, E, B, Et);
    return true;
}

}  // namespace pic
