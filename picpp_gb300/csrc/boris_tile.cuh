// boris_tile.cuh -- fused gather + Boris push + zigzag deposit, one CTA per
// tile of cells (the whole-step path of the explicit Buneman/Tristan solver); in
// small boxes several CTAs share a tile, along axes that 8 does not divide a CTA
// takes a work tile made of several (kParts, kMerge).
//
// Particles are ordered by a tile-major cell key (sort.cuh), so tile t owns
// the contiguous range [off[t*T3], off[(t+1)*T3]) of every species.  A CTA
//   1. stages the six Yee components of the tile plus two cells of halo in
//      shared memory: the gather of a particle in cell c reads nodes c, c+1
//      and cell centres c-1..c+1, so particles up to one cell outside their
//      tile (drift since the last sort) still gather from shared memory;
//   2. walks the tile's particles in chunks of 32 consecutive particles per
//      warp (coalesced loads and stores) and pushes them.  The zigzag current
//      of a particle is two segments, each with 12 terms at fixed positions
//      relative to one cell: the segment from the old position to the relay
//      point (in the old cell) and the one from the relay point to the new
//      position (in the new cell).  Lanes holding the same cell (particles
//      are sorted by cell) sum each segment's 12 values with a segmented
//      shuffle reduction, and the run totals go into a shared-memory current
//      block (tile plus two cells of halo).  FP32 particles: the block is
//      exact 64-bit fixed point in two 32-bit words per entry, added with
//      native 32-bit integer shared atomics (FP32 shared atomics are
//      compare-and-swap loops that collapse under address conflicts), the
//      adds of a warp's run heads spread over its lanes; the block sums are
//      exact and order-independent.  FP64 particles: FP64 shared atomics.
//      Each warp copies its next chunk of particles into shared memory with
//      cp.async while it pushes the current one;
//   3. writes the block, unreduced, to a per-tile partial buffer (for FP32
//      particles the exact fixed-point sums as 64-bit integers).
// k_assemble_j then sums the partials of every cell in a fixed order into
// the FP64 current grid (FP32 particles: exact integer sums, scaled once):
// no global floating-point atomics on the fast path.
// A particle more than one cell outside its tile, or whose zigzag segments
// leave the tile's current block, is left to k_push_deposit_deferred: the
// fused kernel sets its bit in a per-species mask and the deferred pass
// pushes it with the global gather and/or deposits its current with FP64
// global atomics into a correction grid.  The fused kernel itself calls no
// function out of line (a call site costs its hot loop register spills).
#pragma once
#include "boris.cuh"
#include "types.cuh"
#include <type_traits>

namespace pic {

#ifndef PIC_TILE_THREADS
#define PIC_TILE_THREADS 512   // threads per CTA of the fused explicit kernel (64 registers at 2 CTAs/SM)
#endif
constexpr int kTileThreads = PIC_TILE_THREADS;
#ifndef PIC_TILE_MIN_BLOCKS
#define PIC_TILE_MIN_BLOCKS 2   // CTAs per SM the register budget is sized for
#endif
// FP64: one CTA per SM (its blocks fill the shared memory), so 128 registers
template <typename TP>
__host__ __device__ constexpr int tile_ctas() { return sizeof(TP) == sizeof(float) ? PIC_TILE_MIN_BLOCKS : 1; }

template <typename TP>
__device__ __forceinline__ TP lerp(TP a, TP b, TP w) { return fmadd<TP>(w, subr<TP>(b, a), a); }

// Trilinear value of one staggered component from the staged block: base is
// the block index of the lower corner, sy/sz the strides, (wx, wy, wz) the
// weights of the upper corner.
template <typename TP, typename TF>
__device__ __forceinline__ TP tri(const TF* __restrict__ F, int base, int sy, int sz, TP wx, TP wy, TP wz) {
    TP v000 = TP(F[base]), v100 = TP(F[base + 1]);
    TP v010 = TP(F[base + sy]), v110 = TP(F[base + sy + 1]);
    TP v001 = TP(F[base + sz]), v101 = TP(F[base + sz + 1]);
    TP v011 = TP(F[base + sy + sz]), v111 = TP(F[base + sy + sz + 1]);
    TP a = lerp(lerp(v000, v100, wx), lerp(v010, v110, wx), wy);
    TP b = lerp(lerp(v001, v101, wx), lerp(v011, v111, wx), wy);
    return lerp(a, b, wz);
}

// FP32: the interpolations along x and along y two at a time (packed FP32
// operations, each rounded as the single ones: 8 instructions for 14; the kernel
// issues 81% of the time: 128^3, 2,307 -> 2,283 us, 32^3, 57.2 -> 55.7 us).
__device__ __forceinline__ unsigned long long pack2(float a, float b) {
    unsigned long long r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ unsigned long long lerp2(unsigned long long a, unsigned long long b, unsigned long long w) {
    unsigned long long d, r;
    asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(b), "l"(a));
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(w), "l"(d), "l"(a));
    return r;
}
template <>
__device__ __forceinline__ float tri<float, float>(const float* __restrict__ F, int base, int sy, int sz, float wx,
                                                   float wy, float wz) {
    const float* f = F + base;
    const unsigned long long w = pack2(wx, wx);
    // (y, z) corners (0,0) with (0,1), then (1,0) with (1,1)
    const unsigned long long y0 = lerp2(pack2(f[0], f[sz]), pack2(f[1], f[sz + 1]), w);
    const unsigned long long y1 = lerp2(pack2(f[sy], f[sy + sz]), pack2(f[sy + 1], f[sy + sz + 1]), w);
    const unsigned long long z = lerp2(y0, y1, pack2(wy, wy));
    float a, b;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(z));
    return lerp(a, b, wz);
}

// FP64: an offset within 2^-33 of its cell's lower face or 2^-21 of the upper one.
// The zigzag split asks on which side of the face the old position, taken back
// from the new one, lies; for a particle that started on the face the answer is
// in the last bit, and the fused multiply-adds here round it another way than
// the separate operations of the phase calls and the oracle.  The deferred pass,
// compiled with separate operations, takes these particles (a few per million of a
// thermal plasma; one electron on the other side moved E of a 64^3 box by 2e-8).
// FP32: the roundings are fixed.
__device__ __forceinline__ bool near_face(double u) {
    const int h = __double2hiint(u);
    return h < 0x3de00000 || h >= 0x3fefffff;
}
// Of a load on a lattice they may be all.  A chunk takes as long here with one
// particle as with 32, and the deferred pass about as long per particle: from a sixth
// of the lanes on it takes the chunk (64^3, 8 per species and cell, a step with no
// particle on a face 3.6 ms; seven of eight on one 7.5 ms with the others pushed here,
// 5.5 ms so; 7.5 ms in the separately rounded fused kernel that this one replaced).
constexpr int kNearMin = 6;

// tri at node (i, j, k) of a global grid (periodic).
template <typename TP, typename TF>
__device__ __forceinline__ TP tri_global(const GridP& g, const TF* __restrict__ F, int i, int j, int k, TP wx, TP wy, TP wz) {
    const int di = 1, dj = g.y3 ? 1 : 0, dk = g.z3 ? 1 : 0;
    auto at = [&](int a, int b, int c) { return TP(F[linw(g, i + a, j + b, k + c)]); };
    const TP a = lerp(lerp(at(0, 0, 0), at(di, 0, 0), wx), lerp(at(0, dj, 0), at(di, dj, 0), wx), wy);
    const TP b = lerp(lerp(at(0, 0, dk), at(di, 0, dk), wx), lerp(at(0, dj, dk), at(di, dj, dk), wx), wy);
    return lerp(a, b, wz);
}
// The fused kernel's gather from the global grids, in its order of operations.
template <typename TP, typename TF>
__device__ __forceinline__ void tri_gather(const GridP& g, int cell, TP ox, TP oy, TP oz, const TF* __restrict__ E,
                                           const TF* __restrict__ B, TP e[3], TP b[3]) {
    int i, j, k;
    decode(g, cell, i, j, k);
    const bool ey = g.y3, ez = g.z3;
    const int ci = ox < TP(0.5) ? i - 1 : i, cj = ey && oy < TP(0.5) ? j - 1 : j, ck = ez && oz < TP(0.5) ? k - 1 : k;
    const TP wcx = ox < TP(0.5) ? ox + TP(0.5) : ox - TP(0.5);
    const TP wcy = ey ? (oy < TP(0.5) ? oy + TP(0.5) : oy - TP(0.5)) : TP(0);
    const TP wcz = ez ? (oz < TP(0.5) ? oz + TP(0.5) : oz - TP(0.5)) : TP(0);
    const TP wny = ey ? oy : TP(0), wnz = ez ? oz : TP(0);
    e[0] = tri_global<TP, TF>(g, E, ci, j, k, wcx, wny, wnz);
    e[1] = tri_global<TP, TF>(g, E + g.N, i, cj, k, ox, wcy, wnz);
    e[2] = tri_global<TP, TF>(g, E + 2 * g.N, i, j, ck, ox, wny, wcz);
    b[0] = tri_global<TP, TF>(g, B, i, cj, ck, ox, wcy, wcz);
    b[1] = tri_global<TP, TF>(g, B + g.N, ci, j, ck, wcx, wny, wcz);
    b[2] = tri_global<TP, TF>(g, B + 2 * g.N, ci, cj, k, wcx, wcy, wnz);
}

// The 24 zigzag terms of a particle straight into the FP64 correction grid.
template <typename TP>
__device__ __forceinline__ void deposit_global(const GridP& g, TP fcd, TP ox, TP oy, TP oz, const TP v[3], int ni,
                                               int nj, int nk, double* __restrict__ Jfix) {
    zigzag_terms<TP>(g, fcd, ox, oy, oz, v, [&](int comp, int di, int dj, int dk, TP val) {
        atomicAdd(&Jfix[comp * g.N + linw(g, ni + di, nj + dj, nk + dk)], double(val));
    }, g.wall && ni == kTristanWallNode);
}

// Sets the bits of a warp's chunk of particles s0 .. s0 + 31 (bit l for
// particle s0 + l) in a particle bit mask.
__device__ __forceinline__ void set_defer_bits(unsigned* __restrict__ mask, long long s0, unsigned bits) {
    if (!bits) return;
    const long long w = s0 >> 5;
    const int sh = (int)(s0 & 31);
    atomicOr(&mask[w], bits << sh);
    if (sh && (bits >> (32 - sh))) atomicOr(&mask[w + 1], bits >> (32 - sh));
}

// One zigzag segment's 12 terms relative to its cell
// (momentum_collecting.cpp:200-230): Jx at (c, j+dj, k+dk) -> slot 2dk+dj,
// Jy at (i+di, c, k+dk) -> 4+2dk+di, Jz at (i+di, j+dj, c) -> 8+2dj+di.
template <typename TP>
__device__ __forceinline__ void segment_factors(TP Fx, TP Fy, TP Fz, TP Wx, TP Wy, TP Wz, TP b[12], TP f[12]) {
    const TP ux = subr<TP>(TP(1), Wx), uy = subr<TP>(TP(1), Wy), uz = subr<TP>(TP(1), Wz);
    b[0] = b[2] = mulr<TP>(Fx, uy); b[1] = b[3] = mulr<TP>(Fx, Wy);
    b[4] = b[6] = mulr<TP>(Fy, ux); b[5] = b[7] = mulr<TP>(Fy, Wx);
    b[8] = b[10] = mulr<TP>(Fz, ux); b[9] = b[11] = mulr<TP>(Fz, Wx);
    f[0] = f[1] = f[4] = f[5] = uz; f[2] = f[3] = f[6] = f[7] = Wz;
    f[8] = f[9] = uy; f[10] = f[11] = Wy;
}
template <typename TP>
__device__ __forceinline__ void segment_slots(TP Fx, TP Fy, TP Fz, TP Wx, TP Wy, TP Wz, TP a[12]) {
    TP b[12], f[12];
    segment_factors<TP>(Fx, Fy, Fz, Wx, Wy, Wz, b, f);
#pragma unroll
    for (int q = 0; q < 12; ++q) a[q] = mulr<TP>(b[q], f[q]);
}
// ... added to the terms in a[].
template <typename TP>
__device__ __forceinline__ void segment_add(TP Fx, TP Fy, TP Fz, TP Wx, TP Wy, TP Wz, TP a[12]) {
    TP b[12], f[12];
    segment_factors<TP>(Fx, Fy, Fz, Wx, Wy, Wz, b, f);
#pragma unroll
    for (int q = 0; q < 12; ++q) a[q] = fmadd<TP>(b[q], f[q], a[q]);
}

// Segmented sum of a[] over runs of lanes with equal key; returns true in the
// first lane of each run, which then holds the run's totals.
template <typename TP>
__device__ __forceinline__ bool run_sum(int key, TP a[12]) {
    const int lane = threadIdx.x & 31;
    const int prev = __shfl_up_sync(0xffffffffu, key, 1);
    const bool head = lane == 0 || key != prev;
    const unsigned H = __ballot_sync(0xffffffffu, head);
    if (H != 0xffffffffu) {
        const unsigned after = H & ~((2u << lane) - 1u);
        const int seg_end = after ? (__ffs(after) - 2) : 31;
        // only as many doubling rounds as the longest run needs
        const unsigned run = __reduce_max_sync(0xffffffffu, head ? (unsigned)(seg_end - lane + 1) : 1u);
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            if ((unsigned)d >= run) break;
            const bool take = lane + d <= seg_end;
#pragma unroll
            for (int q = 0; q < 12; ++q) {
                TP o = __shfl_down_sync(0xffffffffu, a[q], d);
                if (take) a[q] += o;
            }
        }
    }
    return head;
}

// Adds one run's 12 totals at block cell c (strides X0, XY).
template <typename TP>
__device__ __forceinline__ void add_slots(TP* __restrict__ sJ, long long JC, int c, int X0, int XY, int ey, int ez,
                                          const TP a[12]) {
    TP* jx = sJ;
    TP* jy = sJ + JC;
    TP* jz = sJ + 2 * JC;
    atomicAdd(&jx[c], a[0]);
    if (ey) atomicAdd(&jx[c + X0], a[1]);
    if (ez) atomicAdd(&jx[c + XY], a[2]);
    if (ey && ez) atomicAdd(&jx[c + X0 + XY], a[3]);
    atomicAdd(&jy[c], a[4]);
    atomicAdd(&jy[c + 1], a[5]);
    if (ez) atomicAdd(&jy[c + XY], a[6]);
    if (ez) atomicAdd(&jy[c + 1 + XY], a[7]);
    atomicAdd(&jz[c], a[8]);
    atomicAdd(&jz[c + 1], a[9]);
    if (ey) atomicAdd(&jz[c + X0], a[10]);
    if (ey) atomicAdd(&jz[c + 1 + X0], a[11]);
}

// Fixed-point current block of the FP32 path: a run total a becomes the
// integer x = rint(a * sc) (sc a power of two with |x| < 2^40), and the block
// holds each entry as a 64-bit two's-complement sum in a low (unsigned) and a
// high (signed) 32-bit word, the low word's carry added to the high one.
// Shared 32-bit integer atomics are native; the sums are exact and
// independent of the order of the adds.  The split uses 32-bit conversions
// and integer operations only (64-bit integer conversions run on the FP64
// pipe, which is slow on this GPU): |x| = h 2^31 + l with h < 2^9, l < 2^31.
__device__ __forceinline__ void fx_add(unsigned* __restrict__ lo, int* __restrict__ hi, int e, float xf) {
    const float m = fabsf(xf);
    const float hf = floorf(m * 4.656612873077393e-10f);            // m / 2^31, exact power-of-two scaling
    const unsigned h = (unsigned)hf;
    const unsigned l = __float2uint_rn(m - hf * 2147483648.0f);      // exact remainder, rounded to an integer
    const unsigned al = ((h & 1u) << 31) | l;                        // |x| in base 2^32
    const unsigned ah = h >> 1;
    // two's complement of the 64-bit value for x < 0, without branches (a
    // zero x adds nothing)
    const unsigned sg = xf < 0.f ? 0xffffffffu : 0u;
    const unsigned xl = (al ^ sg) - sg;
    const unsigned xh = (ah ^ sg) + (sg & (xl == 0u ? 1u : 0u));
    const unsigned old = atomicAdd(&lo[e], xl);
    const unsigned carry = (old + xl < old) ? 1u : 0u;
    atomicAdd(&hi[e], (int)(xh + carry));
}

// add_slots in fixed point.
// 32-bit offsets: a block holds 3 x (tile + 4)^3 entries at most.
__device__ __forceinline__ void add_slots_fx(unsigned* __restrict__ lo, int* __restrict__ hi, int JC, int c,
                                             int X0, int XY, int ey, int ez, const float a[12], float sc) {
    const int off[12] = {c, c + X0, c + XY, c + X0 + XY,
                               JC + c, JC + c + 1, JC + c + XY, JC + c + 1 + XY,
                               2 * JC + c, 2 * JC + c + 1, 2 * JC + c + X0, 2 * JC + c + 1 + X0};
    const bool use[12] = {true, ey != 0, ez != 0, ey && ez, true, true, ez != 0, ez != 0, true, true, ey != 0, ey != 0};
#pragma unroll
    for (int q = 0; q < 12; ++q)
        if (use[q]) fx_add(lo, hi, off[q], a[q] * sc);
}

// Run heads whose totals one warp spreads over its lanes, and the per-warp
// shared scratch that holds them (12 totals and the block cell of each head,
// 16-byte aligned).
constexpr int kSpreadHeads = 10;
constexpr int kSpreadBytes = (kSpreadHeads * 12 * 4 + kSpreadHeads * 4 + 15) & ~15;

// The fixed-point adds of one reduced segment: the run heads (head, key >= 0)
// hold 12 totals each.  With at most kSpreadHeads heads in the warp (the
// usual case: particles sorted by cell make runs of about the cell's
// particle count) the heads park their scaled totals in the warp's scratch
// and every lane adds about 12 heads / 32 of them, so that the conversion
// and the two atomics of each add run on all lanes instead of on the heads
// alone; with more heads each head adds its own.  Exact either way: the
// fixed-point sums do not depend on the order of the adds.
__device__ __forceinline__ void add_runs_fx(unsigned* __restrict__ lo, int* __restrict__ hi, int JC, int X0, int XY,
                                            int ey, int ez, bool head, int key, const float a[12], float sc,
                                            float* __restrict__ wv) {
    const int lane = threadIdx.x & 31;
    const bool mine = head && key >= 0;
    const unsigned H = __ballot_sync(0xffffffffu, mine);
    const int nh = __popc(H);
    if (nh > kSpreadHeads) {
        if (mine) add_slots_fx(lo, hi, JC, key, X0, XY, ey, ez, a, sc);
        return;
    }
    int* wk = reinterpret_cast<int*>(wv + kSpreadHeads * 12);
    if (mine) {
        const int o = __popc(H & ((1u << lane) - 1u));
        float4* d = reinterpret_cast<float4*>(wv + 12 * o);
        d[0] = make_float4(a[0] * sc, a[1] * sc, a[2] * sc, a[3] * sc);
        d[1] = make_float4(a[4] * sc, a[5] * sc, a[6] * sc, a[7] * sc);
        d[2] = make_float4(a[8] * sc, a[9] * sc, a[10] * sc, a[11] * sc);
        wk[o] = key;
    }
    __syncwarp();
    // value v = 12 o + q: head o, slot q of segment_slots (component q / 4;
    // bit 0 of q % 4 the first upper neighbour, bit 1 the second)
    for (int v = lane; v < 12 * nh; v += 32) {
        const int o = v / 12, q = v - 12 * o;
        const int comp = q >> 2, sub = q & 3;
        const int s1 = comp == 0 ? X0 : 1, s2 = comp == 2 ? X0 : XY;
        const bool use = ((sub & 1) == 0 || comp != 0 || ey) && ((sub & 2) == 0 || (comp == 2 ? ey : ez));
        if (use) fx_add(lo, hi, comp * JC + wk[o] + (sub & 1) * s1 + (sub >> 1) * s2, wv[v]);
    }
    __syncwarp();
}

// The fused kernel's constants in the particle precision.
template <typename TP>
struct PushSet {
    TP dt, idt, d[3], id[3], hid[3];
    TP q[kMaxSpecies], m[kMaxSpecies], beta[kMaxSpecies], fcd[kMaxSpecies];
    float fx_scale;   // fixed-point scale (FP32)
    int parts;        // CTAs per tile
};

// The tiles of a work tile (kMerge), x fastest: chunks of 32 particles in the
// tiles before each, first particle and count.
constexpr int kMergeTiles = 512;   // tiles of one cell in 8^3
struct MergeTable {
    int before[kMergeTiles + 1];
    unsigned first[kMergeTiles], count[kMergeTiles];
    int warp_total[kTileThreads / 32];
};
// Fills the table for one species (all threads; a thread per tile, or with kRows
// per row of tiles along x, whose particles are consecutive).
template <bool kRows>
__device__ __forceinline__ void merge_table(MergeTable* M, const int* __restrict__ off, const TileGeom& o, int ti, int tj,
                                            int tk) {
    static_assert(kTileThreads == kMergeTiles, "a thread per tile");
    const int e = threadIdx.x, lane = e & 31, warp = e >> 5;
    const int gx = kRows ? 1 : 8 / o.tx, gy = 8 / o.ty, gz = 8 / o.tz;
    const int a = kRows ? ti * (8 / o.tx) : ti * gx + e % gx, b = tj * gy + e / gx % gy, c = tk * gz + e / (gx * gy);
    int first = 0, count = 0;
    if (e < gx * gy * gz && a < o.ntx && b < o.nty && c < o.ntz) {
        const int T3 = o.tx * o.ty * o.tz;
        const long long k0 = ((long long)(c * o.nty + b) * o.ntx + a) * T3;
        first = off[k0];
        count = off[k0 + T3 * (kRows ? min(8 / o.tx, o.ntx - a) : 1)] - first;
    }
    const int mine = (count + 31) / 32;
    int x = mine;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, x, d);
        if (lane >= d) x += y;
    }
    __syncthreads();   // the species before is done with the table
    if (lane == 31) M->warp_total[warp] = x;
    __syncthreads();
    int base = 0;
    for (int w = 0; w < warp; ++w) base += M->warp_total[w];
    M->before[e] = base + x - mine;
    M->first[e] = (unsigned)first;
    M->count[e] = (unsigned)count;
    if (e == kMergeTiles - 1) M->before[kMergeTiles] = base + x;
    __syncthreads();
}

// CT: compile-time tile extent of a cubic 3-D tile (8), or 0 for shapes read
// from TileShape at run time.  kWall: conductor-wall box (GridP::wall), the
// Tristan mover's reflection and escape and the zigzag wall term
// (mover.cpp:744-772, momentum_collecting.cpp:93-99); a particle that
// escaped deposits its current and is marked (cell -1) for the next sort.
// kParts: several CTAs per tile (parts > 1); without it the loop keeps no
// register for the stride (64 are all it has).
// kMerge: t holds work tiles of CT^3 cells, each several of the sort's tiles o
// (ragged at the box's upper ends): a box whose axes no 8-cell tile divides is
// sorted by smaller tiles, and a CTA per such tile would stage and flush more
// cells of halo than it has of its own.  A warp's 32 particles always come from
// one of the sort's tiles, counted from its first, and a particle's distance
// is measured from that tile, so the sums of a run, and which particles are
// left to the deferred pass, are those of a CTA per tile, bit for bit (FP32).
// FP64 sums come in any order, so its chunks are cut from rows of tiles along x
// (35x49x17, tiles of one cell, 5 per species: 15.3 -> 4.7 ms for five steps),
// and distances are measured from the work tile.
// At 100x60x54, 9 per species and cell (tiles of 4x4x2): 428 -> 273 us.
template <typename TP, typename TF, int CT, bool kWall, bool kParts, bool kMerge>
__global__ void __launch_bounds__(kTileThreads, tile_ctas<TP>()) k_push_deposit_tile(GridP g, TileGeom t, TileGeom o, TileShape s,
                                                                       SpeciesSet<TP> S,
                                                                       const __grid_constant__ PushSet<TP> K,
                                                                       const TF* __restrict__ E, const TF* __restrict__ B,
                                                                       double* __restrict__ Jpart) {
    constexpr bool kFixed = sizeof(TP) == sizeof(float);   // FP32 particles: fixed-point block
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int fx = CT ? CT + 4 : s.fx, fy = CT ? CT + 4 : s.fy, fz = CT ? CT + 4 : s.fz;
    const int jx = fx, jy = fy, jz = fz;                 // both blocks: tile + 2 halo on active axes
    const int tx = CT ? CT : t.tx, ty = CT ? CT : t.ty, tz = CT ? CT : t.tz;
    const int hx = 2, hy = CT ? 2 : s.hy, hz = CT ? 2 : s.hz;
    const int F = fx * fy * fz;
    const long long JC = (long long)jx * jy * jz;
    TF* sF = reinterpret_cast<TF*>(smem_raw);   // 6 * F
    TP* sJ = reinterpret_cast<TP*>(smem_raw + ((6 * F * sizeof(TF) + 15) & ~size_t(15)));   // 3 * JC (FP64)
    unsigned* sLo = reinterpret_cast<unsigned*>(sJ);                                        // 3 * JC (FP32)
    int* sHi = reinterpret_cast<int*>(sLo + 3 * JC);                                        // 3 * JC (FP32)
    // FP32: the warps' spread scratch after the block; then every warp's
    // staged chunk of particles
    unsigned char* after_j = reinterpret_cast<unsigned char*>(sJ) + ((24 * JC + 15) & ~15ll);
    float* sW = reinterpret_cast<float*>(after_j + (threadIdx.x >> 5) * kSpreadBytes);
    ChunkBuf<TP>* sBuf = reinterpret_cast<ChunkBuf<TP>*>(after_j + (kFixed ? (blockDim.x >> 5) * kSpreadBytes : 0)) +
                         (threadIdx.x >> 5);
    // kMerge: of the work tile's tiles, the chunks before each and its first
    // particle and count of this species
    MergeTable* sM = reinterpret_cast<MergeTable*>(reinterpret_cast<unsigned char*>(sBuf - (threadIdx.x >> 5)) +
                                                   (kTileThreads / 32) * sizeof(ChunkBuf<TP>));
    const int ntiles = t.ntx * t.nty * t.ntz;
    const long long N = g.N;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    // (in the particle precision already: of the FP64 grid parameters the
    // compiler repeats four conversions per chunk, on the FP64 pipe)
    const TP dt = K.dt, idt = K.idt;
    const TP dx = K.d[0], dy = K.d[1], dz = K.d[2];
    const TP idx = K.id[0], idy = K.id[1], idz = K.id[2];
    const int parts = kParts ? K.parts : 1;
    // extents of the sort's tiles
    constexpr bool kPlace = kMerge && kFixed;   // where a chunk's tile lies in the work tile matters
    const int otx = kPlace ? o.tx : tx, oty = kPlace ? o.ty : ty, otz = kPlace ? o.tz : tz;
    const int ey = CT ? 1 : (g.y3 ? 1 : 0), ez = CT ? 1 : (g.z3 ? 1 : 0);
    const int fsy = ey ? fx : 0, fsz = ez ? fx * fy : 0;

    // `parts` CTAs share a tile: each takes every parts-th chunk of its
    // particles and writes a partial block of its own
    for (int work = blockIdx.x; work < ntiles * parts; work += gridDim.x) {
        const int tile = work / parts, part = work - tile * parts;
        const int ti = tile % t.ntx, tj = (tile / t.ntx) % t.nty, tk = tile / (t.ntx * t.nty);
        const int lox = ti * tx, loy = tj * ty, loz = tk * tz;
        for (int e = threadIdx.x; e < F; e += blockDim.x) {
            int a = e % fx, b = (e / fx) % fy, c = e / (fx * fy);
            long long gi = linw(g, lox - hx + a, loy - hy + b, loz - hz + c);
#pragma unroll
            for (int comp = 0; comp < 3; ++comp) {
                sF[comp * F + e] = E[comp * N + gi];
                sF[(3 + comp) * F + e] = B[comp * N + gi];
            }
        }
        if (kFixed) {
            for (long long e = threadIdx.x; e < 3 * JC; e += blockDim.x) { sLo[e] = 0u; sHi[e] = 0; }
        } else {
            for (long long e = threadIdx.x; e < 3 * JC; e += blockDim.x) sJ[e] = TP(0);
        }
        __syncthreads();

        for (int sp = 0; sp < S.ns; ++sp) {
            const PartView<TP> P = S.p[sp];
            const TP q = K.q[sp], m = K.m[sp], beta = K.beta[sp], fcd = K.fcd[sp];
            // A warp takes chunks of 32 consecutive particles of a tile: chunk
            // warp, warp + nwarps * parts, ... (n0: its first particle, pe: the
            // end of its tile's).  Each warp's next chunk is copied into its
            // shared buffer while it pushes the current one.  (IDX unsigned: a
            // species holds fewer than 2^31 particles.)
            unsigned n0, pe;
            int at = 0, c = part * (kTileThreads / 32) + warp, chunks = 0;   // kMerge: tile of the table, chunk, their number
            auto seek = [&]() {   // kMerge: n0 and pe of chunk c, at or after tile `at`
                unsigned passed;
                do {
                    const int i = at + 1 + lane;
                    passed = __ballot_sync(0xffffffffu, i <= kMergeTiles && sM->before[i < kMergeTiles ? i : kMergeTiles] <= c);
                    at += __popc(passed);
                } while (passed == 0xffffffffu);
                n0 = sM->first[at] + 32u * (unsigned)(c - sM->before[at]);
                pe = sM->first[at] + sM->count[at];
            };
            if constexpr (kMerge) {
                merge_table<!kFixed>(sM, S.off[sp], o, ti, tj, tk);
                chunks = sM->before[kMergeTiles];
                n0 = pe = 0;
                if (c < chunks) seek();
            } else {
                const long long k0 = (long long)tile * (tx * ty * tz);
                n0 = S.off[sp][k0] + part * kTileThreads + 32 * warp;
                pe = S.off[sp][k0 + tx * ty * tz];
            }
            if (n0 + lane < pe) stage_particle(sBuf, P, n0 + lane, lane);
            cp_async_commit();
            while (n0 < pe) {
                const unsigned nb = n0, n = n0 + lane;
                const bool here = n < pe;
                // the tile's place in the work tile
                const int px = kPlace ? (at & (CT / otx - 1)) * otx : 0;
                const int py = kPlace ? (at / (CT / otx) & (CT / oty - 1)) * oty : 0;
                const int pz = kPlace ? at / (CT / otx * (CT / oty)) * otz : 0;
                TP aB[12];
                TP s1[6] = {TP(0), TP(0), TP(0), TP(0), TP(0), TP(0)};   // F1 and W1 of the old-side segment
                int keyA = -1 - lane, keyB = -1 - lane;   // lanes outside a reduction keep unique keys
                bool push_later = false, deposit_later = false;
                // a lane reads and refills only its own slots, and the wait
                // covers the copies it started itself
                cp_async_wait_all();
                const int cell = here ? sBuf->cell[lane] : -1;
                TP ox = sBuf->a[0][lane], oy = sBuf->a[1][lane], oz = sBuf->a[2][lane];
                TP mom[3] = {sBuf->a[3][lane], sBuf->a[4][lane], sBuf->a[5][lane]};
                if constexpr (kMerge) {
                    c += parts * (kTileThreads / 32);
                    if (c < chunks) seek();
                    else n0 = pe;
                } else {
                    n0 += parts * kTileThreads;
                }
                if (n0 + lane < pe) stage_particle(sBuf, P, n0 + lane, lane);
                cp_async_commit();
                // FP64: particles near a face, and with kNearMin of them the whole
                // chunk, are left to the deferred pass
                bool near = false;
                if constexpr (!kFixed) {
                    near = here && (near_face(ox) || (ey && near_face(oy)) || (ez && near_face(oz)));
                    const unsigned all = __ballot_sync(0xffffffffu, near);
                    near = near || __popc(all) >= kNearMin;
                }
                // (an escaped particle of a wall box waits with cell -1 for the sort)
                if (here && (!kWall || cell >= 0)) {
                    int i, j, k;
                    decode(g, cell, i, j, k);
                    auto local = [](int c, int lo, int te, int nn) {
                        int l = c - lo;
                        if (l > te) l -= nn;
                        if (l < -1) l += nn;
                        return l;
                    };
                    const int li = local(i, lox + px, otx, g.nx);
                    const int lj = ey ? local(j, loy + py, oty, g.ny) : 0;
                    const int lk = ez ? local(k, loz + pz, otz, g.nz) : 0;
                    const bool fast = li >= -1 && li <= otx && lj >= -ey && lj <= oty * ey && lk >= -ez && lk <= otz * ez && !near;
                    push_later = !fast;
                    if (fast) {
                        TP e3[3], b3[3];
                        // upper-neighbour weights: node grids (c, c+1) with weight u;
                        // cell-centred grids (c-1, c) with u + 1/2 below the centre,
                        // (c, c+1) with u - 1/2 above it (correlation.cpp:471-496)
                        const int c0 = (lk + pz + hz) * fsz + (lj + py + hy) * fsy + (li + px + hx);
                        const int cxs = ox < TP(0.5) ? -1 : 0;
                        const int cys = (ey && oy < TP(0.5)) ? -fsy : 0;
                        const int czs = (ez && oz < TP(0.5)) ? -fsz : 0;
                        const TP wcx = ox < TP(0.5) ? ox + TP(0.5) : ox - TP(0.5);
                        const TP wcy = ey ? (oy < TP(0.5) ? oy + TP(0.5) : oy - TP(0.5)) : TP(0);
                        const TP wcz = ez ? (oz < TP(0.5) ? oz + TP(0.5) : oz - TP(0.5)) : TP(0);
                        const TP wny = ey ? oy : TP(0), wnz = ez ? oz : TP(0);
                        e3[0] = tri<TP, TF>(sF + 0 * F, c0 + cxs, fsy, fsz, wcx, wny, wnz);
                        e3[1] = tri<TP, TF>(sF + 1 * F, c0 + cys, fsy, fsz, ox, wcy, wnz);
                        e3[2] = tri<TP, TF>(sF + 2 * F, c0 + czs, fsy, fsz, ox, wny, wcz);
                        b3[0] = tri<TP, TF>(sF + 3 * F, c0 + cys + czs, fsy, fsz, ox, wcy, wcz);
                        b3[1] = tri<TP, TF>(sF + 4 * F, c0 + cxs + czs, fsy, fsz, wcx, wny, wcz);
                        b3[2] = tri<TP, TF>(sF + 5 * F, c0 + cxs + cys, fsy, fsz, wcx, wcy, wnz);
                        boris_tile<TP>(q, m, dt, beta, e3, b3, mom);
                        TP v[3];
                        velocity_tile<TP>(mom, m, v);
                        int ni = i, nj = j, nk = k;
                        int wall_r = 0;
                        if constexpr (kWall) {
                            wall_r = tristan_wall_to<TP>(g, ni, ox, fmadd<TP>(mulr<TP>(v[0], dt), idx, ox));
                            if (wall_r & 1) { mom[0] = -mom[0]; v[0] = -v[0]; }   // reflectMomentumX
                        } else {
                            advance_axis<TP>(ox, ni, mulr<TP>(v[0], dt), idx, g.nx);
                        }
                        advance_axis<TP>(oy, nj, mulr<TP>(v[1], dt), idy, g.ny);
                        advance_axis<TP>(oz, nk, mulr<TP>(v[2], dt), idz, g.nz);
                        P.px[n] = mom[0]; P.py[n] = mom[1]; P.pz[n] = mom[2];
                        P.ox[n] = ox; P.oy[n] = oy; P.oz[n] = oz;
                        auto shift = [](int nw, int old, int nn) {
                            int d = nw - old;
                            if (d > 1) d -= nn;
                            if (d < -1) d += nn;
                            return d;
                        };
                        // block cell of the new position (a wall box has no x
                        // wrap; a particle reflected from left of the wall may
                        // land far from its old cell and is deposited by the
                        // deferred pass)
                        const int sxw = kWall ? ni - i : shift(ni, i, g.nx);
                        const bool nearx = !kWall || (sxw >= -1 && sxw <= 1);
                        const int bx = li + sxw + hx;
                        const int by = (ey ? lj + shift(nj, j, g.ny) : 0) + hy;
                        const int bz = (ez ? lk + shift(nk, k, g.nz) : 0) + hz;
                        // zigzag split (zig_axis, momentum_collecting.cpp:91-221) in the
                        // new cell's frame: old position P, relay R, relay shift r
                        const TP X = mulr<TP>(ox, dx), Y = mulr<TP>(oy, dy), Z = mulr<TP>(oz, dz);
                        TP PX = subr<TP>(X, mulr<TP>(v[0], dt));
                        const TP PY = fmadd<TP>(-v[1], dt, Y), PZ = fmadd<TP>(-v[2], dt, Z);
                        if constexpr (kWall) {
                            if (ni == kTristanWallNode && v[0] > TP(0) && PX < TP(0)) PX = -PX;
                        }
                        const TP fxr = dev_floor(PX * idx), fyr = ey ? dev_floor(PY * idy) : TP(0),
                                 fzr = ez ? dev_floor(PZ * idz) : TP(0);
                        const int rx = (int)fxr, ry = (int)fyr, rz = (int)fzr;
                        const TP RX = rx == 0 ? (X + PX) * TP(0.5) : TP(rx > 0 ? rx : 0) * dx;
                        const TP RY = ry == 0 ? (Y + PY) * TP(0.5) : TP(ry > 0 ? ry : 0) * dy;
                        const TP RZ = rz == 0 ? (Z + PZ) * TP(0.5) : TP(rz > 0 ? rz : 0) * dz;
                        const int ax = bx + rx, ay = by + ry, az = bz + rz;   // block cell of the old-side segment
                        // unsigned compares: (unsigned)x < n is 0 <= x < n
                        const int ex_ = kPlace ? otx + 4 : jx, ey_ = kPlace ? oty + 4 : jy, ez_ = kPlace ? otz + 4 : jz;
                        const bool inblock = nearx && (unsigned)(rx + 1) <= 2u && (unsigned)(ry + 1) <= 2u &&
                                             (unsigned)(rz + 1) <= 2u && (unsigned)ax < (unsigned)(ex_ - 1) &&
                                             (unsigned)bx < (unsigned)(ex_ - 1) && (unsigned)ay < (unsigned)(ey_ - ey) &&
                                             (unsigned)by < (unsigned)(ey_ - ey) && (unsigned)az < (unsigned)(ez_ - ez) &&
                                             (unsigned)bz < (unsigned)(ez_ - ez);
                        if (inblock) {
                            const TP F1x = (fcd * (RX - PX)) * idt;
                            const TP F1y = (fcd * (RY - PY)) * idt;
                            const TP F1z = (fcd * (RZ - PZ)) * idt;
                            const TP F2x = (fcd * (X - RX)) * idt;
                            const TP F2y = fmadd<TP>(fcd, v[1], -F1y), F2z = fmadd<TP>(fcd, v[2], -F1z);
                            const TP hxx = K.hid[0], hyy = K.hid[1], hzz = K.hid[2];   // half reciprocals
                            const TP W1x = fmadd<TP>(PX + RX, hxx, -TP(rx));
                            const TP W1y = ey ? fmadd<TP>(PY + RY, hyy, -TP(ry)) : TP(0);
                            const TP W1z = ez ? fmadd<TP>(PZ + RZ, hzz, -TP(rz)) : TP(0);
                            const TP W2x = (X + RX) * hxx;
                            const TP W2y = ey ? (Y + RY) * hyy : TP(0);
                            const TP W2z = ez ? (Z + RZ) * hzz : TP(0);
                            segment_slots<TP>(F2x, F2y, F2z, W2x, W2y, W2z, aB);
                            s1[0] = F1x; s1[1] = F1y; s1[2] = F1z; s1[3] = W1x; s1[4] = W1y; s1[5] = W1z;
                            keyA = ((az + pz) * jy + ay + py) * jx + ax + px;
                            keyB = ((bz + pz) * jy + by + py) * jx + bx + px;
                        }
                        deposit_later = !inblock;
                        // an escaped particle is marked once its current is
                        // deposited (the deferred pass marks its own)
                        P.cell[n] = ((wall_r & 2) && inblock) ? -1 : (int)lin(g, ni, nj, nk);
                    }
                }
                {
                    const unsigned mp = __ballot_sync(0xffffffffu, push_later);
                    const unsigned md = __ballot_sync(0xffffffffu, deposit_later);
                    if ((mp | md) && lane == 0) {
                        set_defer_bits(S.defer[sp], nb, mp);
                        set_defer_bits(S.defer[sp] + S.dwords[sp], nb, md);
                    }
                }
                if (keyB < 0) {
#pragma unroll
                    for (int q2 = 0; q2 < 12; ++q2) aB[q2] = TP(0);
                }
                // a particle that stays in its cell (no relay shift) has both
                // segments in that cell: one set of 12 sums carries both, and
                // the old-side pass is left to the particles that crossed (its
                // 12 values are formed only then, from the six kept in s1)
                if (keyA == keyB && keyA >= 0) {
                    segment_add<TP>(s1[0], s1[1], s1[2], s1[3], s1[4], s1[5], aB);
                    keyA = -1 - lane;
                }
                const bool crossed = __any_sync(0xffffffffu, keyA >= 0);
                if constexpr (kFixed) {
                    const bool hb = run_sum<TP>(keyB, aB);
                    add_runs_fx(sLo, sHi, (int)JC, jx, jx * jy, ey, ez, hb, keyB, (const float*)aB, K.fx_scale, sW);
                } else {
                    if (run_sum<TP>(keyB, aB) && keyB >= 0) add_slots<TP>(sJ, JC, keyB, jx, jx * jy, ey, ez, aB);
                }
                if (crossed) {
                    // lanes without an old-side segment hold unique negative
                    // keys: runs of one lane, whatever their values
                    TP aA[12];
                    segment_slots<TP>(s1[0], s1[1], s1[2], s1[3], s1[4], s1[5], aA);
                    if constexpr (kFixed) {
                        const bool ha = run_sum<TP>(keyA, aA);
                        add_runs_fx(sLo, sHi, (int)JC, jx, jx * jy, ey, ez, ha, keyA, (const float*)aA, K.fx_scale, sW);
                    } else {
                        if (run_sum<TP>(keyA, aA) && keyA >= 0) add_slots<TP>(sJ, JC, keyA, jx, jx * jy, ey, ez, aA);
                    }
                }
            }
        }
        __syncthreads();
        double* dst = Jpart + (long long)work * 3 * JC;
        if (kFixed) {
            // the exact block sums as 64-bit integers (k_assemble_j adds
            // them exactly and scales once per cell): integer operations
            // only, nothing on the FP64 pipe
            long long* dsti = reinterpret_cast<long long*>(dst);
            for (long long e = threadIdx.x; e < 3 * JC; e += blockDim.x)
                dsti[e] = (long long)sHi[e] * 4294967296ll + (long long)sLo[e];
        } else {
            for (long long e = threadIdx.x; e < 3 * JC; e += blockDim.x) dst[e] = sJ[e];
        }
        __syncthreads();
    }
}

// The particles k_push_deposit_tile left over, by their mask bits (each
// word read once and cleared for the next step):
//   * push-later (more than one cell outside their tile): the same gather
//     from global memory, Boris push and move, then the zigzag current;
//   * deposit-later (pushed there, segments outside the tile's current
//     block): the zigzag current of the stored new position and velocity.
// The current goes into Jfix with FP64 global atomics; a particle that left a
// wall box is marked (cell -1) once its current is in.
// FP32: a thread per word (few of which hold a bit).  FP64, where every particle of
// a lattice load may start on a face (near_face): the bits dealt to the lanes, so
// that neighbours move neighbouring particles.
template <typename TP, typename TF>
__global__ void __launch_bounds__(256) k_push_deposit_deferred(GridP g, SpeciesSet<TP> S, const TF* __restrict__ E,
                                                               const TF* __restrict__ B, double* __restrict__ Jfix) {
    const TP dt = TP(g.dt);
    const TP idx = TP(g.idx), idy = TP(g.idy), idz = TP(g.idz);
    const TP vol = TP(g.dx) * TP(g.dy) * TP(g.dz);
    for (int sp = 0; sp < S.ns; ++sp) {
        const PartView<TP> P = S.p[sp];
        const TP q = S.q[sp], m = S.m[sp];
        const TP beta = q * dt / (TP(2) * m);
        const TP fcd = q * S.w[sp] / vol;
        unsigned* mp = S.defer[sp];
        unsigned* md = mp + S.dwords[sp];
        const long long words = (P.n + 31) / 32 + 1;
        auto one = [&](long long n, bool push) {
            TP ox = P.ox[n], oy = P.oy[n], oz = P.oz[n];
            TP mom[3] = {P.px[n], P.py[n], P.pz[n]};
            int ni, nj, nk;
            decode(g, P.cell[n], ni, nj, nk);
            TP v[3];
            if (push) {
                TP e3[3], b3[3];
                if constexpr (sizeof(TP) == sizeof(float)) yee_gather<TP, TF>(g, P.cell[n], ox, oy, oz, E, B, e3, b3);
                else tri_gather<TP, TF>(g, P.cell[n], ox, oy, oz, E, B, e3, b3);
                boris_t<TP>(q, m, dt, beta, e3, b3, mom);
                velocity_t<TP>(mom, m, v);
                if (g.wall) {
                    if (tristan_wall_x<TP>(g, ni, ox, (v[0] * dt) * idx) & 1) {   // reflectMomentumX
                        mom[0] = -mom[0];
                        v[0] = -v[0];
                    }
                } else {
                    advance_axis<TP>(ox, ni, (v[0] * dt) * idx, g.nx);
                }
                advance_axis<TP>(oy, nj, (v[1] * dt) * idy, g.ny);
                advance_axis<TP>(oz, nk, (v[2] * dt) * idz, g.nz);
                P.px[n] = mom[0]; P.py[n] = mom[1]; P.pz[n] = mom[2];
                P.ox[n] = ox; P.oy[n] = oy; P.oz[n] = oz;
            } else {
                velocity_t<TP>(mom, m, v);
            }
            deposit_global<TP>(g, fcd, ox, oy, oz, v, ni, nj, nk, Jfix);
            P.cell[n] = (g.wall && tristan_escaped<TP>(g, ni, ox)) ? -1 : (int)lin(g, ni, nj, nk);
        };
        if constexpr (sizeof(TP) == sizeof(float)) {
            for (long long w = blockIdx.x * (long long)blockDim.x + threadIdx.x; w < words;
                 w += (long long)gridDim.x * blockDim.x) {
                unsigned bp = mp[w], bd = md[w];
                if (!(bp | bd)) continue;
                mp[w] = 0u;
                md[w] = 0u;
                while (bp | bd) {
                    const bool push = bp != 0u;
                    unsigned& bits = push ? bp : bd;
                    const long long n = w * 32 + (__ffs(bits) - 1);
                    bits &= bits - 1u;
                    one(n, push);
                }
            }
        } else {
            // 16 words of either mask per warp, lane by lane, their set bits dealt to the lanes
            const int lane = threadIdx.x & 31, at = lane & 15;
            const long long warps = ((long long)gridDim.x * blockDim.x) >> 5;
            for (long long w0 = ((blockIdx.x * (long long)blockDim.x + threadIdx.x) >> 5) * 16; w0 < words; w0 += warps * 16) {
                unsigned* const mine = (lane < 16 ? mp : md) + w0 + at;
                const unsigned bits = w0 + at < words ? *mine : 0u;
                if (bits) *mine = 0u;
                if (!__any_sync(0xffffffffu, bits != 0u)) continue;
                int upto = __popc(bits);   // bits of the lanes up to this one
#pragma unroll
                for (int d = 1; d < 32; d <<= 1) {
                    const int y = __shfl_up_sync(0xffffffffu, upto, d);
                    if (lane >= d) upto += y;
                }
                const int total = __shfl_sync(0xffffffffu, upto, 31);
                for (int k0 = 0; k0 < total; k0 += 32) {
                    const int k = min(k0 + lane, total - 1);
                    int l = 0;   // the lane that holds bit k
#pragma unroll
                    for (int d = 16; d > 0; d >>= 1)
                        if (__shfl_sync(0xffffffffu, upto, l + d - 1) <= k) l += d;
                    const unsigned word = __shfl_sync(0xffffffffu, bits, l);
                    const int before = __shfl_sync(0xffffffffu, upto, l) - __popc(word);
                    if (k0 + lane < total) one((w0 + (l & 15)) * 32 + (int)__fns(word, 0, k - before + 1), l < 16);
                    __syncwarp();
                }
            }
        }
    }
}

// J[c] = Jfix[c] + sum of every tile partial that covers cell c, tiles and
// periodic images visited in a fixed order (deterministic).  FP32 particles:
// the partials are 64-bit fixed-point integers, summed exactly and scaled by
// inv_scale (a power of two) once; FP64 particles: FP64 partials.
// kWhole: tiles of four or more cells that divide their axis, of which at most
// two cover a cell.  Finding them is cheap, so a thread takes one component of a
// cell: on a small box the loads' latency is the time (32^3, 4 partials per tile:
// 14.8 us with one thread for the three, 8.3 us so; 128^3, bound by the partials'
// traffic: 82 us, 15 less).  Else every tile is tried that may, once for the
// three components (100x60x54 in work tiles: 21 us, 40 us one by one).
template <typename TP, bool kParts, bool kWhole>
__global__ void __launch_bounds__(256) k_assemble_j(GridP g, TileGeom t, TileShape s, const double* __restrict__ Jpart,
                                                    const double* __restrict__ Jfix, double* __restrict__ J,
                                                    double inv_scale, int nparts) {
    constexpr bool kFixed = sizeof(TP) == sizeof(float);
    constexpr int kCand = kWhole ? 2 : 16;
    const int parts = kParts ? nparts : 1;
    const long long JC = s.jcells;
    constexpr int kComp = kWhole ? 1 : 3;        // components of a thread, from the first
    const int first = kWhole ? blockIdx.y : 0;
    for (long long c = blockIdx.x * (long long)blockDim.x + threadIdx.x; c < g.N;
         c += (long long)gridDim.x * blockDim.x) {
        int p[3];
        decode(g, (int)c, p[0], p[1], p[2]);
        const int n[3] = {g.nx, g.ny, g.nz};
        const int te[3] = {t.tx, t.ty, t.tz};
        const int nt[3] = {t.ntx, t.nty, t.ntz};
        const int je[3] = {s.jx, s.jy, s.jz};
        const int hg[3] = {s.gx, s.gy, s.gz};
        // per axis: every (tile, local index) whose current block holds this
        // cell or one of its periodic images
        int cand_t[3][kCand], cand_l[3][kCand], cnt[3];
#pragma unroll
        for (int ax = 0; ax < 3; ++ax) {
            if constexpr (kWhole) {
                const int T = p[ax] / te[ax], l = p[ax] - T * te[ax];
                cand_t[ax][0] = T;
                cand_l[ax][0] = l + hg[ax];
                const bool low = l < hg[ax], up = l >= te[ax] - hg[ax];
                cnt[ax] = low || up ? 2 : 1;
                cand_t[ax][1] = low ? (T > 0 ? T - 1 : nt[ax] - 1) : (T + 1 < nt[ax] ? T + 1 : 0);
                cand_l[ax][1] = l + hg[ax] + (low ? te[ax] : -te[ax]);
            } else {
                cnt[ax] = 0;
                for (int sh = -1; sh <= 1; ++sh) {
                    const int q = p[ax] + sh * n[ax];
                    // block of tile T spans [T*te - hg, T*te - hg + je)
                    int tlo = q + hg[ax] - je[ax] + 1;
                    tlo = tlo >= 0 ? (tlo + te[ax] - 1) / te[ax] : -((-tlo) / te[ax]);
                    int thi = q + hg[ax];
                    thi = thi >= 0 ? thi / te[ax] : -((-thi + te[ax] - 1) / te[ax]);
                    if (tlo < 0) tlo = 0;
                    if (thi > nt[ax] - 1) thi = nt[ax] - 1;
                    for (int T = tlo; T <= thi && cnt[ax] < kCand; ++T) {
                        cand_t[ax][cnt[ax]] = T;
                        cand_l[ax][cnt[ax]] = q - (T * te[ax] - hg[ax]);
                        cnt[ax]++;
                    }
                }
            }
        }
        double acc[kComp];
        long long iacc[kComp] = {};
#pragma unroll
        for (int q = 0; q < kComp; ++q) acc[q] = Jfix[(first + q) * g.N + c];
        auto add = [&](int a, int b, int d) {
            const long long tile = ((long long)cand_t[2][d] * t.nty + cand_t[1][b]) * t.ntx + cand_t[0][a];
            const long long e = ((long long)cand_l[2][d] * s.jy + cand_l[1][b]) * s.jx + cand_l[0][a] + first * JC;
#pragma unroll(kWhole ? 4 : 1)
            for (int r = 0; r < parts; ++r) {
                const double* src = Jpart + (tile * parts + r) * 3 * JC + e;
#pragma unroll
                for (int q = 0; q < kComp; ++q) {
                    if constexpr (kFixed) iacc[q] += *reinterpret_cast<const long long*>(src + q * JC);
                    else acc[q] += src[q * JC];
                }
            }
        };
        if constexpr (kWhole) {
#pragma unroll
            for (int a = 0; a < kCand; ++a)
#pragma unroll
                for (int b = 0; b < kCand; ++b)
#pragma unroll
                    for (int d = 0; d < kCand; ++d)
                        if (a < cnt[0] && b < cnt[1] && d < cnt[2]) add(a, b, d);
        } else {
            for (int a = 0; a < cnt[0]; ++a)
                for (int b = 0; b < cnt[1]; ++b)
                    for (int d = 0; d < cnt[2]; ++d) add(a, b, d);
        }
#pragma unroll
        for (int q = 0; q < kComp; ++q) {
            if constexpr (kFixed) acc[q] += (double)iacc[q] * inv_scale;
            J[(first + q) * g.N + c] = acc[q];
        }
    }
}

}  // namespace pic
