// implicit_tile.cuh -- moment deposition of the implicit path over tiles of
// cells (updateElectroMagneticParameters, PIC++/momentum_collecting.cpp
// 365-584, with the pressure tensor at the particle's own cells).
//
// Particles are ordered by the tile-major cell key (sort.cuh).  One CTA owns
// a tile (right after a sort: a box of cells of its own) and accumulates, in
// shared memory,
//   * on nodes (tile + h halo + 1):  J-hat (3) and mu (9), 8 nodes/particle;
//   * on cells (tile + h halo + 2):  rho-hat (1) and Pi (6 of the symmetric
//     9), 8 of the 27 cells around the particle's cell.
// A warp takes one cell key at a time and walks its particles 32 at a time.
// Lanes holding the same (current) cell share one stencil base, so their
// 96 node and 189 cell products (27 slots, zero weight outside the
// particle's octant) are summed over the run before one shared-memory atomic
// per sum: FP32 particles as small TF32 tensor-core products at FP32
// accuracy (tc_run_sums), FP64 ones by a butterfly
// transpose-reduction (after five exchange rounds lane L holds the warp total
// of product L of a 32-product pass).  Runs of only a few lanes add their
// products directly; particles more than h cells
// outside the tile add theirs to the FP64 grids with global atomics.  The
// tile's block is finally added to the FP64 grids (global atomics only on
// block entries, 22 per node/cell).
#pragma once
#include "implicit_particles.cuh"

namespace pic {

#ifndef PIC_IMP_THREADS
#define PIC_IMP_THREADS 256   // threads per CTA of the tiled implicit deposit (2 CTAs/SM, 128 registers)
#endif
#ifndef PIC_MOVER_THREADS
#define PIC_MOVER_THREADS 256   // threads per CTA of the tiled implicit mover (2 CTAs/SM)
#endif
constexpr int kImpThreads = PIC_IMP_THREADS;
// FP64 particles keep 256 threads (128 registers): their accumulators spill at 64
template <typename T>
__host__ __device__ constexpr int imp_threads() { return sizeof(T) == sizeof(float) ? kImpThreads : 256; }
constexpr int kMoverThreads = PIC_MOVER_THREADS;
constexpr int kXposeMin = 4;   // fewest lanes of one cell that take the transpose-reduction (FP64)
constexpr int kTcMin = 1;      // fewest lanes of one cell that take the tensor-core run sums (FP32)


// Node weights (c, c + 1) and cell weights (c - 1, c, c + 1) of one axis
// (node_w and cell_w of common.cuh without branches).
template <typename T>
__device__ __forceinline__ void axis_weights(T u, bool act, T wn[2], T wc[3]) {
    if (!act) { wn[0] = T(1); wn[1] = T(0); wc[0] = T(0); wc[1] = T(1); wc[2] = T(0); return; }
    wn[0] = T(1) - u;
    wn[1] = u;
    const T d = u - T(0.5);
    wc[0] = d < T(0) ? -d : T(0);
    wc[1] = T(1) - (d < T(0) ? -d : d);
    wc[2] = d < T(0) ? T(0) : d;
}

// Local index of global cell index c on an axis of n cells relative to a
// tile starting at x0, chosen within [-h, t - 1 + h] when a periodic image
// lies there; false if none does.
__device__ __forceinline__ bool local_axis(int c, int x0, int t, int h, int n, int& l) {
    l = c - x0;
    if (l >= -h && l <= t - 1 + h) return true;
    if (l - n >= -h && l - n <= t - 1 + h) { l -= n; return true; }
    if (l + n >= -h && l + n <= t - 1 + h) { l += n; return true; }
    return false;
}

// Weights of the eight corners (x fastest) from the upper weight of each axis;
// kFlat: the four of a box of one cell along z (wz is 0).
template <typename T, bool kFlat = false>
__device__ __forceinline__ void corners(T wx, T wy, T wz, T w[8]) {
    const T ux = T(1) - wx, uy = T(1) - wy, uz = T(1) - wz;
    if constexpr (kFlat) {
        w[0] = ux * uy; w[1] = wx * uy; w[2] = ux * wy; w[3] = wx * wy;
        return;
    }
    const T yz[4] = {uy * uz, wy * uz, uy * wz, wy * wz};
#pragma unroll
    for (int q = 0; q < 4; ++q) { w[2 * q] = ux * yz[q]; w[2 * q + 1] = wx * yz[q]; }
}
// Three components gathered with corner weights that they share (12 products
// and 24 multiply-adds; nested interpolations are 14 operations per component): from three planes of a staged block, `plane`
// entries apart, or from a block of float4 nodes or cells (x, y, z, unused),
// one 16-byte load per corner.
template <typename T, bool kFlat = false>
__device__ __forceinline__ void gather3(const T* __restrict__ F, int plane, int base, int sx, int sy, int sz,
                                        const T w[8], T out[3]) {
#pragma unroll
    for (int q = 0; q < 3; ++q) {
        const T* f = F + q * plane + base;
        T v = w[0] * f[0];
        v = fma(w[1], f[sx], v);
        v = fma(w[2], f[sy], v);
        v = fma(w[3], f[sy + sx], v);
        if constexpr (kFlat) {
            out[q] = v;
            continue;
        }
        v = fma(w[4], f[sz], v);
        v = fma(w[5], f[sz + sx], v);
        v = fma(w[6], f[sz + sy], v);
        out[q] = fma(w[7], f[sz + sy + sx], v);
    }
}
// (x, y) in one packed FP32 multiply-add, z (and the unused fourth) in another:
// the FP32 mover, bound by instruction issue, 448 -> 428 us at 64x64x16.
__device__ __forceinline__ unsigned long long twice(float a) {
    unsigned long long r;
    asm("mov.b64 %0, {%1, %1};" : "=l"(r) : "f"(a));
    return r;
}
__device__ __forceinline__ void fma2(unsigned long long& acc, unsigned long long a, unsigned long long b) {
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc) : "l"(a), "l"(b));
}
__device__ __forceinline__ void split2(unsigned long long p, float& lo, float& hi) {
    asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(p));
}
__device__ __forceinline__ void gather3(const float4* __restrict__ F, int base, int sx, int sy, int sz, const float w[8],
                                        float out[3]) {
    const ulonglong2* f = reinterpret_cast<const ulonglong2*>(F + base);
    const int at[8] = {0, sx, sy, sy + sx, sz, sz + sx, sz + sy, sz + sy + sx};
    unsigned long long xy = 0, z = 0;
#pragma unroll
    for (int q = 0; q < 8; ++q) {
        const ulonglong2 v = f[at[q]];
        const unsigned long long ww = twice(w[q]);
        fma2(xy, ww, v.x);
        fma2(z, ww, v.y);
    }
    float none;
    split2(xy, out[0], out[1]);
    split2(z, out[2], none);
}
// ---- tensor-core reduction of one run (FP32 accumulators) -------------------
// The 96 node sums  N[q][c] = sum_p QN_p[q] wn_p[c]  and 189 cell sums
// C[s][q] = sum_p wc_p[s] QC_p[q]  of a run of particles are small matrix
// products with the particles as the inner dimension.  Each lane writes its
// particle's raw quantities (rv 3, alpha 9, per-axis node weights 2 x 3,
// per-axis cell weights 3 x 3) to a per-warp scratch of 32 rows; the warp
// then runs m16n8k8 TF32 MMAs, eight particles per MMA, in the 3 x TF32 form
// (x = hi + lo, products hi*hi + hi*lo + lo*hi, FP32 accumulation), which
// keeps the sums at FP32 accuracy.  The per-species factors (cq, cm) are
// applied to the sums.
constexpr int kScrRow = 27;         // scratch floats per particle
constexpr int kScrParticles = 32;   // scratch rows per warp

// x = hi + lo + e with hi, lo in the 19-bit TF32 format (low 13 bits zero),
// both truncated: x - hi is exact in FP32 (at most 13 significant bits) and
// |e| < 2^-21 |x|.  Three integer/FP32 operations per split.
__device__ __forceinline__ void tf32_split(float x, unsigned& hi, unsigned& lo) {
    hi = __float_as_uint(x) & 0xffffe000u;
    lo = __float_as_uint(x - __uint_as_float(hi)) & 0xffffe000u;
}

// D (16x8, FP32) += A (16x8, TF32, row) * B (8x8, TF32, col)
__device__ __forceinline__ void mma_tf32(float d[4], const unsigned a[4], const unsigned b[2]) {
    asm volatile("mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
}

// D += A * B at FP32 accuracy from pre-split B
__device__ __forceinline__ void mma_tf32x3(float d[4], const float a[4], const unsigned bh[2], const unsigned bl[2]) {
    unsigned ah[4], al[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) tf32_split(a[i], ah[i], al[i]);
    mma_tf32(d, al, bh);
    mma_tf32(d, ah, bl);
    mma_tf32(d, ah, bh);
}

// The scratch-row columns a lane reads in tc_run_sums, which depend on the
// lane only: byte k of sx / sy / sz is the column of the x / y / z weight
// of cell slot g + 8k (g = lane / 4); bytes of nb: the node weight columns
// 12 + gx, 14 + gy, 16 + gz and the rv columns ia, ib of pressure
// component g - 1.  Built once per CTA into a shared table.
struct TcLane {
    unsigned sx, sy, sz, nb;
};
__device__ __forceinline__ TcLane tc_lane(int lane) {
    const int g = lane >> 2;
    TcLane t{0u, 0u, 0u, 0u};
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const int sl = g + 8 * k;
        t.sx |= (unsigned)(18 + sl % 3) << (8 * k);
        t.sy |= (unsigned)(21 + (sl / 3) % 3) << (8 * k);
        t.sz |= (unsigned)(sl < 27 ? 24 + sl / 9 : 24) << (8 * k);
    }
    const int ia = g >= 1 && g <= 6 ? sym_a(g - 1) : 0, ib = g >= 1 && g <= 6 ? sym_b(g - 1) : 0;
    t.nb = (unsigned)(12 + (g & 1)) | (unsigned)(14 + ((g >> 1) & 1)) << 8 | (unsigned)(16 + (g >> 2)) << 16 |
           (unsigned)(ia | ib << 4) << 24;
    return t;
}
__device__ __forceinline__ int tc_byte(unsigned w, int k) { return (int)((w >> (8 * k)) & 0xffu); }

// Sums of one run over the warp, added to dn and dc: mem = lanes in the run;
// row = this lane's raw quantities (used only when the lane is in the run);
// tl = this lane's TcLane.  Lane (g = lane/4, t = lane%4) holds
// dn[i] = N[g + 8(i/2)][2t + i%2] and dc[4k + i] = C[16k + g + 8(i/2)][2t + i%2].
__device__ __forceinline__ void tc_run_sums(float* __restrict__ scr, int lane, bool me, unsigned mem,
                                            const float row[kScrRow], float dn[4], float dc[8], const TcLane tl) {
    const int g = lane >> 2, tq = lane & 3;
    const int cnx = tc_byte(tl.nb, 0), cny = tc_byte(tl.nb, 1), cnz = tc_byte(tl.nb, 2);
    const int ia = tc_byte(tl.nb, 3) & 15, ib = tc_byte(tl.nb, 3) >> 4;
    int sox[4], soy[4], soz[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        sox[k] = tc_byte(tl.sx, k);
        soy[k] = tc_byte(tl.sy, k);
        soz[k] = tc_byte(tl.sz, k);
    }
    {
        float* r = scr + lane * kScrRow;
#pragma unroll
        for (int f = 0; f < kScrRow; ++f) r[f] = me ? row[f] : 0.f;
    }
    __syncwarp();
#pragma unroll 1
    for (int s2 = 0; s2 < 4; ++s2) {
        if (((mem >> (8 * s2)) & 0xffu) == 0) continue;
        const float* P0 = scr + (8 * s2 + tq) * kScrRow;
        const float* P1 = P0 + 4 * kScrRow;
        unsigned bh[2], bl[2];
        float a[4];
        // nodes: A[q][p] = (rv, alpha)[q], q = g and g + 8 (< 12); B[p][c] = node weight of corner c = g
        tf32_split(P0[cnx] * P0[cny] * P0[cnz], bh[0], bl[0]);
        tf32_split(P1[cnx] * P1[cny] * P1[cnz], bh[1], bl[1]);
        a[0] = P0[g];
        a[1] = g < 4 ? P0[g + 8] : 0.f;
        a[2] = P1[g];
        a[3] = g < 4 ? P1[g + 8] : 0.f;
        mma_tf32x3(dn, a, bh, bl);
        // cells: A[s][p] = slot weight, s = 16k + g (+ 8); B[p][q] = 1, rv_a rv_b (q = g < 7)
        tf32_split(g == 0 ? 1.f : (g < 7 ? P0[ia] * P0[ib] : 0.f), bh[0], bl[0]);
        tf32_split(g == 0 ? 1.f : (g < 7 ? P1[ia] * P1[ib] : 0.f), bh[1], bl[1]);
#pragma unroll
        for (int k = 0; k < 2; ++k) {
            const int j0 = 2 * k, j1 = 2 * k + 1;   // slots 16k + g and 16k + g + 8
            const bool v1 = 16 * k + g + 8 < 27;
            a[0] = P0[sox[j0]] * P0[soy[j0]] * P0[soz[j0]];
            a[1] = v1 ? P0[sox[j1]] * P0[soy[j1]] * P0[soz[j1]] : 0.f;
            a[2] = P1[sox[j0]] * P1[soy[j0]] * P1[soz[j0]];
            a[3] = v1 ? P1[sox[j1]] * P1[soy[j1]] * P1[soz[j1]] : 0.f;
            mma_tf32x3(dc + 4 * k, a, bh, bl);
        }
    }
    __syncwarp();
}

// Adds the run sums of tc_run_sums (lane layout as there) to the shared
// blocks at node base nb and cell base cb, times the species factors.
template <typename A>
__device__ __forceinline__ void add_run_sums(A* __restrict__ sN, A* __restrict__ sC, int NB, int CB, int nb,
                                             int cb, int oxn, int oyn, int ozn, int oxc, int oyc, int ozc, int lane,
                                             const float dn[4], const float dc[8], float cq, float cm) {
    const int gq = lane >> 2, tq = lane & 3;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int q = gq + 8 * (i >> 1), c = 2 * tq + (i & 1);
        if (q < 12 && dn[i] != 0.f)
            atomicAdd(&sN[q * NB + nb + (c & 1) * oxn + ((c >> 1) & 1) * oyn + (c >> 2) * ozn], A(dn[i] * (q < 3 ? cq : cm)));
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const int sl = 16 * (i >> 2) + gq + 8 * ((i >> 1) & 1), q = 2 * tq + (i & 1);
        if (sl < 27 && q < 7 && dc[i] != 0.f)
            atomicAdd(&sC[q * CB + cb + (sl % 3) * oxc + ((sl / 3) % 3) * oyc + (sl / 9) * ozc], A(dc[i] * cq));
    }
}

// Deposited quantities of one particle from its raw row: QN = (rv cq, alpha cm),
// QC = (cq, cq rv_a rv_b) over the symmetric pressure components.
template <typename A, typename T>
__device__ __forceinline__ void run_quantities(const T row[kScrRow], double cq, double cm, A QN[12], A QC[7]) {
    const A rv[3] = {A(row[0]), A(row[1]), A(row[2])};
#pragma unroll
    for (int d = 0; d < 3; ++d) QN[d] = rv[d] * A(cq);
#pragma unroll
    for (int d = 0; d < 9; ++d) QN[3 + d] = A(row[3 + d]) * A(cm);
    QC[0] = A(cq);
#pragma unroll
    for (int q = 0; q < 6; ++q) QC[1 + q] = A(cq) * (rv[sym_a(q)] * rv[sym_b(q)]);
}

// Node (8 corners) and cell (27 slots) weights from the per-axis weights of a row.
template <typename A, typename T>
__device__ __forceinline__ void run_weights(const T row[kScrRow], A wn[8], A wc[27]) {
#pragma unroll
    for (int c = 0; c < 8; ++c) wn[c] = A(row[12 + (c & 1)] * row[14 + ((c >> 1) & 1)] * row[16 + (c >> 2)]);
#pragma unroll
    for (int q = 0; q < 27; ++q) wc[q] = A(row[18 + q % 3] * row[21 + (q / 3) % 3] * row[24 + q / 9]);
}

// Direct shared-memory adds of one particle of a short run (rolled loops:
// rare, so kept small next to the hot code).
template <typename T>
__device__ __forceinline__ T pick2(const T* w, int i) { return i ? w[1] : w[0]; }
template <typename T>
__device__ __forceinline__ T pick3(const T* w, int i) { return i == 0 ? w[0] : (i == 1 ? w[1] : w[2]); }

template <typename A, typename T>
__device__ __forceinline__ void imp_deposit_direct(const T row[kScrRow], double cq, double cm, A* __restrict__ sN,
                                                   A* __restrict__ sC, int NB, int CB, int nb, int cb, int oxn, int oyn,
                                                   int ozn, int oxc, int oyc, int ozc) {
    A QN[12], QC[7];
    run_quantities<A, T>(row, cq, cm, QN, QC);
#pragma unroll 1
    for (int c = 0; c < 8; ++c) {
        const A w = A(pick2(row + 12, c & 1) * pick2(row + 14, (c >> 1) & 1) * pick2(row + 16, c >> 2));
        if (w == A(0)) continue;
        const int o = nb + (c & 1) * oxn + ((c >> 1) & 1) * oyn + (c >> 2) * ozn;
#pragma unroll
        for (int q = 0; q < 12; ++q) atomicAdd(&sN[q * NB + o], QN[q] * w);
    }
#pragma unroll 1
    for (int sl = 0; sl < 27; ++sl) {
        const A w = A(pick3(row + 18, sl % 3) * pick3(row + 21, (sl / 3) % 3) * pick3(row + 24, sl / 9));
        if (w == A(0)) continue;
        const int o = cb + (sl % 3) * oxc + ((sl / 3) % 3) * oyc + (sl / 9) * ozc;
#pragma unroll
        for (int q = 0; q < 7; ++q) atomicAdd(&sC[q * CB + o], QC[q] * w);
    }
}

// All 8 node and 8 cell contributions of one particle to the FP64 grids
// (particles outside the tile's block; rare).
template <typename T>
__device__ __noinline__ void imp_deposit_global(const GridP g, int i, int j, int k, T ox, T oy, T oz,
                                                const double* QN, const double* QC, double* __restrict__ J,
                                                double* __restrict__ mu, double* __restrict__ rho,
                                                double* __restrict__ Pi) {
    int X[2], Y[2], Z[2];
    T wx[2], wy[2], wz[2];
    node_w(ox, i, g.nx, X, wx); node_w(oy, j, g.ny, Y, wy); node_w(oz, k, g.nz, Z, wz);
    for (int a = 0; a < 2; ++a)
        for (int b = 0; b < 2; ++b)
            for (int c = 0; c < 2; ++c) {
                double wgt = double(wx[a]) * double(wy[b]) * double(wz[c]);
                if (wgt == 0.0) continue;
                long long id = lin(g, X[a], Y[b], Z[c]);
                for (int d = 0; d < 3; ++d) atomicAdd(&J[d * g.N + id], QN[d] * wgt);
                for (int d = 0; d < 9; ++d) atomicAdd(&mu[d * g.N + id], QN[3 + d] * wgt);
            }
    cell_w(ox, i, g.nx, X, wx); cell_w(oy, j, g.ny, Y, wy); cell_w(oz, k, g.nz, Z, wz);
    for (int a = 0; a < 2; ++a)
        for (int b = 0; b < 2; ++b)
            for (int c = 0; c < 2; ++c) {
                double wgt = double(wx[a]) * double(wy[b]) * double(wz[c]);
                if (wgt == 0.0) continue;
                long long id = lin(g, X[a], Y[b], Z[c]);
                atomicAdd(&rho[id], QC[0] * wgt);
                for (int s = 0; s < 6; ++s) {
                    double v = QC[1 + s] * wgt;
                    atomicAdd(&Pi[(3 * sym_a(s) + sym_b(s)) * g.N + id], v);
                    if (sym_a(s) != sym_b(s)) atomicAdd(&Pi[(3 * sym_b(s) + sym_a(s)) * g.N + id], v);
                }
            }
}

// Global trilinear gathers of E (nodes) and B (cells), out of line for the
// staged kernel, where a particle outside its tile cannot occur after a sort.
// The grid in and the six components out by value: an address taken of the
// caller's arrays would send their every store to the stack.
template <typename T>
struct EB6 {
    T e[3], b[3];
};
template <typename T>
__device__ __noinline__ EB6<T> gather_eb_global(const GridP g, int i, int j, int k, T ox, T oy, T oz,
                                                const T* __restrict__ E, const T* __restrict__ B) {
    EB6<T> r;
    gather_node<T, T>(g, i, j, k, ox, oy, oz, E, r.e);
    gather_cell<T, T>(g, i, j, k, ox, oy, oz, B, r.b);
    return r;
}

// The run sums of the lanes `me` (one stencil base) with FP64 accumulators: a
// butterfly per 32 products, one shared atomic per lane and pass.
// kFlat (one cell along z): 4 corners and 9 slots, 4 passes instead of 9.
template <typename A, typename T, bool kFlat = false>
__device__ __forceinline__ void butterfly_sums(const T row[kScrRow], bool me, double cq, double cm, A* __restrict__ sN,
                                               A* __restrict__ sC, int NB, int CB, int nb, int cb, int oxn, int oyn,
                                               int ozn, int oxc, int oyc, int ozc, int lane) {
    A QN[12], QC[7], wn[8], wc[27];
    run_quantities<A, T>(row, cq, cm, QN, QC);
    run_weights<A, T>(row, wn, wc);
    constexpr int NC = kFlat ? 4 : 8, NS = kFlat ? 9 : 27, Z = kFlat ? 9 : 0;   // corners, slots (of z slot 1), first slot
    A vv[32];
#pragma unroll
    for (int r = 0; r < (12 * NC + 31) / 32; ++r) {
#pragma unroll
        for (int x = 0; x < 32; ++x) {
            const int idx = 32 * r + x;
            vv[x] = (idx < 12 * NC && me) ? QN[idx / NC] * wn[idx % NC] : A(0);
        }
        const A sum = xpose_sum<A>(vv, lane);
        const int idx = 32 * r + lane, q = idx / NC, c = idx % NC;
        if (idx < 12 * NC && sum != A(0))
            atomicAdd(&sN[q * NB + nb + (c & 1) * oxn + ((c >> 1) & 1) * oyn + (c >> 2) * ozn],
                      sum);
    }
#pragma unroll
    for (int r = 0; r < (7 * NS + 31) / 32; ++r) {
#pragma unroll
        for (int x = 0; x < 32; ++x) {
            const int idx = 32 * r + x;
            vv[x] = (idx < 7 * NS && me) ? QC[idx / NS] * wc[Z + idx % NS] : A(0);
        }
        const A sum = xpose_sum<A>(vv, lane);
        const int idx = 32 * r + lane;
        if (idx < 7 * NS && sum != A(0)) {
            const int q = idx / NS, sl = idx % NS;
            atomicAdd(&sC[q * CB + cb + (sl % 3) * oxc + ((sl / 3) % 3) * oyc + (sl / 9) * ozc],
                      sum);
        }
    }
}

// A particle outside the block (rare): its raw row into the FP64 grids.
template <typename A, typename T>
__device__ __forceinline__ void deposit_row_global(const GridP& g, int cell, T ox, T oy, T oz, const T row[kScrRow],
                                                   double cq, double cm, double* __restrict__ J, double* __restrict__ mu,
                                                   double* __restrict__ rho, double* __restrict__ Pi) {
    int i, j, k;
    decode(g, cell, i, j, k);
    A QN[12], QC[7];
    run_quantities<A, T>(row, cq, cm, QN, QC);
    double qn[12], qc[7];
#pragma unroll
    for (int d = 0; d < 12; ++d) qn[d] = double(QN[d]);
#pragma unroll
    for (int d = 0; d < 7; ++d) qc[d] = double(QC[d]);
    imp_deposit_global<T>(g, i, j, k, ox, oy, oz, qn, qc, J, mu, rho, Pi);
}

// The tiled deposit's constants per species: beta and m in the particle
// precision, the factors of J-hat, rho-hat, Pi (q w / V) and of mu.
template <typename T>
struct DepositSet {
    T beta[kMaxSpecies], m[kMaxSpecies];
    double cq[kMaxSpecies], cm[kMaxSpecies];
};

// E and B come in the particle precision (FP32 copies for the FP32 path:
// no FP64 conversion per gather).
// kStaged (right after a sort, h = 0): a particle of key k lies in cell k, so a
// chunk of 32 particles of one key has one stencil base; E and B are staged in
// shared memory next to the accumulators (FP32: float4 nodes and cells, one
// 16-byte load per corner), the keys' offsets too, and each warp copies its
// next chunk of particles with cp.async while it works on the current one.
// What bounds it is instruction issue at 16 warps per SM (two CTAs: the run
// sums' accumulators take 128 registers).  t holds boxes of cells then, of
// which two fit on an SM (deposit_boxes, api.cu), some a cell smaller than
// others (box_start); they need not follow the sort's tiles o, a cell's particles being found by
// its key.  Not staged: t holds the sort's tiles.
// A: FP64 too for FP32 particles in a box of several of the sort's tiles: the
// tiles' sums met in the FP64 grids before, and so they still do (39x27x23, 60
// per species and cell: E after a step 8.5e-7 from 64 bits, with FP32
// accumulators 1.1e-6; 39x57x53: 985 us, with FP32 ones 846 us).
// kFlat (FP64, one cell along z): without the corners and slots that weigh 0;
// the FP64 pipe is what bounds it (pairs of 32x32x1: 192 -> 117 us).
template <typename T, typename A, bool kStaged, bool kFlat>
__global__ void __launch_bounds__(imp_threads<T>(), 2) k_implicit_deposit_tile(GridP g, TileGeom t, TileGeom o, ImpBlock bk,
                                                                       const __grid_constant__ ImpSpecies<T> S,
                                                                       const __grid_constant__ DepositSet<T> K,
                                                                       const T* __restrict__ E,
                                                                       const T* __restrict__ B,
                                                                       double* __restrict__ J, double* __restrict__ mu,
                                                                       double* __restrict__ rho,
                                                                       double* __restrict__ Pi) {
    extern __shared__ __align__(16) unsigned char imp_smem[];
    A* sN = reinterpret_cast<A*>(imp_smem);   // [12][NB]
    A* sC = sN + 12 * bk.NB;                  // [7][CB]
    // staged E and B: three planes each, FP32 one float4 per node / cell
    constexpr bool kVec = sizeof(T) == sizeof(float);
    T* sE = reinterpret_cast<T*>(imp_smem + bk.stage_at());
    T* sB = sE + 3 * bk.NB;
    float4* sE4 = reinterpret_cast<float4*>(sE);
    float4* sB4 = sE4 + bk.NB;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
    const int T3 = t.tx * t.ty * t.tz;
    const int ntiles = t.ntx * t.nty * t.ntz;
    const bool ax = g.nx > 1, ay = g.y3, az = g.z3;
    const int hx = ax ? bk.h : 0, hy = ay ? bk.h : 0, hz = az ? bk.h : 0;
    const int nsy = bk.nbx, nsz = bk.nbx * bk.nby;
    const int csy = bk.cbx, csz = bk.cbx * bk.cby;
    const int oxn = ax ? 1 : 0, oyn = ay ? nsy : 0, ozn = az ? nsz : 0;   // corner strides
    const int oxc = ax ? 1 : 0, oyc = ay ? csy : 0, ozc = az ? csz : 0;   // slot strides
    const int tot = 12 * bk.NB + 7 * bk.CB;
    constexpr bool kTc = sizeof(T) == sizeof(float);   // FP32 particles: tensor-core run sums
    unsigned char* after = imp_smem + bk.scratch_at();
    float* scr0 = reinterpret_cast<float*>(after);
    float* scr = scr0 + warp * (kScrParticles * kScrRow);
    // the lane table of tc_run_sums follows the scratch rows of all warps
    TcLane* s_lane = reinterpret_cast<TcLane*>(scr0 + nwarps * (kScrParticles * kScrRow));
    // staged: every warp's next chunk, then first particle and end of the
    // box's cells, of all species
    ChunkBuf<T>* buf = reinterpret_cast<ChunkBuf<T>*>(kTc ? reinterpret_cast<unsigned char*>(s_lane + 32) : after) + warp;
    int2* sOff = reinterpret_cast<int2*>(buf - warp + nwarps);
    if (kTc && threadIdx.x < 32) s_lane[threadIdx.x] = tc_lane(threadIdx.x);

    for (int tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
        const int ti = tile % t.ntx, tj = (tile / t.ntx) % t.nty, tk = tile / (t.ntx * t.nty);
        const int x0 = box_start(g.nx, ti, t.ntx), y0 = box_start(g.ny, tj, t.nty), z0 = box_start(g.nz, tk, t.ntz);
        for (int e = threadIdx.x; e < tot; e += blockDim.x) sN[e] = A(0);
        const int x1 = box_start(g.nx, ti + 1, t.ntx), y1 = box_start(g.ny, tj + 1, t.nty), z1 = box_start(g.nz, tk + 1, t.ntz);
        if (kStaged) {   // with h = 0 the blocks cover exactly the stencils of the box's own cells
            for (int e = threadIdx.x; e < bk.NB; e += blockDim.x) {
                const int lx = e % bk.nbx, ly = (e / bk.nbx) % bk.nby, lz = e / (bk.nbx * bk.nby);
                const long long id = linw(g, x0 + lx, y0 + ly, z0 + lz);
                if constexpr (kVec) {
                    sE4[e] = make_float4(E[id], E[g.N + id], E[2 * g.N + id], 0.f);
                } else {
#pragma unroll
                    for (int c = 0; c < 3; ++c) sE[c * bk.NB + e] = E[c * g.N + id];
                }
            }
            for (int e = threadIdx.x; e < bk.CB; e += blockDim.x) {
                const int lx = e % bk.cbx, ly = (e / bk.cbx) % bk.cby, lz = e / (bk.cbx * bk.cby);
                const long long id = linw(g, x0 - (ax ? 1 : 0) + lx, y0 - (ay ? 1 : 0) + ly, z0 - (az ? 1 : 0) + lz);
                if constexpr (kVec) {
                    sB4[e] = make_float4(B[id], B[g.N + id], B[2 * g.N + id], 0.f);
                } else {
#pragma unroll
                    for (int c = 0; c < 3; ++c) sB[c * bk.CB + e] = B[c * g.N + id];
                }
            }
            for (int e = threadIdx.x; e < T3; e += blockDim.x) {
                const int i = x0 + e % t.tx, j = y0 + (e / t.tx) % t.ty, k = z0 + e / (t.tx * t.ty);
                const bool in = i < x1 && j < y1 && k < z1;
                const int kk = in ? cell_key(o, i, j, k) : 0;
                for (int s = 0; s < S.ns; ++s)
                    sOff[s * T3 + e] = in ? make_int2(S.off[s][kk], S.off[s][kk + 1]) : make_int2(0, 0);
            }
        }
        __syncthreads();
        if constexpr (kStaged) {
            // the warp's chunks: keys warp, warp + nwarps, ... (a cell of one
            // species: all cells of the first, then of the next; empty ones
            // skipped), each 32 particles at a time
            const int2* __restrict__ of = sOff;
            const int keys = S.ns * T3;
            auto next_key = [&](int lc) {
                while (lc < keys && of[lc].x == of[lc].y) lc += nwarps;
                return lc;
            };
            int lc = next_key(warp), c0 = lc < keys ? of[lc].x : 0;
            if (lc < keys && c0 + lane < of[lc].y) stage_particle(buf, S.p[lc / T3], c0 + lane, lane);
            cp_async_commit();
            int key = -1, s = 0, cellK = 0, nbK = 0, cbK = 0;
            float an[4] = {0.f, 0.f, 0.f, 0.f}, ac[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
            while (lc < keys) {
                if (lc != key) {
                    key = lc;
                    s = lc / T3;
                    const int cell = lc - s * T3, li = cell % t.tx, q = cell / t.tx, lj = q % t.ty, lk = q / t.ty;
                    nbK = lk * nsz + lj * nsy + li;
                    cbK = lk * csz + lj * csy + li;
                    cellK = (int)lin(g, x0 + li, y0 + lj, z0 + lk);
                }
                const bool valid = c0 + lane < of[lc].y;
                cp_async_wait_all();   // a lane's own slots
                const int cell = buf->cell[lane];
                const T ox = buf->a[0][lane], oy = buf->a[1][lane], oz = buf->a[2][lane];
                const T mom[3] = {buf->a[3][lane], buf->a[4][lane], buf->a[5][lane]};
                int nlc = lc, nc0 = c0 + 32;
                if (nc0 >= of[lc].y) {
                    nlc = next_key(lc + nwarps);
                    nc0 = nlc < keys ? of[nlc].x : 0;
                }
                if (nlc < keys && nc0 + lane < of[nlc].y) stage_particle(buf, S.p[nlc / T3], nc0 + lane, lane);
                cp_async_commit();
                const double cq = K.cq[s], cm = K.cm[s];
                const T beta = K.beta[s], ms = K.m[s];
                // raw quantities: rv (3), alpha (9), node weights x/y/z (2 each), cell weights x/y/z (3 each)
                T row[kScrRow];
                const bool mine = valid && cell == cellK;   // (always, after a sort)
                if (valid) {
                    T gam, v[3];
                    gamma_vel<T>(mom, ms, gam, v);
                    T* nw = row + 12;
                    T* cw = row + 18;
                    axis_weights<T>(ox, ax, nw, cw);
                    axis_weights<T>(oy, ay, nw + 2, cw + 3);
                    axis_weights<T>(oz, az, nw + 4, cw + 6);
                    T e[3], bf[3];
                    if (mine) {
                        T w[8];
                        corners<T, kFlat>(nw[1], nw[3], nw[5], w);
                        if constexpr (kVec) gather3(sE4, nbK, oxn, oyn, ozn, w, e);
                        else gather3<T, kFlat>(sE, bk.NB, nbK, oxn, oyn, ozn, w, e);
                        // cell pair (c - 1, c) below the centre, (c, c + 1) above
                        const bool bx = ox < T(0.5), by = oy < T(0.5), bz = oz < T(0.5);
                        corners<T, kFlat>(bx ? cw[1] : cw[2], by ? cw[4] : cw[5], bz ? cw[7] : cw[8], w);
                        const int cbase = cbK + (bx ? 0 : oxc) + (by ? 0 : oyc) + (bz ? 0 : ozc);
                        if constexpr (kVec) gather3(sB4, cbase, oxc, oyc, ozc, w, bf);
                        else gather3<T, kFlat>(sB, bk.CB, cbase, oxc, oyc, ozc, w, bf);
                    } else {
                        int i, j, k;
                        decode(g, cell, i, j, k);
                        const EB6<T> r = gather_eb_global<T>(g, i, j, k, ox, oy, oz, E, B);
#pragma unroll
                        for (int c = 0; c < 3; ++c) { e[c] = r.e[c]; bf[c] = r.b[c]; }
                    }
                    T al[9];
                    alpha_tensor<T>(beta, v, gam, e, bf, al);
                    const T vg[3] = {v[0] * gam, v[1] * gam, v[2] * gam};
#pragma unroll
                    for (int a = 0; a < 3; ++a) row[a] = al[3 * a] * vg[0] + al[3 * a + 1] * vg[1] + al[3 * a + 2] * vg[2];
#pragma unroll
                    for (int d = 0; d < 9; ++d) row[3 + d] = al[d];
                    if (!mine) deposit_row_global<A, T>(g, cell, ox, oy, oz, row, cq, cm, J, mu, rho, Pi);
                } else {
#pragma unroll
                    for (int q = 0; q < kScrRow; ++q) row[q] = T(0);
                }
                const unsigned mm = __ballot_sync(0xffffffffu, mine);
                if constexpr (kTc) {
                    if (mm) tc_run_sums(scr, lane, mine, mm, row, an, ac, s_lane[lane]);
                    if (nlc != lc) {   // the key's sums reach the block once
                        add_run_sums(sN, sC, bk.NB, bk.CB, nbK, cbK, oxn, oyn, ozn, oxc, oyc, ozc, lane, an, ac, float(cq),
                                     float(cm));
#pragma unroll
                        for (int q = 0; q < 4; ++q) an[q] = 0.f;
#pragma unroll
                        for (int q = 0; q < 8; ++q) ac[q] = 0.f;
                    }
                } else if (__popc(mm) >= kXposeMin) {
                    butterfly_sums<A, T, kFlat>(row, mine, cq, cm, sN, sC, bk.NB, bk.CB, nbK, cbK, oxn, oyn, ozn, oxc, oyc, ozc,
                                         lane);
                } else if (mine) {
                    imp_deposit_direct<A, T>(row, cq, cm, sN, sC, bk.NB, bk.CB, nbK, cbK, oxn, oyn, ozn, oxc, oyc, ozc);
                }
                lc = nlc;
                c0 = nc0;
            }
        } else {
            for (int s = 0; s < S.ns; ++s) {
                const PartView<T> p = S.p[s];
                const double cq = K.cq[s], cm = K.cm[s];
                const T beta = K.beta[s], ms = K.m[s];
                const int* __restrict__ off = S.off[s];
                for (int lc = warp; lc < T3; lc += nwarps) {
                    const int kk = tile * T3 + lc;
                    const int b0 = off[kk], b1 = off[kk + 1];
                    for (int c0 = b0; c0 < b1; c0 += 32) {
                        const int n = c0 + lane;
                        const bool valid = n < b1;
                        // raw quantities: rv (3), alpha (9), node weights x/y/z (2 each), cell weights x/y/z (3 each)
                        T row[kScrRow];
#pragma unroll
                        for (int f = 0; f < kScrRow; ++f) row[f] = T(0);
                        int cell = -1, nb = 0, cb = 0;
                        bool inb = false;
                        if (valid) {
                            cell = p.cell[n];
                            int i, j, k;
                            decode(g, cell, i, j, k);
                            const T ox = p.ox[n], oy = p.oy[n], oz = p.oz[n];
                            T mom[3] = {p.px[n], p.py[n], p.pz[n]};
                            T gam, v[3];
                            gamma_vel<T>(mom, ms, gam, v);
                            T* nw = row + 12;
                            T* cw = row + 18;
                            axis_weights<T>(ox, ax, nw, cw);
                            axis_weights<T>(oy, ay, nw + 2, cw + 3);
                            axis_weights<T>(oz, az, nw + 4, cw + 6);
                            int li = 0, lj = 0, lk = 0;
                            inb = local_axis(i, x0, t.tx, hx, g.nx, li) && local_axis(j, y0, t.ty, hy, g.ny, lj) &&
                                  local_axis(k, z0, t.tz, hz, g.nz, lk);
                            if (inb) {
                                nb = (lk + hz) * nsz + (lj + hy) * nsy + (li + hx);
                                cb = (lk + hz) * csz + (lj + hy) * csy + (li + hx);
                            }
                            T e[3], bf[3];
                            gather_node<T, T>(g, i, j, k, ox, oy, oz, E, e);
                            gather_cell<T, T>(g, i, j, k, ox, oy, oz, B, bf);
                            T al[9];
                            alpha_tensor<T>(beta, v, gam, e, bf, al);
                            const T vg[3] = {v[0] * gam, v[1] * gam, v[2] * gam};
#pragma unroll
                            for (int a = 0; a < 3; ++a) row[a] = al[3 * a] * vg[0] + al[3 * a + 1] * vg[1] + al[3 * a + 2] * vg[2];
#pragma unroll
                            for (int d = 0; d < 9; ++d) row[3 + d] = al[d];
                            if (!inb) deposit_row_global<A, T>(g, cell, ox, oy, oz, row, cq, cm, J, mu, rho, Pi);
                        }
                        unsigned pending = __ballot_sync(0xffffffffu, valid && inb);
                        while (pending) {
                            const int leader = __ffs(pending) - 1;
                            const int lcell = __shfl_sync(0xffffffffu, cell, leader);
                            const bool me = ((pending >> lane) & 1u) && cell == lcell;
                            const unsigned mem = __ballot_sync(0xffffffffu, me);
                            pending &= ~mem;
                            if (__popc(mem) >= (kTc ? kTcMin : kXposeMin)) {
                                const int nbL = __shfl_sync(0xffffffffu, nb, leader);
                                const int cbL = __shfl_sync(0xffffffffu, cb, leader);
                                if constexpr (kTc) {
                                    float dn[4] = {0.f, 0.f, 0.f, 0.f}, dc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
                                    tc_run_sums(scr, lane, me, mem, row, dn, dc, s_lane[lane]);
                                    add_run_sums(sN, sC, bk.NB, bk.CB, nbL, cbL, oxn, oyn, ozn, oxc, oyc, ozc, lane, dn, dc,
                                                 float(cq), float(cm));
                                } else {
                                    butterfly_sums<A, T>(row, me, cq, cm, sN, sC, bk.NB, bk.CB, nbL, cbL, oxn, oyn, ozn, oxc, oyc, ozc,
                                                         lane);
                                }
                            } else if (me) {
                                imp_deposit_direct<A, T>(row, cq, cm, sN, sC, bk.NB, bk.CB, nb, cb, oxn, oyn, ozn, oxc, oyc, ozc);
                            }
                        }
                    }
                }
            }
        }
        __syncthreads();
        // flush the block into the FP64 grids
        for (int e = threadIdx.x; e < bk.NB; e += blockDim.x) {
            const int lx = e % bk.nbx, ly = (e / bk.nbx) % bk.nby, lz = e / (bk.nbx * bk.nby);
            const long long id = linw(g, x0 - hx + lx, y0 - hy + ly, z0 - hz + lz);
#pragma unroll
            for (int d = 0; d < 3; ++d) {
                const A v = sN[d * bk.NB + e];
                if (v != A(0)) atomicAdd(&J[d * g.N + id], double(v));
            }
#pragma unroll
            for (int d = 0; d < 9; ++d) {
                const A v = sN[(3 + d) * bk.NB + e];
                if (v != A(0)) atomicAdd(&mu[d * g.N + id], double(v));
            }
        }
        for (int e = threadIdx.x; e < bk.CB; e += blockDim.x) {
            const int lx = e % bk.cbx, ly = (e / bk.cbx) % bk.cby, lz = e / (bk.cbx * bk.cby);
            const long long id = linw(g, x0 - hx - (ax ? 1 : 0) + lx, y0 - hy - (ay ? 1 : 0) + ly,
                                      z0 - hz - (az ? 1 : 0) + lz);
            const A r = sC[e];
            if (r != A(0)) atomicAdd(&rho[id], double(r));
#pragma unroll
            for (int q = 0; q < 6; ++q) {
                const A v = sC[(1 + q) * bk.CB + e];
                if (v == A(0)) continue;
                atomicAdd(&Pi[(3 * sym_a(q) + sym_b(q)) * g.N + id], double(v));
                if (sym_a(q) != sym_b(q)) atomicAdd(&Pi[(3 * sym_b(q) + sym_a(q)) * g.N + id], double(v));
            }
        }
        __syncthreads();
    }
}

}  // namespace pic

namespace pic {


// Field blocks of the tiled mover: nodes (E^n, E^theta) over tile + 2H + 1,
// cells (B^n) over tile + 2H + 2 on active axes.
struct MoverBlock {
    int nbx, nby, nbz, NB;
    int cbx, cby, cbz, CB;
};

// The rows of tiles along x of a mover's work box (y fastest), species after
// species: chunks of 32 particles in the rows before each, the row's first
// particle and its end.  In shared memory, sized by the launch.
struct RowTable {
    int *before, *first, *end;   // before[n]: all chunks
    int n;
    __device__ RowTable(int* mem, int rows) : before(mem), first(mem + rows + 1), end(mem + 2 * rows + 1), n(rows) {}
    // The row of chunk c, at or after row `at` (a warp's lanes together; the
    // last one for a c past the end).
    __device__ int row_of(int c, int at, int lane) const {
        unsigned passed;
        do {
            const int i = at + 1 + lane;
            passed = __ballot_sync(0xffffffffu, i < n && before[i < n ? i : 0] <= c);
            at += __popc(passed);
        } while (passed == 0xffffffffu);
        return at;
    }
    // Filled by the first warp for the box (ti, tj, tk) of t.
    template <typename T>
    __device__ void fill(const ImpSpecies<T>& S, const TileGeom& o, const TileGeom& t, int ti, int tj, int tk) {
        const int lane = threadIdx.x;
        if (lane >= 32) return;
        const int gy = t.ty / o.ty, gz = t.tz / o.tz, T3 = o.tx * o.ty * o.tz;
        const int a0 = box_start(o.ntx, ti, t.ntx), a1 = box_start(o.ntx, ti + 1, t.ntx);
        const int b0 = box_start(o.nty, tj, t.nty), b1 = box_start(o.nty, tj + 1, t.nty);
        const int c0 = box_start(o.ntz, tk, t.ntz), c1 = box_start(o.ntz, tk + 1, t.ntz);
        int done = 0;
        for (int h = 0; h < n; h += 32) {
            const int e = h + lane, s = e / (gy * gz), w = e - s * (gy * gz);
            const int b = b0 + w % gy, c = c0 + w / gy;
            int x0 = 0, x1 = 0;
            if (e < n && b < b1 && c < c1) {
                const long long row = ((long long)c * o.nty + b) * o.ntx;
                x0 = S.off[s][(row + a0) * T3];
                x1 = S.off[s][(row + a1) * T3];
            }
            const int mine = (x1 - x0 + 31) / 32;
            int x = mine;
#pragma unroll
            for (int d = 1; d < 32; d <<= 1) {
                const int y = __shfl_up_sync(0xffffffffu, x, d);
                if (lane >= d) x += y;
            }
            if (e < n) {
                before[e] = done + x - mine;
                first[e] = x0;
                end[e] = x1;
            }
            done += __shfl_sync(0xffffffffu, x, 31);
        }
        if (lane == 0) before[n] = done;
    }
};

// The tiled mover's constants in the particle precision.
template <typename T>
struct MoverSet {
    T dt, eta, edt, redt, dx2;   // dx2: dx squared (Picard test)
    T id[3];
    T beta[kMaxSpecies], qdt[kMaxSpecies], m[kMaxSpecies];
};

// moveParticle (PIC++/mover.cpp:194-491), one CTA per tile of tile-ordered
// particles: E^n and E^{n+theta} (nodes) and B^n (cells) of the tile and a
// two-cell halo are staged in shared memory in the particle precision, so
// the predictor and the up to three Picard gathers read shared memory.  A
// particle with a position whose stencil leaves the block is left untouched
// and its bit set in S.defer: k_implicit_push_deferred moves it from the
// FP64 grids (the kernel itself calls nothing out of line, which would cost
// its hot loop register spills).  Same arithmetic as k_implicit_push.
// kRows: t holds work boxes of one or several of the sort's tiles o (some a tile
// smaller than others, box_start; along an axis that 8 does not divide those
// tiles are 4, 2 or 1 cells wide, and their two-cell halo would be most of what
// a CTA stages), and `nparts` CTAs share a box.  The particles are the box's rows of tiles along x,
// one range of indices each and of all species one after the other, which the
// warps take 32 at a time: in a small box, where a CTA has a few hundred
// particles, all its warps work at once.  Without it: a CTA per tile, species by
// species.
// FP32 beams of 39x57x53 (tiles of one cell), 60 per species and cell: 3,170 ->
// 762 us; shock of 112x51x5: 192 -> 135 us; FP64 pairs of 61x43x1: 525 -> 310 us;
// of 32x32x1, 32 per species and cell (whole tiles, 19 CTAs each): 207 -> 82 us.
// kFlat (FP64, one cell along z): gathers from four corners, where eight keep the
// FP64 pipe busy with weights of 0 (32x32x1: 108 -> 82 us).
template <typename T, bool kWall, bool kRows, bool kFlat>
__global__ void __launch_bounds__(kMoverThreads, 2) k_implicit_push_tile(GridP g, TileGeom t, TileGeom o, MoverBlock mb,
                                                            const __grid_constant__ ImpSpecies<T> S,
                                                            const __grid_constant__ MoverSet<T> K,
                                                            const double* __restrict__ E, const double* __restrict__ B,
                                                            const double* __restrict__ Et, int nparts) {
    extern __shared__ __align__(16) unsigned char mv_smem[];
    // FP32: E^theta and B^n, gathered two or three times per particle, as
    // float4 nodes / cells (one 16-byte load per corner); E^n, gathered
    // once, as three scalar planes.  FP64: three scalar planes each.
    constexpr bool kVec = sizeof(T) == sizeof(float);
    float4* sEt4 = reinterpret_cast<float4*>(mv_smem);   // [NB] (FP32)
    float4* sB4 = sEt4 + mb.NB;                           // [CB] (FP32)
    T* sE = kVec ? reinterpret_cast<T*>(sB4 + mb.CB) : reinterpret_cast<T*>(mv_smem);   // [3][NB]
    T* sEt = sE + 3 * mb.NB;                 // [3][NB] (FP64)
    T* sB = sEt + 3 * mb.NB;                 // [3][CB] (FP64)
    // after the field blocks: every thread's next particle, copied with
    // cp.async while it moves the current one ([6][threads] values, then
    // [threads] cells)
    const size_t fld = kVec ? ((size_t)mb.NB + mb.CB) * 16 + 3 * (size_t)mb.NB * sizeof(float)
                            : (6 * (size_t)mb.NB + 3 * (size_t)mb.CB) * sizeof(T);
    T* sPre = reinterpret_cast<T*>(mv_smem + ((fld + 15) & ~size_t(15)));
    int* sPreCell = reinterpret_cast<int*>(sPre + 6 * blockDim.x);
    auto stage = [&](const PartView<T>& pv, int m) {
        const int me = threadIdx.x, bdim = blockDim.x;
        cp_async<4>(&sPreCell[me], pv.cell + m);
        cp_async<sizeof(T)>(&sPre[0 * bdim + me], pv.ox + m);
        cp_async<sizeof(T)>(&sPre[1 * bdim + me], pv.oy + m);
        cp_async<sizeof(T)>(&sPre[2 * bdim + me], pv.oz + m);
        cp_async<sizeof(T)>(&sPre[3 * bdim + me], pv.px + m);
        cp_async<sizeof(T)>(&sPre[4 * bdim + me], pv.py + m);
        cp_async<sizeof(T)>(&sPre[5 * bdim + me], pv.pz + m);
    };
    const int ntiles = t.ntx * t.nty * t.ntz;
    const int T3 = t.tx * t.ty * t.tz;
    const bool ax = g.nx > 1, ay = g.y3, az = g.z3;
    const int hx = ax ? kMoverHalo : 0, hy = ay ? kMoverHalo : 0, hz = az ? kMoverHalo : 0;
    const int nsx = ax ? 1 : 0, nsy = ay ? mb.nbx : 0, nsz = az ? mb.nbx * mb.nby : 0;
    const int csx = ax ? 1 : 0, csy = ay ? mb.cbx : 0, csz = az ? mb.cbx * mb.cby : 0;
    // (in the particle precision already: conversions from the FP64 grid
    // parameters run on the FP64 pipe, and the compiler repeats them in the
    // loop rather than hold their results)
    const T dt = K.dt, eta = K.eta, edt = K.edt, redt = K.redt;
    const T id[3] = {K.id[0], K.id[1], K.id[2]};
    const int nn[3] = {g.nx, g.ny, g.nz};
    const int parts = kRows ? nparts : 1;
    const int nrows = kRows ? S.ns * (t.ty / o.ty) * (t.tz / o.tz) : 0;
    RowTable rows(sPreCell + blockDim.x, nrows);   // (kRows)
    for (int work = blockIdx.x; work < ntiles * parts; work += gridDim.x) {
        const int tile = work / parts, part = work - tile * parts;
        const int ti = tile % t.ntx, tj = (tile / t.ntx) % t.nty, tk = tile / (t.ntx * t.nty);
        const int x0 = box_start(o.ntx, ti, t.ntx) * o.tx, y0 = box_start(o.nty, tj, t.nty) * o.ty,
                  z0 = box_start(o.ntz, tk, t.ntz) * o.tz;
        __syncthreads();   // previous tile's particles are done with the blocks
        for (int e = threadIdx.x; e < mb.NB; e += blockDim.x) {
            const int lx = e % mb.nbx, ly = (e / mb.nbx) % mb.nby, lz = e / (mb.nbx * mb.nby);
            const long long gid = linw_any(g, x0 - hx + lx, y0 - hy + ly, z0 - hz + lz);
#pragma unroll
            for (int c = 0; c < 3; ++c) sE[c * mb.NB + e] = T(E[c * g.N + gid]);
            if constexpr (kVec) {
                sEt4[e] = make_float4(float(Et[gid]), float(Et[g.N + gid]), float(Et[2 * g.N + gid]), 0.f);
            } else {
#pragma unroll
                for (int c = 0; c < 3; ++c) sEt[c * mb.NB + e] = T(Et[c * g.N + gid]);
            }
        }
        for (int e = threadIdx.x; e < mb.CB; e += blockDim.x) {
            const int lx = e % mb.cbx, ly = (e / mb.cbx) % mb.cby, lz = e / (mb.cbx * mb.cby);
            const long long gid = linw_any(g, x0 - hx - (ax ? 1 : 0) + lx, y0 - hy - (ay ? 1 : 0) + ly,
                                           z0 - hz - (az ? 1 : 0) + lz);
            if constexpr (kVec) {
                sB4[e] = make_float4(float(B[gid]), float(B[g.N + gid]), float(B[2 * g.N + gid]), 0.f);
            } else {
#pragma unroll
                for (int c = 0; c < 3; ++c) sB[c * mb.CB + e] = T(B[c * g.N + gid]);
            }
        }
        if constexpr (kRows) rows.fill(S, o, t, ti, tj, tk);
        __syncthreads();
        // moves particle n of species s, staged in this thread's slot, whose copy
        // of the next one `refill` starts once the slot is read
        auto move = [&](int s, const PartView<T>& p, T beta, T qdt, T mm, int n, auto refill) {
            const int bdim = blockDim.x, me = threadIdx.x;
            const int cell_n = sPreCell[me];
            const T pu[3] = {sPre[0 * bdim + me], sPre[1 * bdim + me], sPre[2 * bdim + me]};
            const T pm[3] = {sPre[3 * bdim + me], sPre[4 * bdim + me], sPre[5 * bdim + me]};
            refill();
            cp_async_commit();
            int ci[3];
            decode(g, cell_n, ci[0], ci[1], ci[2]);
            // A position (cell c, offset u) is located once: its node and cell
            // stencils in the staged block (bases, upper weights), shared by the
            // two or three gathers there; a stencil that leaves the block
            // gathers from the FP64 grids.
            struct Loc {
                bool inb;
                int nbase, cbase;
                T wn[3], wc[3];
            };
            // from tile-local cells l (the block holds l in [-h, t - 1 + h])
            auto locate_l = [&](const int l[3], const T u[3], Loc& L) {
                L.inb = l[0] >= -hx && l[0] <= t.tx - 1 + hx && l[1] >= -hy && l[1] <= t.ty - 1 + hy &&
                        l[2] >= -hz && l[2] <= t.tz - 1 + hz;
                if (!L.inb) return;
                int lo[3];
#pragma unroll
                for (int a = 0; a < 3; ++a) {
                    // upper weights: u of the nodes (c, c + 1); of the cell
                    // pair (c - 1, c) below the centre u + 1/2, (c, c + 1)
                    // above it u - 1/2
                    const bool act = nn[a] > 1, below = act && u[a] < T(0.5);
                    L.wn[a] = act ? u[a] : T(0);
                    L.wc[a] = act ? u[a] + (below ? T(0.5) : T(-0.5)) : T(0);
                    lo[a] = below ? l[a] - 1 : l[a];
                }
                L.nbase = (l[2] + hz) * nsz + (l[1] + hy) * nsy + (l[0] + hx) * nsx;
                const int ex = ax ? 1 : 0, ey = ay ? 1 : 0, ez = az ? 1 : 0;
                L.cbase = (lo[2] + hz + ez) * csz + (lo[1] + hy + ey) * csy + (lo[0] + hx + ex) * csx;
            };
            // from global cells c: the periodic image inside the block, if any
            auto locate = [&](const int c[3], const T u[3], Loc& L, int l[3]) {
                if (!(local_axis(c[0], x0, t.tx, hx, g.nx, l[0]) && local_axis(c[1], y0, t.ty, hy, g.ny, l[1]) &&
                      local_axis(c[2], z0, t.tz, hz, g.nz, l[2]))) {
                    L.inb = false;
                    return;
                }
                locate_l(l, u, L);
            };
            // gathers at a located position inside the block: E^theta
            // (nodes, corner weights w) and B^n (cells), float4 blocks for FP32
            auto gatEt = [&](const Loc& L, const T w[8], T out[3]) {
                if constexpr (kVec) gather3(sEt4, L.nbase, nsx, nsy, nsz, w, out);
                else gather3<T, kFlat>(sEt, mb.NB, L.nbase, nsx, nsy, nsz, w, out);
            };
            auto gatB = [&](const Loc& L, T out[3]) {
                T w[8];
                corners<T, kFlat>(L.wc[0], L.wc[1], L.wc[2], w);
                if constexpr (kVec) gather3(sB4, L.cbase, csx, csy, csz, w, out);
                else gather3<T, kFlat>(sB, mb.CB, L.cbase, csx, csy, csz, w, out);
            };
            auto defer = [&]() { atomicOr(&S.defer[s][n >> 5], 1u << (n & 31)); };
            T u0[3] = {pu[0], pu[1], pu[2]};
            T mom0[3] = {pm[0], pm[1], pm[2]};
            T gam, v[3];
            gamma_vel<T>(mom0, mm, gam, v);
            T e[3], e0[3], b[3], al[9];
            Loc L0;
            int l0[3];
            locate(ci, u0, L0, l0);
            if (!L0.inb) {
                defer();
                return;
            }
            {
                T w[8];
                corners<T, kFlat>(L0.wn[0], L0.wn[1], L0.wn[2], w);
                gather3<T, kFlat>(sE, mb.NB, L0.nbase, nsx, nsy, nsz, w, e0);
                gatEt(L0, w, e);
            }
            gatB(L0, b);
            alpha_tensor<T>(beta, v, gam, e0, b, al);
            T vxb[3] = {v[1] * b[2] - v[2] * b[1], -v[0] * b[2] + v[2] * b[0], v[0] * b[1] - v[1] * b[0]};
            T pnew[3];
#pragma unroll
            for (int d = 0; d < 3; ++d) pnew[d] = mom0[d] + (e[d] + vxb[d]) * qdt;
            T vnew[3];
            evaluate_velocity<T>(pnew, mm, vnew);
            T mv[3];
#pragma unroll
            for (int d = 0; d < 3; ++d) mv[d] = v[d] * (T(1) - eta) + vnew[d] * eta;
            if constexpr (kWall) {
                if (wall_left_of<T>(ci[0], u0[0], (mv[0] * edt) * id[0])) {
                    wall_reflect_trial<T>(g, ci, u0, mv, vnew, mm, edt, redt, id, pnew);
                    p.px[n] = pnew[0]; p.py[n] = pnew[1]; p.pz[n] = pnew[2];
                    p.ox[n] = u0[0]; p.oy[n] = u0[1]; p.oz[n] = u0[2];
                    p.cell[n] = tristan_escaped<T>(g, ci[0], u0[0]) ? -1 : (int)lin(g, ci[0], ci[1], ci[2]);
                    return;
                }
            }
            T vh[3];
#pragma unroll
            for (int a = 0; a < 3; ++a)
                vh[a] = (al[3 * a] * gam) * v[0] + (al[3 * a + 1] * gam) * v[1] + (al[3 * a + 2] * gam) * v[2];
            const T momNorm = (mom0[0] * mom0[0] + mom0[1] * mom0[1] + mom0[2] * mom0[2]);
            T err = ((mom0[0] - pnew[0]) * (mom0[0] - pnew[0]) + (mom0[1] - pnew[1]) * (mom0[1] - pnew[1]) +
                             (mom0[2] - pnew[2]) * (mom0[2] - pnew[2]));
            const T dxN = K.dx2;
            T cerr = dxN;
            T newDisp[3] = {mv[0] * edt, mv[1] * edt, mv[2] * edt};
            T prevDisp[3];
            int it = 0;
            bool reflected = false, left = false;
            while (picard_continue<T>(err, momNorm, cerr, dxN, it)) {
                ++it;
                const T prevMom[3] = {pnew[0], pnew[1], pnew[2]};
#pragma unroll
                for (int d = 0; d < 3; ++d) prevDisp[d] = newDisp[d];
                T re[3];
#pragma unroll
                for (int a = 0; a < 3; ++a) re[a] = al[3 * a] * e[0] + al[3 * a + 1] * e[1] + al[3 * a + 2] * e[2];
#pragma unroll
                for (int d = 0; d < 3; ++d) mv[d] = vh[d] + re[d] * beta;
#pragma unroll
                for (int d = 0; d < 3; ++d) newDisp[d] = mv[d] * edt;
                if constexpr (kWall) {
                    if (wall_left_of<T>(ci[0], u0[0], newDisp[0] * id[0])) {
                        wall_reflect_trial<T>(g, ci, u0, mv, vnew, mm, edt, redt, id, pnew);
                        reflected = true;
                        break;
                    }
                }
                // the trial position x^n + newDisp: the offsets as advance_axis
                // forms them, the cell in tile-local terms (no periodic wrap)
                T tu[3];
                int tl[3];
                Loc L1;
#pragma unroll
                for (int d = 0; d < 3; ++d) {
                    const T sd = u0[d] + newDisp[d] * id[d];
                    const T fd = dev_floor(sd);
                    T ud = sd - fd;
                    int cd = l0[d] + (int)fd;
                    if (ud >= T(1)) { ud -= T(1); cd += 1; }
                    tl[d] = nn[d] > 1 ? cd : 0;
                    tu[d] = ud;
                }
                locate_l(tl, tu, L1);
                if (!L1.inb) {
                    left = true;
                    break;
                }
                {
                    T w[8];
                    corners<T, kFlat>(L1.wn[0], L1.wn[1], L1.wn[2], w);
                    gatEt(L1, w, e);
                }
                gatB(L1, b);
                const T mvxb[3] = {mv[1] * b[2] - mv[2] * b[1], -mv[0] * b[2] + mv[2] * b[0], mv[0] * b[1] - mv[1] * b[0]};
#pragma unroll
                for (int d = 0; d < 3; ++d) pnew[d] = mom0[d] + (e[d] + mvxb[d]) * qdt;
                err = ((prevMom[0] - pnew[0]) * (prevMom[0] - pnew[0]) +
                               (prevMom[1] - pnew[1]) * (prevMom[1] - pnew[1]) +
                               (prevMom[2] - pnew[2]) * (prevMom[2] - pnew[2]));
                cerr = ((prevDisp[0] - newDisp[0]) * (prevDisp[0] - newDisp[0]) +
                                (prevDisp[1] - newDisp[1]) * (prevDisp[1] - newDisp[1]) +
                                (prevDisp[2] - newDisp[2]) * (prevDisp[2] - newDisp[2]));
            }
            if (left) {   // nothing written yet: the deferred pass moves it from the start
                defer();
                return;
            }
            if (!reflected) {
                if constexpr (kWall) {
                    const int o = wall_final_x<T>(g, ci[0], u0[0], (mv[0] * dt) * id[0]);
                    if (o == 2) { p.cell[n] = -1; return; }   // escaped through the open boundary
                    if (o == 1) pnew[0] = -pnew[0];
#pragma unroll
                    for (int d = 1; d < 3; ++d) advance_axis<T>(u0[d], ci[d], (mv[d] * dt) * id[d], nn[d]);
                } else {
#pragma unroll
                    for (int d = 0; d < 3; ++d) advance_axis<T>(u0[d], ci[d], (mv[d] * dt) * id[d], nn[d]);
                }
            }
            p.px[n] = pnew[0]; p.py[n] = pnew[1]; p.pz[n] = pnew[2];
            p.ox[n] = u0[0]; p.oy[n] = u0[1]; p.oz[n] = u0[2];
            p.cell[n] = kWall && tristan_escaped<T>(g, ci[0], u0[0]) ? -1 : (int)lin(g, ci[0], ci[1], ci[2]);
        };
        if constexpr (kRows) {
            const int lane = threadIdx.x & 31, warps = blockDim.x >> 5, per = (t.ty / o.ty) * (t.tz / o.tz);
            int c = part * warps + (threadIdx.x >> 5), at = 0, n0 = 0, pe = 0, s = 0;   // chunk, row, first particle, row's end, species
            auto seek = [&]() {
                at = rows.row_of(c, at, lane);
                const bool some = c < rows.before[nrows];
                n0 = some ? rows.first[at] + 32 * (c - rows.before[at]) : 0;
                pe = some ? rows.end[at] : 0;
                s = at / per;
            };
            seek();
            if (lane < pe - n0) stage(S.p[s], n0 + lane);
            cp_async_commit();
            while (n0 < pe) {
                cp_async_wait_all();   // this thread's particle (its own slot)
                const int n = n0 + lane, here = pe - n0, sn = s;
                c += parts * warps;
                seek();
                auto refill = [&]() {
                    if (lane < pe - n0) stage(S.p[s], n0 + lane);
                };
                if (lane < here) {
                    move(sn, S.p[sn], K.beta[sn], K.qdt[sn], K.m[sn], n, refill);
                } else {
                    refill();
                    cp_async_commit();
                }
                __syncwarp();
            }
        } else {
            for (int s = 0; s < S.ns; ++s) {
                const PartView<T> p = S.p[s];
                const T beta = K.beta[s], qdt = K.qdt[s], mm = K.m[s];
                const int b0 = S.off[s][tile * T3], b1 = S.off[s][(tile + 1) * T3], step = blockDim.x;
                if (b0 + (int)threadIdx.x < b1) stage(p, b0 + threadIdx.x);
                cp_async_commit();
                for (int n = b0 + threadIdx.x; n < b1; n = b1 - n > step ? n + step : b1) {   // (no int overflow)
                    cp_async_wait_all();   // this thread's particle n (its own slot)
                    move(s, p, beta, qdt, mm, n, [&]() {
                        if (b1 - n > step) stage(p, n + step);
                    });
                }
            }
        }
    }
}

}  // namespace pic
