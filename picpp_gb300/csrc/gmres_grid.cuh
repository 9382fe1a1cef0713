// gmres_grid.cuh -- a whole GMRES solve of the implicit Maxwell system in one
// cooperative launch: the operator, the orthogonalisation, the Givens
// rotations, the stopping rule and the solution update, with grid-wide
// barriers between phases.
//
// What bounds it: the FP64 pipe (two multiply-adds per SM and clock, so a
// warp instruction holds it for 16 clocks) on large systems, the barriers'
// latency (a few microseconds per iteration) on small ones.  So
//   * a thread owns the same elements in every phase, and only mu v and the
//     operator's stencil read what other threads wrote: three barriers per
//     iteration (after mu v, after the dot products, after the norm), where
//     separate kernels took 7 to 60 launches and a host round trip;
//   * the sums over lanes are a transposed reduction (16 values with 16
//     additions per lane instead of 80): with one block_sum per value the
//     additions of the reductions took longer than the dot products;
//   * every CTA adds the CTAs' partial sums and does the small algebra
//     (Hessenberg column, Givens rotation, stopping test) itself, in the same
//     order, so that all CTAs agree without another exchange.  All sums have
//     a fixed order: a solve is reproducible bit for bit.
// What it measured against the kernel-per-operation form stands at
// launch_gmres_grid (gmres_launch.cuh).
#pragma once
#include <algorithm>
#include "common.cuh"
#include "kernels.hpp"

namespace pic {

// Values of one dot-product phase at most.
__host__ __device__ inline int gmres_vals(int cols) { return 2 * (cols + 2); }
inline size_t gmres_smem(int cols, int workers, bool reference) {
    const size_t tri = (size_t)cols * (cols + 1) / 2;
    return sizeof(double) * (tri * (reference ? 2 : 1) + 4 * (size_t)(cols + 2) + gmres_vals(cols) +
                             std::max<size_t>((size_t)gmres_vals(cols) * (workers / 32), 2 * (size_t)workers));
}

// NW worker threads own the vectors' elements, one more warp does the small
// algebra beside them; KB basis vectors per pass over the elements.  kNode: a
// worker owns whole nodes, the elements c, N + c, 2N + c (mu v and the decoding
// of the node once for all three, more independent operations in flight);
// else single elements (three times the threads, for small boxes).
template <int NW, int KB, bool kNode>
struct GmresCta {
    const GmresArgs& A;
    double *sR, *sL, *sg, *scs, *ssn, *sy, *sh, *sw;   // R and Gram triangles, rotated right part, rotations, y, sums, warps' sums
    bool* bad;
    unsigned target = 0;                                // arrivals that complete the next barrier

    __device__ bool worker() const { return threadIdx.x < NW; }
    // Items of a worker: first, first + stride, ... < items; item c holds the
    // elements c + d N, d < kD.
    static constexpr int kD = kNode ? 3 : 1;
    __device__ long long items() const { return kNode ? A.g.N : 3 * A.g.N; }
    __device__ long long first() const { return worker() ? blockIdx.x * (long long)NW + threadIdx.x : items(); }
    __device__ long long stride() const { return (long long)gridDim.x * NW; }

    // Barrier over the grid; false when it gave up (then every thread leaves).
    __device__ bool barrier() {
        target += gridDim.x;
        __syncthreads();
        if (threadIdx.x == 0) {
            __threadfence();
            atomicAdd(A.bar, 1u);
            unsigned polls = 0, seen;
            do {
                asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(seen) : "l"(A.bar) : "memory");
            } while ((int)(seen - target) < 0 && ++polls < A.polls);
            *bad = (int)(seen - target) < 0;
            if (*bad) A.bar[1] = 1u;
            __threadfence();
        }
        __syncthreads();
        return !*bad;
    }

    // Sums over a warp's lanes of acc[0..KA): lane pairs exchange halves of the
    // values, so KA values take about KA additions per lane.  Lane l ends with
    // the sum of value l / (32 / KA).
    template <int KA>
    __device__ double warp_sums(double acc[KA]) const {
        const int lane = threadIdx.x & 31;
        int w = 16;
#pragma unroll
        for (int h = KA / 2; h >= 1; h >>= 1, w >>= 1) {
            const bool up = (lane & w) != 0;
#pragma unroll
            for (int i = 0; i < h; ++i) {
                const double send = up ? acc[i] : acc[i + h];
                const double keep = up ? acc[i + h] : acc[i];
                acc[i] = keep + __shfl_xor_sync(0xffffffffu, send, w);
            }
        }
#pragma unroll
        for (int o = 16 / KA; o >= 1; o >>= 1) acc[0] += __shfl_xor_sync(0xffffffffu, acc[0], o);
        return acc[0];
    }
    __device__ double* warp_row() const { return sw + (threadIdx.x >> 5) * gmres_vals(A.cols); }
    // One value per thread: its warp's sum to value v.
    __device__ void warp_sum1(double s, int v) {
        if (!worker()) return;
        s = warp_sum(s);
        if ((threadIdx.x & 31) == 0) warp_row()[v] = s;
    }
    // The CTA's sums of K values from its warps' to the partials of buffer `buf`
    // (0: up to gmres_vals values, 1: up to two).  A CTA may be collecting from a
    // buffer until it arrives at the next barrier, so between a collect and the
    // next publish of the same buffer there is always one.
    __device__ void publish(int K, int buf) {
        const int kv = gmres_vals(A.cols);
        __syncthreads();
        double* dst = A.part + (buf ? (long long)gridDim.x * kv + blockIdx.x * 2 : (long long)blockIdx.x * kv);
        for (int v = threadIdx.x; v < K; v += blockDim.x) {
            double s = 0.0;
#pragma unroll 8
            for (int w = 0; w < NW / 32; ++w) s += sw[w * kv + v];
            dst[v] = s;
        }
    }
    // After the barrier: the grid's sums to sh[0..K) (valid after the closing
    // __syncthreads): P lanes per row of partials (P a power of two >= K, at
    // most 32), the rows dealt to NW / P groups, the groups' sums added in order.
    __device__ void collect(int K, int buf) {
        const int kv = gmres_vals(A.cols), ld = buf ? 2 : kv;
        const double* src = A.part + (buf ? (long long)gridDim.x * kv : 0);
        const int P = K <= 1 ? 1 : (K <= 8 ? 8 : (K <= 16 ? 16 : 32)), groups = NW / P > (int)gridDim.x ? gridDim.x : NW / P;
        for (int v0 = 0; v0 < K; v0 += P) {
            const int v = v0 + threadIdx.x % P, gr = threadIdx.x / P;
            if (gr < groups && v < K) {
                double s = 0.0;
#pragma unroll 4
                for (int c = gr; c < (int)gridDim.x; c += groups) s += __ldcg(&src[(long long)c * ld + v]);
                sw[gr * P + threadIdx.x % P] = s;
            }
            __syncthreads();
            if (threadIdx.x < 32) {
                // 32 / P strands per value, then a shuffle over the strands
                const int vv = v0 + threadIdx.x % P, strand = threadIdx.x / P;
                double s = 0.0;
                if (vv < K)
#pragma unroll 4
                    for (int q = strand; q < groups; q += 32 / P) s += sw[q * P + threadIdx.x % P];
                for (int o = 16; o >= P; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
                if (vv < K && strand == 0) sh[vv] = s;
            }
            __syncthreads();
        }
    }

    // |a|^2 over the grid.
    __device__ bool norm2(const double* a, double& out) {
        double s = 0.0;
        for (long long c = first(); c < items(); c += stride())
#pragma unroll
            for (int d = 0; d < kD; ++d) s = fma(a[c + d * A.g.N], a[c + d * A.g.N], s);
        warp_sum1(s, 0);
        publish(1, 1);
        if (!barrier()) return false;
        collect(1, 1);
        out = sh[0];
        return true;
    }

    // Component and node of element e.
    __device__ void where(long long e, int& a, long long& c) const {
        const long long N = A.g.N;
        a = e >= 2 * N ? 2 : (e >= N ? 1 : 0);
        c = e - a * N;
    }

    // dst = src * f, mx = mu dst (kDiv: src / f, the reference's division)
    template <bool kDiv>
    __device__ void scale_mu(double* dst, const double* src, double f) {
        const long long N = A.g.N;
        for (long long e = first(); e < items(); e += stride()) {
            int a = 0;
            long long c = e;
            if (!kNode) where(e, a, c);
            const double s0 = src[c], s1 = src[N + c], s2 = src[2 * N + c];
            const double v0 = kDiv ? s0 / f : s0 * f, v1 = kDiv ? s1 / f : s1 * f, v2 = kDiv ? s2 / f : s2 * f;
#pragma unroll
            for (int d = 0; d < kD; ++d) {
                const int q = kNode ? d : a;
                const double* m = A.mu + 3 * q * N + c;
                dst[c + q * N] = q == 0 ? v0 : (q == 1 ? v1 : v2);
                A.mx[c + q * N] = m[0] * v0 + m[N] * v1 + m[2 * N] * v2;
            }
        }
    }

    // The elements of item e of (A - sig) v from v and mx = mu v (the terms of
    // k_maxwell_stencil, and the wall box's boundary rows of k_wall_rows).
    __device__ void rows(long long e, const double* v, double sig, double y[kD]) const {
        const GridP& g = A.g;
        const long long N = g.N;
        int a = 0;
        long long c = e;
        if (!kNode) where(e, a, c);
        int i, j, k;
        decode(g, (int)c, i, j, k);
        if (g.wall && (i == 0 || i >= g.nx - 2)) {
#pragma unroll
            for (int d = 0; d < kD; ++d) {
                const double x = v[e + d * N];
                double r = x;
                if (i == 0 && (kNode ? d : a) == 0) r -= v[e + 1];
                y[d] = fma(-sig, x, r);
            }
            return;
        }
        const long long sy = g.nx, sz = (long long)g.nx * g.ny;
        const long long ux = i + 1 == g.nx ? -(long long)(g.nx - 1) : 1, dx = i == 0 ? g.nx - 1 : -1;
        const long long uy = j + 1 == g.ny ? -(g.ny - 1) * sy : sy, dy = j == 0 ? (g.ny - 1) * sy : -sy;
        const long long uz = k + 1 == g.nz ? -(g.nz - 1) * sz : sz, dz = k == 0 ? (g.nz - 1) * sz : -sz;
        if constexpr (kNode) {
#pragma unroll
            for (int q = 0; q < 3; ++q) y[q] = one_row(q, c, v, sig, ux, dx, uy, dy, uz, dz);
        } else {
            y[0] = one_row(a, c, v, sig, ux, dx, uy, dy, uz, dz);
        }
    }
    __device__ __forceinline__ double one_row(int a, long long c, const double* v, double sig, long long ux, long long dx,
                                              long long uy, long long dy, long long uz, long long dz) const {
        const long long N = A.g.N;
        const long long e = a * N + c;
        // the row's own axis a and the two others b, d
        const int b = a == 2 ? 0 : a + 1, d = a == 0 ? 2 : a - 1;
        const long long ua = a == 0 ? ux : (a == 1 ? uy : uz), da = a == 0 ? dx : (a == 1 ? dy : dz);
        const long long ub = b == 0 ? ux : (b == 1 ? uy : uz), db = b == 0 ? dx : (b == 1 ? dy : dz);
        const long long ud = d == 0 ? ux : (d == 1 ? uy : uz), dd = d == 0 ? dx : (d == 1 ? dy : dz);
        const bool ha = A.oc.has[a], hb = A.oc.has[b], hd = A.oc.has[d];
        const double ka = A.oc.kd2[a], kb = A.oc.kd2[b], kd = A.oc.kd2[d];
        const double* x = v + e;
        const double* w = A.mx + e;
        double diag = 1.0 - sig, c1 = 1.0;
        if (ha) { diag += 2.0 * ka; c1 += 2.0 * ka; }
        if (hb) diag += 2.0 * kb;
        if (hd) diag += 2.0 * kd;
        double y = fma(-c1, w[0], diag * x[0]);
        if (ha) y = fma(ka, (w[ua] + w[da]) - (x[ua] + x[da]), y);
        if (hb) y = fma(-kb, x[ub] + x[db], y);
        if (hd) y = fma(-kd, x[ud] + x[dd], y);
        if (ha && hb) {
            const double* q = A.mx + b * N + c;
            y = fma(A.oc.kx4[a][b], (q[ua + ub] - q[ua + db]) - (q[da + ub] - q[da + db]), y);
        }
        if (ha && hd) {
            const double* q = A.mx + d * N + c;
            y = fma(A.oc.kx4[a][d], (q[ua + ud] - q[ua + dd]) - (q[da + ud] - q[da + dd]), y);
        }
        return y;
    }

    // Dot products of w with k vectors to values 0 .. k - 1: the basis, self:
    // w itself as the last; kTwo: also of the vector u with the first k - 1 of
    // them, to values k .. 2 k - 2.
    template <bool kTwo>
    __device__ int dots(int k, const double* w, const double* u, bool self) {
        constexpr int KA = kTwo ? 2 * KB : KB;
        const long long L = 3 * A.g.N;
        const int K = kTwo ? 2 * k - 1 : k;
        if (worker())
            for (int k0 = 0; k0 < k; k0 += KB) {
                double acc[KA] = {};
                for (long long c = first(); c < items(); c += stride())
#pragma unroll
                    for (int d = 0; d < kD; ++d) {
                        const long long e = c + d * A.g.N;
                        const double wd = w[e];
                        const double ud = kTwo ? u[e] : 0.0;
                        const double* v = A.V + (long long)k0 * L + e;
                        double vm[KB];
#pragma unroll
                        for (int m = 0; m < KB; ++m)
                            vm[m] = k0 + m < k - (self ? 1 : 0) ? v[(long long)m * L] : wd;
#pragma unroll
                        for (int m = 0; m < KB; ++m)
                            if (k0 + m < k) {
                                acc[m] = fma(vm[m], wd, acc[m]);
                                if (kTwo) acc[KB + m] = fma(vm[m], ud, acc[KB + m]);
                            }
                    }
                const double s = warp_sums<KA>(acc);
                constexpr int per = 32 / KA;   // lanes that hold one value
                const int lane = threadIdx.x & 31, i = lane / per, m = k0 + i % KB;
                if (lane % per == 0) {
                    if (i < KB) {
                        if (m < k) warp_row()[m] = s;
                    } else if (m < k - 1) {
                        warp_row()[k + m] = s;
                    }
                }
            }
        publish(K, 0);
        return K;
    }

    // w -= sum_{m < k} sh[m] V[m], then |w|^2 to value 0 of the second buffer.
    __device__ void update(double* w, int k) {
        const long long L = 3 * A.g.N;
        double nrm = 0.0;
        for (long long c = first(); c < items(); c += stride()) {
            double s[kD];
#pragma unroll
            for (int d = 0; d < kD; ++d) s[d] = w[c + d * A.g.N];
            const double* v = A.V + c;
#pragma unroll 4
            for (int m = 0; m < k; ++m)
#pragma unroll
                for (int d = 0; d < kD; ++d) s[d] = fma(-sh[m], v[(long long)m * L + d * A.g.N], s[d]);
#pragma unroll
            for (int d = 0; d < kD; ++d) {
                w[c + d * A.g.N] = s[d];
                nrm = fma(s[d], s[d], nrm);
            }
        }
        warp_sum1(nrm, 0);
        publish(1, 1);
    }

    // Column j of the least-squares problem: entries sy[0..j], hn below them
    // (one thread of every CTA, the same arithmetic in all).
    __device__ void givens(int j, double hn) {
        double* col = sR + (long long)j * (j + 1) / 2;
        double t = sy[0];
        for (int i = 0; i < j; ++i) {
            const double lo = sy[i + 1];
            col[i] = fma(scs[i], t, ssn[i] * lo);
            t = fma(-ssn[i], t, scs[i] * lo);
        }
        const double mod = sqrt(fma(t, t, hn * hn));   // (entries of the order of the operator's, about 1)
        const double inv = mod > 0 ? 1.0 / mod : 0.0;
        const double cs = mod > 0 ? t * inv : 1.0, sn = hn * inv;
        col[j] = mod;
        scs[j] = cs;
        ssn[j] = sn;
        sg[j + 1] = -sn * sg[j];
        sg[j] = cs * sg[j];
    }
    // y = R^{-1} g over k columns, to sy (first warp).
    __device__ void backsolve(int k) {
        __syncthreads();
        const int lane = threadIdx.x;
        if (lane < 32) {
            for (int i = lane; i < k; i += 32) sy[i] = sg[i];
            __syncwarp();
            for (int i = k - 1; i >= 0; --i) {
                const double* col = sR + (long long)i * (i + 1) / 2;
                const double yi = col[i] != 0 ? sy[i] / col[i] : 0.0;
                __syncwarp();
                for (int q = lane; q < i; q += 32) sy[q] = fma(-col[q], yi, sy[q]);
                if (lane == 0) sy[i] = yi;
                __syncwarp();
            }
        }
        __syncthreads();
    }
    __device__ void zero(double* a) const {
        for (long long c = first(); c < items(); c += stride())
#pragma unroll
            for (int d = 0; d < kD; ++d) a[c + d * A.g.N] = 0.0;
    }
    __device__ void finish(double status, double its, double restarts, double rel) {
        if (blockIdx.x == 0 && threadIdx.x == 0) {
            A.out[kGmStatus] = status; A.out[kGmIterations] = its; A.out[kGmRestarts] = restarts; A.out[kGmRel] = rel;
        }
    }
};

__device__ __forceinline__ bool finite_bits(double v) { return (__double2hiint(v) & 0x7ff00000) != 0x7ff00000; }

// Restarted GMRES(cols): classical Gram-Schmidt with a second pass where the
// first leaves less than 1/sqrt(2) of the vector, true residual at every
// restart.  The vector that is orthogonalised is A v_j - s v_j - t v_{j-1} with
// s = h_{j-1,j-1} and t = h_{j,j-1} of the column before (added back to the
// column's entries): the operator is close to a multiple of the identity and
// nearly symmetric, so A v_j itself is almost in the basis and every column
// took the second pass.
// Reference: generalizedMinimalResidualMethod semantics
// (PIC++/specialmath.cpp:367-671), unrestarted, modified Gram-Schmidt; its
// coefficients r_m = V_m . (w - sum_{j<m} r_j V_j) come from one pass over the
// basis as the forward substitution r_m = V_m . w - sum_{j<m} (V_m . V_j) r_j
// with the basis' own products V_m . V_j (the inverse compact WY form of
// modified Gram-Schmidt, Swirydowicz et al., Numer. Linear Algebra Appl. 28,
// e2343, 2021), one barrier instead of one per basis vector.
template <int NW, int KB, bool kNode, bool kRef>
__global__ void __launch_bounds__(NW + 32) k_gmres_grid(const __grid_constant__ GmresArgs A) {
    extern __shared__ __align__(16) double gm_smem[];
    __shared__ bool s_bad;
    const int C = A.cols;
    const long long N = A.g.N, L = 3 * N;
    using Cta = GmresCta<NW, KB, kNode>;
    constexpr int kD = Cta::kD;
    Cta T{A};
    T.bad = &s_bad;
    double* p = gm_smem;
    T.sR = p; p += (long long)C * (C + 1) / 2;
    T.sL = p; if (kRef) p += (long long)C * (C + 1) / 2;
    T.sg = p; p += C + 2;
    T.scs = p; p += C + 2;
    T.ssn = p; p += C + 2;
    T.sy = p; p += C + 2;
    T.sh = p; p += gmres_vals(C);
    T.sw = p;
    auto Vp = [&](int j) { return A.V + (long long)j * L; };

    // |b|^2, and whether b or mu hold a non-finite entry
    double sum = 0.0, count = 0.0;
    for (long long c = T.first(); c < T.items(); c += T.stride())
#pragma unroll
        for (int d = 0; d < kD; ++d) {
            const long long e = c + d * N;
            const double v = A.b[e];
            sum = fma(v, v, sum);
            if (!(finite_bits(v) && finite_bits(A.mu[e]) && finite_bits(A.mu[L + e]) && finite_bits(A.mu[2 * L + e])))
                count = 1.0;
        }
    T.warp_sum1(sum, 0);
    T.warp_sum1(count, 1);
    T.publish(2, 0);   // (not buffer 1: the reference method's norm2 comes without a barrier between)
    if (!T.barrier()) return;
    T.collect(2, 0);
    if (T.sh[1] > 0) { T.finish(kGmNonFiniteSystem, 0, 0, 0); return; }
    const double bnorm = sqrt(T.sh[0]);
    if (bnorm == 0) {
        T.zero(A.x);
        T.finish(kGmOk, 0, 0, 0);
        return;
    }
    int total = 0, restarts = 0;
    double rel = 1.0, beta = bnorm, normR = 1.0;
    for (;;) {
        if (!kRef) {
            rel = beta / bnorm;
            if (!finite_bits(rel)) { T.finish(kGmNonFiniteResidual, total, restarts, rel); return; }
            if (rel <= A.tol || total >= A.max_iter) break;
            T.template scale_mu<false>(Vp(0), restarts ? A.r : A.b, 1.0 / beta);
            if (threadIdx.x == 0) T.sg[0] = beta;
            if (!T.barrier()) return;
        } else {
            T.template scale_mu<true>(Vp(0), A.b, bnorm);
            double n2;
            if (threadIdx.x == 0) T.sg[0] = 1.0;
            if (!T.norm2(Vp(0), n2)) return;   // (its barrier also orders mu v before the stencil)
            normR = sqrt(n2);
        }
        int j = 0;
        double s = 0.0, t = 0.0, hn = 0.0;
        const bool go = !kRef || (1.0 > A.tol && A.max_iter > 2);
        for (bool rotate = false; go;) {
            // the column's candidate and its dot products; beside the workers the
            // algebra warp rotates the column before and so tells whether this one
            // is needed (a stop wastes these two phases once)
            double* w = A.w;
            const double* vj = Vp(j);
            if (rotate && threadIdx.x == NW) T.givens(j - 1, hn);
            for (long long c = T.first(); c < T.items(); c += T.stride()) {
                double y[kD];
                T.rows(c, vj, kRef ? 0.0 : s, y);
#pragma unroll
                for (int d = 0; d < kD; ++d) {
                    if (!kRef && j > 0) y[d] = fma(-t, vj[c + d * N - L], y[d]);
                    w[c + d * N] = y[d];
                }
            }
            int K;
            if constexpr (kRef) K = T.template dots<true>(j + 1, w, vj, false);
            else K = T.template dots<false>(j + 2, w, nullptr, true);
            if (rotate) {   // (dots' __syncthreads stands between)
                const double g1 = fabs(T.sg[j]);
                if (kRef) rel = g1 / normR;
                if (kRef ? !(rel > A.tol) : g1 / bnorm <= A.tol) break;
            }
            if (!T.barrier()) return;
            T.collect(K, 0);
            double before2 = 0.0;
            if (kRef) {
                // sh: d_0 .. d_j, then V_j . V_0 .. V_j . V_{j-1}: row j of the
                // Gram triangle, and the forward substitution by the first warp
                double* row = T.sL + (long long)j * (j - 1) / 2;
                if (threadIdx.x < 32) {
                    for (int i = threadIdx.x; i < j; i += 32) row[i] = T.sh[j + 1 + i];
                    __syncwarp();
                    for (int q = 0; q < j; ++q) {
                        const double hq = T.sh[q];
                        for (int i = q + 1 + threadIdx.x; i <= j; i += 32)
                            T.sh[i] = fma(-T.sL[(long long)i * (i - 1) / 2 + q], hq, T.sh[i]);
                        __syncwarp();
                    }
                }
                __syncthreads();
            } else {
                before2 = T.sh[j + 1];
            }
            for (int i = threadIdx.x; i <= j; i += blockDim.x)
                T.sy[i] = T.sh[i] + (kRef ? 0.0 : (i == j ? s : (i == j - 1 ? t : 0.0)));
            T.update(w, j + 1);
            if (!T.barrier()) return;
            T.collect(1, 1);
            hn = sqrt(T.sh[0]);
            if (!kRef && !(hn >= 0.7071067811865476 * sqrt(fmax(before2, 0.0)))) {
                T.template dots<false>(j + 1, w, nullptr, false);
                if (!T.barrier()) return;
                T.collect(j + 1, 0);
                for (int i = threadIdx.x; i <= j; i += blockDim.x) T.sy[i] += T.sh[i];
                T.update(w, j + 1);
                if (!T.barrier()) return;
                T.collect(1, 1);
                hn = sqrt(T.sh[0]);
            }
            s = T.sy[j];
            t = hn;
            ++j;
            ++total;
            // the last column for certain: its rotation now, no candidate after it
            if (j == C || (kRef ? j + 2 >= A.max_iter : total >= A.max_iter || hn == 0)) {
                __syncthreads();
                if (threadIdx.x == NW) T.givens(j - 1, hn);
                __syncthreads();
                if (kRef) rel = fabs(T.sg[j]) / normR;
                break;
            }
            T.template scale_mu<false>(Vp(j), w, hn > 0 ? 1.0 / hn : 0.0);
            if (!T.barrier()) return;
            rotate = true;
        }
        T.backsolve(j);
        const double f = kRef ? bnorm : 1.0;
        for (long long c = T.first(); c < T.items(); c += T.stride())
#pragma unroll
            for (int d = 0; d < kD; ++d) {
                const long long e = c + d * N;
                double x = !kRef && restarts ? A.x[e] : 0.0;
#pragma unroll 8
                for (int m = 0; m < j; ++m) x += Vp(m)[e] * T.sy[m] * f;
                A.x[e] = x;
            }
        if (kRef) {
            T.finish(kGmOk, total, 0, rel);
            return;
        }
        if (!T.barrier()) return;
        T.template scale_mu<false>(A.w, A.x, 1.0);   // (mu x)
        if (!T.barrier()) return;
        for (long long c = T.first(); c < T.items(); c += T.stride()) {
            double y[kD];
            T.rows(c, A.x, 0.0, y);
#pragma unroll
            for (int d = 0; d < kD; ++d) A.r[c + d * N] = A.b[c + d * N] - y[d];
        }
        ++restarts;
        double n2;
        if (!T.norm2(A.r, n2)) return;
        beta = sqrt(n2);
    }
    // a solve that never entered a cycle leaves x = 0
    if (!kRef && restarts == 0) T.zero(A.x);
    T.finish(rel <= A.tol ? kGmOk : kGmNotConverged, total, restarts, rel);
}

}  // namespace pic
