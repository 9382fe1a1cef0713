// diag.cuh -- diagnostics pass of updateDensityParameters
// (PIC++/momentum_collecting.cpp:760-1020): per species concentration,
// energy density and bulk velocity on cells, and the charge density.
#pragma once
#include "common.cuh"

namespace pic {

// Cell-weight deposit of one species: conc += w S / V, energy += w gamma m
// S / V, mom[3] += w p S / V (FP64 global atomics; a diagnostic, run every
// output interval).  Bound by the FP64 pipe (two lane operations per SM and
// clock): the products are factored, six for the eight weights' parts and five
// per corner, and the one division is by a constant (4.2 million particles:
// 852 us with each corner's weights multiplied out and p^2 divided by m^2).
// kTurn, for boxes of few cells with many particles each, where the adds to the few
// addresses are the time: each warp of a CTA begins at another corner (8^3 cells, 1,000
// per species and cell, FP32 and FP64: 1,277 and 1,346 us; all from the first corner 1,558 and
// 1,632, and with the weights multiplied out, which left more time between the
// adds, 1,387 and 1,395.  8^3 with 100: 115, 126, 130).
template <typename T, bool kTurn>
__global__ void __launch_bounds__(256) k_density_deposit(GridP g, PartView<T> p, double m, double w,
                                                         double* __restrict__ conc, double* __restrict__ energy,
                                                         double* __restrict__ mom) {
    const double wv = w / (g.dx * g.dy * g.dz), im2 = 1.0 / (m * m);
    for (long long n = blockIdx.x * (long long)blockDim.x + threadIdx.x; n < p.n;
         n += (long long)gridDim.x * blockDim.x) {
        int i, j, k;
        decode(g, p.cell[n], i, j, k);
        const double px = double(p.px[n]), py = double(p.py[n]), pz = double(p.pz[n]);
        const double gm = sqrt(fma(fma(px, px, fma(py, py, pz * pz)), im2, 1.0)) * m;
        int X[2], Y[2], Z[2];
        T wx[2], wy[2], wz[2];
        cell_w(p.ox[n], i, g.nx, X, wx); cell_w(p.oy[n], j, g.ny, Y, wy); cell_w(p.oz[n], k, g.nz, Z, wz);
        const double x0 = double(wx[0]) * wv, x1 = double(wx[1]) * wv;
        const double y0 = double(wy[0]), y1 = double(wy[1]), z0 = double(wz[0]), z1 = double(wz[1]);
        const double yz[4] = {y0 * z0, y1 * z0, y0 * z1, y1 * z1};
#pragma unroll
        for (int q = 0; q < 8; ++q) {
            const int c = kTurn ? (q + (int)(threadIdx.x >> 5)) & 7 : q;
            if ((!g.y3 && (c & 2)) || (!g.z3 && (c & 4))) continue;
            const long long id = lin(g, c & 1 ? X[1] : X[0], c & 2 ? Y[1] : Y[0], c & 4 ? Z[1] : Z[0]);
            const double s = (c & 1 ? x1 : x0) * (c & 4 ? (c & 2 ? yz[3] : yz[2]) : (c & 2 ? yz[1] : yz[0]));
            atomicAdd(&conc[id], s);
            atomicAdd(&energy[id], s * gm);
            atomicAdd(&mom[id], s * px);
            atomicAdd(&mom[g.N + id], s * py);
            atomicAdd(&mom[2 * g.N + id], s * pz);
        }
    }
}

}  // namespace pic
