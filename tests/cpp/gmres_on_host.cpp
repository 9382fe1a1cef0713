// gmres_on_host.cpp -- the one-launch GMRES kernel (csrc/gmres_grid.cuh) run on
// the CPU, a thread of the host per thread of the GPU: what tests of its
// exchanges between CTAs need and a GPU does not offer, a CTA held up at a
// point of choice.  The test that compiles this writes gmres_grid_host.cuh, the
// kernel's header with shared memory and the acquiring load given by functions of
// host_cuda.hpp.
//
//   gmres_on_host SYSTEM OUT late nth polls
// SYSTEM: int32 nx ny nz reference cols max_iter ctas, float64 dx dy dz dt theta
// cfix tol, then mu (9N) and b (3N).  CTA `late` waits between the nth barrier and the
// collection of partial sums that follows it (-1: none does); a barrier of the grid gives
// up after `polls` polls (0: as many as the library takes).  OUT: float64 status, iterations, restarts, residual, x (3N).
#include "host_cuda.hpp"

#include <cstdio>
#include <cstdlib>

#include "gmres_grid_host.cuh"

using namespace pic;

template <bool kRef>
static void run(const GmresArgs& a, int ctas) {
    constexpr int NW = 32;
    blockDim.x = NW + 32;
    gridDim.x = ctas;
    std::vector<std::unique_ptr<Cta>> cta;
    for (int c = 0; c < ctas; ++c) cta.push_back(std::make_unique<Cta>(NW + 32, gmres_smem(a.cols, NW, kRef)));
    std::vector<std::thread> threads;
    for (int c = 0; c < ctas; ++c)
        for (int t = 0; t < NW + 32; ++t)
            threads.emplace_back([&, c, t] {
                here = cta[c].get();
                threadIdx.x = t;
                blockIdx.x = c;
                k_gmres_grid<NW, 8, false, kRef>(a);
            });
    for (auto& t : threads) t.join();
}

int main(int argc, char** argv) {
    if (argc != 6) return 2;
    std::FILE* f = std::fopen(argv[1], "rb");
    int n[7];
    double d[7];
    if (!f || std::fread(n, 4, 7, f) != 7 || std::fread(d, 8, 7, f) != 7) return 2;
    GmresArgs a{};
    GridP& g = a.g;
    g.nx = n[0]; g.ny = n[1]; g.nz = n[2];
    g.N = (long long)n[0] * n[1] * n[2];
    g.dx = d[0]; g.dy = d[1]; g.dz = d[2]; g.dt = d[3]; g.theta = d[4];
    const long long L = 3 * g.N;
    a.reference = n[3]; a.cols = n[4]; a.max_iter = n[5];
    const int ctas = n[6];
    a.tol = d[6];
    a.oc.K = (g.theta * g.dt) * (g.theta * g.dt) * (d[5] * d[5]);
    for (int i = 0; i < 3; ++i) {
        a.oc.has[i] = n[i] > 1;
        a.oc.kd2[i] = a.oc.K / (d[i] * d[i]);
        for (int j = 0; j < 3; ++j) a.oc.kx4[i][j] = a.oc.K / (4 * d[i] * d[j]);
    }
    std::vector<double> mu(3 * L), b(L), x(L, -1.0), V((a.cols + 1) * L), mx(L), w(L), r(L),
        part(ctas * (gmres_vals(a.cols) + 2)), out(kGmOutLen);
    unsigned bar[2] = {0, 0};
    if (std::fread(mu.data(), 8, 3 * L, f) != (size_t)(3 * L) || std::fread(b.data(), 8, L, f) != (size_t)L) return 2;
    std::fclose(f);
    a.mu = mu.data(); a.b = b.data(); a.x = x.data(); a.V = V.data(); a.mx = mx.data(); a.w = w.data(); a.r = r.data();
    a.part = part.data(); a.bar = bar; a.out = out.data();
    a.polls = std::atoi(argv[5]) > 0 ? (unsigned)std::atoi(argv[5]) : kGmresPolls;
    if (a.polls != kGmresPolls) late_ms = 1000;   // longer than the others take for their polls
    late_cta = std::atoi(argv[3]);
    late_at = std::atoi(argv[4]);
    if (a.reference) run<true>(a, ctas);
    else run<false>(a, ctas);
    if (bar[1]) out[kGmStatus] = -1;   // a barrier gave up
    f = std::fopen(argv[2], "wb");
    if (!f) return 2;
    std::fwrite(out.data(), 8, kGmOutLen, f);
    std::fwrite(x.data(), 8, L, f);
    std::fclose(f);
    return 0;
}
