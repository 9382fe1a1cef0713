// gmres_launch_on_host.cpp -- the host side of the one-launch GMRES solve
// (csrc/gmres_launch.cuh, csrc/solver.cu) against a CUDA runtime of its own, which keeps
// memory on the host, checks launches as the real one does and runs no
// kernel.  gmres_grid_host.cuh: see gmres_on_host.cpp.
//
//   gmres_launch_on_host threads   two threads' solves, the second one's launch
//                                  between the first one's preparation and launch
//   gmres_launch_on_host device SMS COOPERATIVE   a solve of each plain method on a
//                                  device of SMS multiprocessors, which takes cooperative
//                                  launches or does not
//   gmres_launch_on_host runs-out  a solve one of whose barriers gave up, then another
// Prints the solves' statuses and, of a device, the grid of the last launch (0: none)
// and how many dot products were launched by themselves.
#include "host_cuda.hpp"

#include <cstdio>
#include <cstdlib>
#include <functional>
#include <future>
#include <map>
#include <mutex>
#include <string>

#include "gmres_grid_host.cuh"
#include "gmres_launch.cuh"
#include "solver.cu"

using namespace pic;

namespace {
std::mutex lock;
std::map<const void*, size_t> most_smem;          // opted-in dynamic shared memory
std::function<void()> after_attribute;            // called once, after an attribute is set
int last_grid = 0, dots = 0, multiprocessors = 152, cooperative = 1, runs_out = 0;
}  // namespace

extern "C" {
cudaError_t cudaFuncSetAttribute(const void* f, cudaFuncAttribute, int v) {
    std::function<void()> then;
    {
        std::lock_guard<std::mutex> l(lock);
        most_smem[f] = (size_t)v;
        std::swap(then, after_attribute);
    }
    if (then) then();
    return cudaSuccess;
}
cudaError_t cudaLaunchCooperativeKernel(const void* f, dim3 grid, dim3, void** args, size_t smem, cudaStream_t) {
    std::lock_guard<std::mutex> l(lock);
    if (smem > std::max<size_t>(48 * 1024, most_smem[f])) return cudaErrorInvalidValue;
    if (!cooperative) return cudaErrorNotSupported;
    if ((int)grid.x > multiprocessors) return cudaErrorCooperativeLaunchTooLarge;   // one CTA of these per SM
    last_grid = (int)grid.x;
    const GmresArgs& a = *static_cast<const GmresArgs*>(args[0]);
    if (runs_out) a.bar[1] = 1;
    else
        for (int i = 0; i < kGmOutLen; ++i) a.out[i] = 0;
    return cudaSuccess;
}
cudaError_t cudaGetDevice(int* d) { *d = 0; return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr what, int) {
    *v = what == cudaDevAttrMultiProcessorCount ? multiprocessors : 0;
    return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessor(int* n, const void*, int, size_t) { *n = 1; return cudaSuccess; }
cudaError_t cudaMalloc(void** p, size_t n) { *p = std::calloc(n, 1); return cudaSuccess; }
cudaError_t cudaFree(void* p) { std::free(p); return cudaSuccess; }
cudaError_t cudaMemsetAsync(void* p, int v, size_t n, cudaStream_t) { std::memset(p, v, n); return cudaSuccess; }
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t) { std::memcpy(d, s, n); return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
const char* cudaGetErrorString(cudaError_t) { return "error of the test's runtime"; }
cudaError_t cudaEventCreate(cudaEvent_t*) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t, cudaEvent_t) { *ms = 0; return cudaSuccess; }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
}

// The operations that a solve of a right part 0 takes by themselves.
namespace pic {
void launch_nonfinite(cudaStream_t, const double*, long long, int*) {}
void launch_dot(cudaStream_t, const double*, const double*, long long, double*, int, double* out, int) {
    ++dots;
    *out = 0;
}
}  // namespace pic

// A box, its system (right part 0) and a workspace of its own.
struct Caller {
    GridP g{};
    std::vector<double> mu, b, x, partials;
    int flag = 0;
    Krylov k{};
    std::string text;
    Caller(int nx, int ny, int nz) {
        g.nx = nx; g.ny = ny; g.nz = nz;
        g.N = (long long)nx * ny * nz;
        g.dx = g.dy = g.dz = g.dt = 1; g.theta = 0.5; g.cfix = 1;
        mu.resize(9 * g.N); b.resize(3 * g.N); x.resize(3 * g.N); partials.resize(8192);
    }
    int solve(int method, int restart) {
        SolveCtx c{nullptr, &g, mu.data(), partials.data(), &flag, &k, &text};
        pic_solve_opts o{};
        o.method = method; o.restart = restart; o.max_iter = 50; o.tol = 1e-8;
        pic_solve_info info{};
        const int st = krylov_solve(c, b.data(), x.data(), o, &info);
        krylov_free(k);
        return st;
    }
};

int main(int argc, char** argv) {
    const std::string what = argc > 1 ? argv[1] : "";
    if (what == "threads") {
        Caller one(20, 20, 20), two(20, 20, 20);
        std::future<int> second;
        after_attribute = [&] {
            second = std::async(std::launch::async, [&] { return two.solve(PIC_GMRES_RESTARTED, 30); });
            second.wait_for(std::chrono::milliseconds(500));
        };
        const int first = one.solve(PIC_GMRES_RESTARTED, 128);
        std::printf("%d %d\n", first, second.get());
        return 0;
    }
    if (what == "device" && argc == 4) {
        multiprocessors = std::atoi(argv[2]);
        cooperative = std::atoi(argv[3]);
        Caller one(20, 20, 20);
        const int a = one.solve(PIC_GMRES_REFERENCE, 0), b = one.solve(PIC_GMRES_RESTARTED, 30);
        std::printf("%d %d %d %d\n", a, b, last_grid, dots);
        return 0;
    }
    if (what == "runs-out") {
        Caller one(20, 20, 20);
        runs_out = 1;
        const int a = one.solve(PIC_GMRES_REFERENCE, 0);
        runs_out = 0;
        std::printf("%d %s\n%d\n", a, one.text.c_str(), one.solve(PIC_GMRES_REFERENCE, 0));
        return 0;
    }
    return 2;
}
