// host_cuda.hpp -- what a kernel of one warp-synchronous CTA after another needs to
// compile and run on host threads: indices, barriers of a CTA and of a warp,
// shuffles, atomics, and a CTA that can be held up (late_cta, late_at).
#pragma once
#include <cuda_runtime.h>
#undef __launch_bounds__
#define __launch_bounds__(...)

#include <atomic>
#include <barrier>
#include <chrono>
#include <cmath>
#include <cstring>
#include <memory>
#include <thread>
#include <vector>

struct Index { int x = 0, y = 0, z = 0; };
static thread_local Index threadIdx, blockIdx;
static Index blockDim, gridDim;

struct Cta {
    std::barrier<> all;
    std::vector<std::unique_ptr<std::barrier<>>> warp;
    std::vector<double> lanes, smem;
    bool flag = false;
    int fences = 0;   // two per barrier of the grid, by the CTA's first thread
    Cta(int threads, size_t bytes) : all(threads), lanes(threads), smem(bytes / sizeof(double) + 1) {
        for (int w = 0; w < threads / 32; ++w) warp.push_back(std::make_unique<std::barrier<>>(32));
    }
};
static thread_local Cta* here = nullptr;
static thread_local bool held = false;
static int late_cta = -1, late_at = 0, late_ms = 150;

static double* host_smem() { return here->smem.data(); }
static bool& host_flag() { return here->flag; }
static unsigned host_acquire(unsigned* p) {
    std::this_thread::yield();
    return __atomic_load_n(p, __ATOMIC_ACQUIRE);
}
static void __syncthreads() { here->all.arrive_and_wait(); }
static void __syncwarp() { here->warp[threadIdx.x / 32]->arrive_and_wait(); }
static double __shfl_xor_sync(unsigned, double v, int o) {
    here->lanes[threadIdx.x] = v;
    __syncwarp();
    const double r = here->lanes[threadIdx.x ^ o];
    __syncwarp();
    return r;
}
static void __threadfence() {
    std::atomic_thread_fence(std::memory_order_seq_cst);
    ++here->fences;
}
static unsigned atomicAdd(unsigned* p, unsigned v) { return __atomic_fetch_add(p, v, __ATOMIC_ACQ_REL); }
static int __double2hiint(double v) {
    long long b;
    std::memcpy(&b, &v, 8);
    return (int)(b >> 32);
}
static double __ldcg(const double* p) {
    if (blockIdx.x == late_cta && here->fences == 2 * late_at && !held) {
        held = true;
        std::this_thread::sleep_for(std::chrono::milliseconds(late_ms));
    }
    return *p;
}
// not reached by the kernel, named in the headers it includes
static unsigned __umulhi(unsigned a, unsigned b) { return (unsigned)(((unsigned long long)a * b) >> 32); }
static float __fmaf_rn(float a, float b, float c) { return std::fmaf(a, b, c); }
static float __fmul_rn(float a, float b) { return a * b; }
static float __fsub_rn(float a, float b) { return a - b; }
static size_t __cvta_generic_to_shared(const void* p) { return (size_t)p; }
using std::fabs;
using std::fma;
using std::fmax;
using std::sqrt;
