// gmres_launch.cuh -- launch of the one-launch GMRES solve (gmres_grid.cuh).
#pragma once
#include <algorithm>
#include "gmres_grid.cuh"

namespace pic {

template <int NW, int KB, bool kNode, bool kRef>
static cudaError_t gmres_grid(cudaStream_t s, const GmresArgs& a) {
    const size_t smem = gmres_smem(a.cols, NW, kRef);
    // the attribute belongs to the function, not to the caller's context: always
    // the most that any solve takes, so that a solve of another thread, between
    // this and the launch, sets the same
    cudaError_t e = cudaFuncSetAttribute((const void*)k_gmres_grid<NW, KB, kNode, kRef>,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)gmres_smem(kGmresMaxCols, NW, kRef));
    if (e != cudaSuccess) return e;
    // as many CTAs as run at once on the SMs that this process sees, at most one
    // per SM of a whole GB300 (what the partial sums have room for)
    int device = 0, sms = 0, per_sm = 0;
    if ((e = cudaGetDevice(&device)) != cudaSuccess ||
        (e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device)) != cudaSuccess ||
        (e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, (const void*)k_gmres_grid<NW, KB, kNode, kRef>, NW + 32,
                                                           smem)) != cudaSuccess)
        return e;
    const long long most = std::min<long long>(kNumSM, (long long)sms * per_sm);
    if (most < 1) return cudaErrorCooperativeLaunchTooLarge;
    const int grid = (int)std::min<long long>(most, ((kNode ? 1 : 3) * a.g.N + NW - 1) / NW);
    void* args[] = {(void*)&a};
    return cudaLaunchCooperativeKernel((const void*)k_gmres_grid<NW, KB, kNode, kRef>, grid, NW + 32, args, smem, s);
}

// Workers per CTA by the box: few, each with one element, while the barriers'
// and reductions' latency is the time; many, each with whole nodes, once the
// FP64 work is (more warps hide the loads of the basis).  Restarted GMRES(30)
// to 1e-8, us per solve (16 iterations), the kernel-per-operation form first:
//   32x32x1      26x20x18     64x64x32     128x128x32    256x256x64
//   (1,750)      2,120        3,942        6,694         30,000
//   128: 261     256: 384     480: 1,063   736: 3,075    992: 19,498
// and the neighbours of each choice:
//   256: 306     128: 435     736: 1,506   480: 3,292    736: 19,857
// (128x64x32: 480 1,754, 736 2,007; 128x128x64: 736 5,720, 992 5,429.)
// The reference method to its own stop (20 to 31 columns; two dot products per
// vector, so half as many vectors per pass: with KB doubled every box takes 1% to
// 17% longer), us per solve:
//   32x32x1      32x32x24     64x64x32     128x128x32    256x256x64
//   128: 397     256: 881     480: 2,325   736: 7,574    992: 55,209
//   256: 443     128: 1,269   736: 3,321   480: 7,831    736: 58,282
// (16x16x16: 128 592, 256 617; 26x20x18: 256 682, 128 851; 40x40x40: 480 1,442, 256
// 1,540; 96x64x64: 480 6,053, 736 6,224; 128x128x48: 736 11,683, 480 10,781, 992
// 11,605; 128x128x64: 992 14,120, 736 15,356.)
cudaError_t launch_gmres_grid(cudaStream_t s, const GmresArgs& a) {
    cudaError_t e = cudaMemsetAsync(a.bar, 0, 2 * sizeof(unsigned), s);
    if (e != cudaSuccess) return e;
    const long long n = a.g.N;
    if (a.reference) {
        if (n <= 4096) return gmres_grid<128, 8, false, true>(s, a);
        if (n <= 24576) return gmres_grid<256, 8, false, true>(s, a);
        if (n <= 393216) return gmres_grid<480, 4, true, true>(s, a);
        if (n <= 786432) return gmres_grid<736, 4, true, true>(s, a);
        return gmres_grid<992, 4, true, true>(s, a);
    }
    if (n <= 4096) return gmres_grid<128, 16, false, false>(s, a);
    if (n <= 24576) return gmres_grid<256, 16, false, false>(s, a);
    if (n <= 393216) return gmres_grid<480, 8, true, false>(s, a);
    if (n <= 786432) return gmres_grid<736, 8, true, false>(s, a);
    return gmres_grid<992, 8, true, false>(s, a);
}

}  // namespace pic
