// nn_kernels.cuh -- kernels of the learned preconditioner's network besides
// the tensor-core convolution (conv_tc.cuh): pooling / upsampling / skip
// concatenation, their backward passes, weight gradients, the loss and Adam.
//
// Activations are NDHWC BF16 with channel counts that are multiples of 16;
// a voxel's channels are one contiguous 16-byte-aligned run.
#pragma once
#include <cuda_bf16.h>
#include <cstdint>

namespace pic {
namespace nn {

using bf16 = __nv_bfloat16;

struct Dims {
    int N, D, H, W;
    __host__ __device__ long long vox() const { return (long long)N * D * H * W; }
};

// Weight gradients dW[tap][co][ci] += sum_v gy[v][co] x[v + off(tap)][ci] and
// db[co] += sum_v gy[v][co] on the tensor cores: per tap a COUT x CC product
// with the voxels as the inner dimension.
//
// A CTA takes output bricks of 2 x 4 x 16 voxels (d, h, w): the brick of gy
// and, with its halo, of CC channels of x arrive in shared memory by cp.async,
// the next brick's while this one is multiplied.  Warp (kd, kh) keeps the
// three taps kw of its row in FP32 accumulators over all the CTA's bricks: a
// tap is only another row of the staged x, so x is read from memory once for
// 27 taps, and an A fragment (16 voxels of gy) serves three taps.  mma.sync
// m16n8k16 (BF16 in, FP32 accumulator): tcgen05.mma takes at least 64 rows of
// A, four times the 16 output channels of the layers that cost most, and its
// operands would have to be transposed copies of these; both fragments come
// from the voxel-major rows by ldmatrix.trans here.  Rows are padded by 16
// bytes, so that eight of them lie in distinct banks.  Each CTA adds its sums
// to dW once, at its end.
// The FP32 kernel this replaces converted 128-voxel chunks of x for every tap
// and multiplied them on CUDA cores, adding every chunk's sums with atomics;
// times of both at the launcher (nn.cu).
constexpr int kWgD = 2, kWgH = 4, kWgW = 16;                              // output brick
constexpr int kWgXv = (kWgD + 2) * (kWgH + 2) * (kWgW + 2);               // its x with halo
constexpr int kWgGv = kWgD * kWgH * kWgW;
constexpr int kWgThreads = 9 * 32;
__host__ __device__ constexpr int wg_row(int c) { return 2 * c + 16; }    // bytes of a padded row of c channels
__host__ __device__ constexpr int wg_stage(int cc, int co) { return kWgXv * wg_row(cc) + kWgGv * wg_row(co); }

__device__ __forceinline__ void wg_cp16(unsigned dst, const void* src, bool in) {
    const int n = in ? 16 : 0;   // 0: zeros
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(n) : "memory");
}
__device__ __forceinline__ void wg_ldsm(unsigned r[4], unsigned addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void wg_mma(float d[4], const unsigned a[4], unsigned b0, unsigned b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

template <int CIN, int COUT, int CC>
__global__ void __launch_bounds__(kWgThreads) k_wgrad(const bf16* __restrict__ x, const bf16* __restrict__ gy, Dims dm,
                                                      float* __restrict__ dW, float* __restrict__ db) {
    static_assert(CIN % CC == 0 && CC % 16 == 0 && COUT % 16 == 0, "channel counts");
    constexpr int XS = wg_row(CC), GS = wg_row(COUT), kStage = wg_stage(CC, COUT);
    extern __shared__ __align__(16) unsigned char wg_smem[];
    const unsigned base = (unsigned)__cvta_generic_to_shared(wg_smem);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int kd = warp / 3, kh = warp % 3;
    const int c0 = blockIdx.y * CC;   // first input channel
    const int bw = (dm.W + kWgW - 1) / kWgW, bh = (dm.H + kWgH - 1) / kWgH, bd = (dm.D + kWgD - 1) / kWgD;
    const int bricks = dm.N * bd * bh * bw;
    auto load = [&](int brick, int buf) {
        const int w0 = brick % bw * kWgW, h0 = brick / bw % bh * kWgH, d0 = brick / (bw * bh) % bd * kWgD;
        const long long n = brick / (bw * bh * bd);
        const unsigned sx = base + buf * kStage, sg = sx + kWgXv * XS;
        for (int e = threadIdx.x; e < kWgXv * (CC / 8); e += kWgThreads) {
            const int p = e % (CC / 8), v = e / (CC / 8);
            const int w = w0 + v % (kWgW + 2) - 1, h = h0 + v / (kWgW + 2) % (kWgH + 2) - 1,
                      d = d0 + v / ((kWgW + 2) * (kWgH + 2)) - 1;
            const bool in = w >= 0 && w < dm.W && h >= 0 && h < dm.H && d >= 0 && d < dm.D;
            const long long vox = in ? ((n * dm.D + d) * dm.H + h) * dm.W + w : 0;
            wg_cp16(sx + v * XS + p * 16, x + vox * CIN + c0 + p * 8, in);
        }
        for (int e = threadIdx.x; e < kWgGv * (COUT / 8); e += kWgThreads) {
            const int p = e % (COUT / 8), v = e / (COUT / 8);
            const int w = w0 + v % kWgW, h = h0 + v / kWgW % kWgH, d = d0 + v / (kWgW * kWgH);
            const bool in = w < dm.W && h < dm.H && d < dm.D;
            const long long vox = in ? ((n * dm.D + d) * dm.H + h) * dm.W + w : 0;
            wg_cp16(sg + v * GS + p * 16, gy + vox * COUT + p * 8, in);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    float acc[3][COUT / 16][CC / 8][4] = {};
    float bias = 0.f;
    constexpr int kStrands = kWgThreads / COUT;   // threads per output channel of db
    const int bco = threadIdx.x % COUT, strand = threadIdx.x / COUT;
    // this lane's row and column in the four 8 x 8 matrices of a fragment load
    const int r8 = lane & 7, m8 = lane >> 3;
    const int ka = r8 + (m8 >> 1) * 8, ma = (m8 & 1) * 8;   // A: k, co
    const int kb = r8 + (m8 & 1) * 8, nb8 = (m8 >> 1) * 8;  // B: k, ci
    int buf = 0;
    if ((int)blockIdx.x < bricks) load(blockIdx.x, 0);
    for (int brick = blockIdx.x; brick < bricks; brick += gridDim.x, buf ^= 1) {
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        __syncthreads();   // this brick is there, and the other buffer's is used up
        if (brick + (int)gridDim.x < bricks) load(brick + gridDim.x, buf ^ 1);
        const unsigned sx = base + buf * kStage, sg = sx + kWgXv * XS;
#pragma unroll 1
        for (int s = 0; s < kWgD * kWgH; ++s) {
            unsigned a[COUT / 16][4];
#pragma unroll
            for (int m = 0; m < COUT / 16; ++m) wg_ldsm(a[m], sg + (s * kWgW + ka) * GS + (m * 16 + ma) * 2);
            const int row = ((s / kWgH + kd) * (kWgH + 2) + s % kWgH + kh) * (kWgW + 2);
#pragma unroll
            for (int kw = 0; kw < 3; ++kw)
#pragma unroll
                for (int q = 0; q < CC / 16; ++q) {
                    unsigned b[4];
                    wg_ldsm(b, sx + (row + kw + kb) * XS + (q * 16 + nb8) * 2);
#pragma unroll
                    for (int m = 0; m < COUT / 16; ++m) {
                        wg_mma(acc[kw][m][2 * q], a[m], b[0], b[1]);
                        wg_mma(acc[kw][m][2 * q + 1], a[m], b[2], b[3]);
                    }
                }
        }
        if (blockIdx.y == 0 && strand < kStrands) {
            const unsigned char* g = wg_smem + buf * kStage + kWgXv * XS + bco * 2;
            for (int v = strand; v < kWgGv; v += kStrands)
                bias += __bfloat162float(*reinterpret_cast<const bf16*>(g + v * GS));
        }
    }
    if ((int)blockIdx.x >= bricks) return;
    const int gq = lane >> 2, t = lane & 3;
#pragma unroll
    for (int kw = 0; kw < 3; ++kw)
#pragma unroll
        for (int m = 0; m < COUT / 16; ++m)
#pragma unroll
            for (int q = 0; q < CC / 8; ++q)
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const int co = m * 16 + gq + (i >> 1) * 8, ci = c0 + q * 8 + 2 * t + (i & 1);
                    atomicAdd(&dW[((size_t)(warp * 3 + kw) * COUT + co) * CIN + ci], acc[kw][m][q][i]);
                }
    if (blockIdx.y == 0 && strand < kStrands) atomicAdd(&db[bco], bias);
}

// 2x2x2 average pooling (NDHWC, C channels), dims of the input.
__global__ void k_pool(const bf16* __restrict__ x, bf16* __restrict__ y, Dims di, int C) {
    // one thread per (coarse voxel, 8-channel chunk): 16-byte loads and stores, 32-bit index math
    const int D2 = di.D / 2, H2 = di.H / 2, W2 = di.W / 2, C8 = C / 8;
    const int tot = di.N * D2 * H2 * W2 * C8;
    for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < tot; e += gridDim.x * blockDim.x) {
        const int c8 = e % C8, v = e / C8;
        const int w = v % W2, h = (v / W2) % H2, d = (v / (W2 * H2)) % D2, n = v / (W2 * H2 * D2);
        float s[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int q = 0; q < 8; ++q) {
            const int dd = 2 * d + (q >> 2), hh = 2 * h + ((q >> 1) & 1), ww = 2 * w + (q & 1);
            const uint4 u = *reinterpret_cast<const uint4*>(
                x + ((((long long)n * di.D + dd) * di.H + hh) * di.W + ww) * C + c8 * 8);
            const __nv_bfloat162* p2 = reinterpret_cast<const __nv_bfloat162*>(&u);
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const float2 f = __bfloat1622float2(p2[i]);
                s[2 * i] += f.x;
                s[2 * i + 1] += f.y;
            }
        }
        __align__(16) __nv_bfloat162 o[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) o[i] = __floats2bfloat162_rn(s[2 * i] * 0.125f, s[2 * i + 1] * 0.125f);
        *reinterpret_cast<uint4*>(y + (long long)v * C + c8 * 8) = *reinterpret_cast<const uint4*>(o);
    }
}

// y[v] = concat(lo[v / 2] (C1 channels, nearest upsampling), skip[v] (C2)),
// dims of the fine level.  One thread per (voxel, 8-channel chunk).
__global__ void k_up_concat(const bf16* __restrict__ lo, const bf16* __restrict__ skip, bf16* __restrict__ y, Dims df,
                            int C1, int C2) {
    const int C8 = (C1 + C2) / 8, L8 = C1 / 8;
    const int tot = (int)df.vox() * C8;
    for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < tot; e += gridDim.x * blockDim.x) {
        const int c8 = e % C8, v = e / C8;
        uint4 u;
        if (c8 >= L8) {
            u = *reinterpret_cast<const uint4*>(skip + (long long)v * C2 + (c8 - L8) * 8);
        } else {
            const int w = v % df.W, h = (v / df.W) % df.H, d = (v / (df.W * df.H)) % df.D, n = v / (df.W * df.H * df.D);
            const long long vl = (((long long)n * (df.D / 2) + d / 2) * (df.H / 2) + h / 2) * (df.W / 2) + w / 2;
            u = *reinterpret_cast<const uint4*>(lo + vl * C1 + c8 * 8);
        }
        *reinterpret_cast<uint4*>(y + (long long)e * 8) = u;
    }
}

// The next three move four channels per thread (channel counts are multiples of
// 16), with 32-bit indices: element by element their time was the 64-bit index
// divisions (4 x 16x64x64 voxels, per training pass: 42 -> 18, 45 -> 12 and
// 71 -> 49 us).  (Fewer than 2^31 quads: the FP32 gradients of one level then
// take less than 34 GB, and several such buffers have to fit.)
__device__ __forceinline__ float4 add4(float4 a, float4 b) { return make_float4(a.x + b.x, a.y + b.y, a.z + b.z, a.w + b.w); }

// Backward of k_up_concat: glo[vl] = sum of the 8 children's first C1
// channels; gskip[v] = the last C2 channels (FP32; dims of the fine level).
__global__ void k_up_concat_bwd(const float* __restrict__ gy, float* __restrict__ glo, float* __restrict__ gskip,
                                Dims df, int C1, int C2) {
    const unsigned C = (C1 + C2) / 4, L = C1 / 4, S = C2 / 4;   // quads
    const float4* y4 = reinterpret_cast<const float4*>(gy);
    const unsigned tot_skip = (unsigned)df.vox() * S, step = gridDim.x * blockDim.x;
    for (unsigned e = blockIdx.x * blockDim.x + threadIdx.x; e < tot_skip; e += step) {
        const unsigned v = e / S;
        reinterpret_cast<float4*>(gskip)[e] = y4[v * C + L + (e - v * S)];
    }
    const unsigned D2 = df.D / 2, H2 = df.H / 2, W2 = df.W / 2;
    const unsigned tot_lo = (unsigned)df.N * D2 * H2 * W2 * L;
    for (unsigned e = blockIdx.x * blockDim.x + threadIdx.x; e < tot_lo; e += step) {
        const unsigned v = e / L, c = e - v * L;
        const unsigned r = v / W2, w = v - r * W2, q = r / H2, h = r - q * H2, n = q / D2, d = q - n * D2;
        float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            const unsigned dd = 2 * d + (k >> 2), hh = 2 * h + ((k >> 1) & 1), ww = 2 * w + (k & 1);
            s = add4(s, y4[(((n * df.D + dd) * df.H + hh) * df.W + ww) * C + c]);
        }
        reinterpret_cast<float4*>(glo)[e] = s;
    }
}

// gfine[v] += gcoarse[v / 2] / 8 (backward of the average pooling; dims of
// the fine level).
__global__ void k_pool_bwd_add(const float* __restrict__ gc, float* __restrict__ gf, Dims df, int channels) {
    const unsigned C = channels / 4, tot = (unsigned)df.vox() * C, step = gridDim.x * blockDim.x;
    for (unsigned e = blockIdx.x * blockDim.x + threadIdx.x; e < tot; e += step) {
        const unsigned v = e / C, c = e - v * C;
        const unsigned r = v / df.W, w = v - r * df.W, q = r / df.H, h = r - q * df.H, n = q / df.D, d = q - n * df.D;
        const unsigned vl = ((n * (df.D / 2) + d / 2) * (df.H / 2) + h / 2) * (df.W / 2) + w / 2;
        const float4 g = reinterpret_cast<const float4*>(gc)[vl * C + c];
        float4 f = reinterpret_cast<float4*>(gf)[e];
        f.x += g.x * 0.125f; f.y += g.y * 0.125f; f.z += g.z * 0.125f; f.w += g.w * 0.125f;
        reinterpret_cast<float4*>(gf)[e] = f;
    }
}

// g16 = g32 * (y > 0) (ReLU backward) in BF16; y == nullptr: no mask.  n: quads.
__global__ void k_relu_bwd(const float* __restrict__ g32, const bf16* __restrict__ y, bf16* __restrict__ g16, unsigned n) {
    for (unsigned e = blockIdx.x * blockDim.x + threadIdx.x; e < n; e += gridDim.x * blockDim.x) {
        const float4 g = reinterpret_cast<const float4*>(g32)[e];
        float v[4] = {g.x, g.y, g.z, g.w};
        if (y) {
            __align__(8) bf16 m[4];
            *reinterpret_cast<uint2*>(m) = reinterpret_cast<const uint2*>(y)[e];
#pragma unroll
            for (int k = 0; k < 4; ++k)
                if (!(__bfloat162float(m[k]) > 0.f)) v[k] = 0.f;
        }
        __align__(8) bf16 o[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) o[k] = __float2bfloat16(v[k]);
        reinterpret_cast<uint2*>(g16)[e] = *reinterpret_cast<const uint2*>(o);
    }
}

// Weighted mean-squared loss over the first OC channels of out (C channels
// per voxel): g[v][c] = 2 w (out - t) / (OC V) for c < OC, else 0; w times
// the mean square added to *loss.
// One thread per voxel: the FP64 squares of three channels in every lane,
// where a thread per element left 13 of 16 lanes of the slow FP64 pipe idle
// (42 -> 11 us at 262,144 voxels).  C a multiple of 4.
__global__ void k_mse(const float* __restrict__ out, const float* __restrict__ t, float* __restrict__ g, long long V,
                      int C, int OC, float w, double* __restrict__ loss) {
    double s = 0.0;
    const float sc = 2.f * w / (float)(OC * V);
    for (long long v = blockIdx.x * (long long)blockDim.x + threadIdx.x; v < V; v += (long long)gridDim.x * blockDim.x)
        for (int c = 0; c < C; c += 4) {
            float gv[4] = {0.f, 0.f, 0.f, 0.f};
            if (c < OC) {
                const float4 o4 = *reinterpret_cast<const float4*>(out + v * C + c);
                const float o[4] = {o4.x, o4.y, o4.z, o4.w};
#pragma unroll
                for (int i = 0; i < 4; ++i)
                    if (c + i < OC) {
                        const float d = o[i] - t[v * OC + c + i];
                        s += (double)d * d;
                        gv[i] = sc * d;
                    }
            }
            *reinterpret_cast<float4*>(g + v * C + c) = make_float4(gv[0], gv[1], gv[2], gv[3]);
        }
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if ((threadIdx.x & 31) == 0 && s != 0.0) atomicAdd(loss, (double)w * s / (double)(OC * V));
}

// Adam (Kingma & Ba 2015) with bias correction; c1 = lr / (1 - b1^t),
// c2 = 1 / (1 - b2^t).
__global__ void k_adam(float* __restrict__ p, const float* __restrict__ g, float* __restrict__ m, float* __restrict__ v,
                       long long n, float b1, float b2, float eps, float c1, float c2) {
    for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < n; e += (long long)gridDim.x * blockDim.x) {
        const float gv = g[e];
        const float mv = b1 * m[e] + (1.f - b1) * gv;
        const float vv = b2 * v[e] + (1.f - b2) * gv * gv;
        m[e] = mv;
        v[e] = vv;
        p[e] -= c1 * mv / (sqrtf(vv * c2) + eps);
    }
}

// BF16 copies of one layer's weights: forward Wk[tap][co][ci] and the
// flipped, transposed kernel of the input gradient Wt[26 - tap][ci][co].
__global__ void k_weights_bf16(const float* __restrict__ W, bf16* __restrict__ Wk, bf16* __restrict__ Wt, int cin,
                               int cout) {
    const int n = 27 * cin * cout;
    for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < n; e += gridDim.x * blockDim.x) {
        const int ci = e % cin, co = (e / cin) % cout, tap = e / (cin * cout);
        const bf16 b = __float2bfloat16(W[e]);
        Wk[e] = b;
        Wt[((size_t)(26 - tap) * cin + ci) * cout + co] = b;
    }
}

}  // namespace nn
}  // namespace pic
