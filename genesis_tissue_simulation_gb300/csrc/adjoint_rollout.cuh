// Device helpers shared by the rollout kernels (whole-GPU, one CTA, bricks).
#pragma once
#include "adjoint_kernels.h"

namespace gbt {

__device__ __forceinline__ FrameCoeffs frameCoeffs(const DiffCoeffs& dc) {
    FrameCoeffs fc{};
    fc.alphaTilde = dc.alphaTilde; fc.betaGammaHS = dc.betaGammaHS; fc.omega = dc.omega;
    fc.dampingOverH = dc.dampingOverH; fc.fallback = 0; fc.fallbackInvEh2 = 0.f;
    fc.invScale = 1.f / (1.f + fc.dampingOverH); fc.invBulkScale = fc.invScale;
    return fc;
}

// Capsule of global substep g: frame f lerps command f -> f + 1 at t = (s + 1) / N.
__device__ __forceinline__ Capsule capsuleAt(const DiffBuffers& b, const DiffCoeffs& dc, int g, int N) {
    int f = g / N, s = g - f * N;
    float t = fminf(1.f, (float)(s + 1) / (float)N);
    const float* a = b.path + 6 * f;
    const float* c = b.path + 6 * (f + 1);
    Capsule k;
    k.sa = lerpTool(a[0], a[1], a[2], c[0], c[1], c[2], t);
    k.sb = lerpTool(a[3], a[4], a[5], c[3], c[4], c[5], t);
    k.radius = b.radius;
    k.alpha = dc.contactAlphaH2;
    return k;
}

__device__ __forceinline__ float4 f4(f3 v, float w) { return make_float4(v.x, v.y, v.z, w); }

// Sum of six floats over the block, deterministic (fixed lanes and warps); thread 0 gets it.
__device__ __forceinline__ void blockSum6(float v[6], float* out) {
    __shared__ float part[32][6];
#pragma unroll
    for (int c = 0; c < 6; c++)
        for (int o = 16; o > 0; o >>= 1) v[c] += __shfl_down_sync(0xffffffffu, v[c], o);
    int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (lane == 0)
        for (int c = 0; c < 6; c++) part[warp][c] = v[c];
    __syncthreads();
    if (threadIdx.x == 0) {
        int warps = (blockDim.x + 31) >> 5;
        for (int c = 0; c < 6; c++) {
            float s = 0.f;
            for (int w = 0; w < warps; w++) s += part[w][c];
            out[c] = s;
        }
    }
    __syncthreads();
}

}  // namespace gbt
