// The learned denoiser's 5x5 filter of one pixel: softmax over its 25 logits
// and the weighted sum of the noisy radiance around it. Used by the filter
// and loss kernels (kpcn.cu) and by the output convolution's epilogue
// (conv.cu).
#pragma once
#include "common.cuh"

namespace crt {

constexpr int kTaps5 = 25;

#ifdef __CUDACC__

__device__ __forceinline__ int clampi(int v, int lo, int hi) { return v < lo ? lo : (v > hi ? hi : v); }

// Softmax over l[0 .. 24], weights in w.
template <int kN>
__device__ __forceinline__ void softmax25(const float (&l)[kN], float (&w)[kTaps5]) {
    float mx = l[0];
#pragma unroll
    for (int k = 1; k < kTaps5; ++k) mx = fmaxf(mx, l[k]);
    float s = 0.f;
#pragma unroll
    for (int k = 0; k < kTaps5; ++k) {
        w[k] = expf(l[k] - mx);
        s += w[k];
    }
    const float inv = 1.f / s;
#pragma unroll
    for (int k = 0; k < kTaps5; ++k) w[k] *= inv;
}

// sum_k w_k * noisy[clamp(pixel + off5(k))] for pixel (x, y) of the h x w
// image at `img`.
__device__ __forceinline__ float4 filter25(const float (&wt)[kTaps5], const float4 *img, int x, int y, int h, int w) {
    float r = 0.f, g = 0.f, b = 0.f;
#pragma unroll
    for (int k = 0; k < kTaps5; ++k) {
        const int sy = clampi(y + k / 5 - 2, 0, h - 1), sx = clampi(x + k % 5 - 2, 0, w - 1);
        const float4 v = __ldg(img + (int64_t)sy * w + sx);
        r += wt[k] * v.x;
        g += wt[k] * v.y;
        b += wt[k] * v.z;
    }
    return make_float4(r, g, b, 0.f);
}

#endif  // __CUDACC__

}  // namespace crt
