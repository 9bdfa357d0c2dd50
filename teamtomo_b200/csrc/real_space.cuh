// Index shifts and the sinc^2 weight shared by the kernels around the
// transforms of project_3d_to_2d and backproject_2d_to_3d.
#pragma once
#include <cuda_runtime.h>

namespace tt {

// i mod n for i in (-n, 2n), the range every shift here produces.
__device__ __forceinline__ int wrap(int i, int n) { return i < 0 ? i + n : (i >= n ? i - n : i); }

// f32(k) * f32(1/n) for unshifted index k of an axis of length n.
__device__ __forceinline__ float fftfreq_at(int k, int n, float inv_n) {
    const int kk = (k < (n + 1) / 2) ? k : k - n;
    return __fmul_rn((float)kk, inv_n);
}

// Frequency at fftshifted position a of an axis of length n.
__device__ __forceinline__ float shifted_fftfreq(int a, int n, float inv_n) {
    return fftfreq_at(wrap(a - n / 2, n), n, inv_n);
}

// sinc(|f|)^2 from the squared frequency norm's two leading terms (f0^2 +
// f1^2, rounded as the reference sums them) and the third frequency, on the
// fftshifted norm grid (fftfreq_grid(rfft=False, fftshift=True, norm=True)).
__device__ __forceinline__ float sinc2_from(float f01, float f2) {
    const float r = __fsqrt_rn(__fadd_rn(f01, __fmul_rn(f2, f2)));
    if (r == 0.0f) return 1.0f;
    const float px = __fmul_rn(3.14159265358979323846f, r);
    const float s = __fdiv_rn(sinpif(r), px);
    return s * s;
}

}  // namespace tt
