// Generic 3D interpolation primitives of torch_image_interpolation
// (image_interpolation_3d.py:11-101 sample_image_3d, :104-275 insert_into_image_3d).
//
// sample: one thread per coordinate.  Trilinear follows grid_sample with
//   padding_mode='border', align_corners=True: the 8 corners of the clamped
//   coordinate, corners past the last index contribute nothing, and samples
//   whose coordinate is outside [0, n-1] on any axis are zero.  Nearest rounds
//   half to even (nearbyint).
// insert: one thread per value.  Coordinates are float32 (the reference casts
//   with .float()); points outside [0, n-1] on any axis are dropped; trilinear
//   splats with floor/ceil corners and float32 (1-t)/t weight products cast to
//   the weight dtype; nearest adds the value and a weight of 1 at rint(c).
// Element types: float32, float64, complex64, complex128 (dtype codes 0-3).
#include <cuda_runtime.h>

#include "capi_util.cuh"
#include "slice_ops.cuh"

namespace tt {

template <typename T>
__device__ __forceinline__ void atomic_add_real(T* p, T v) {
    atomicAdd(p, v);
}

// One sample of the (C, D, H, W) image at (cz, cy, cx) into o[0 .. C*E).
template <typename T, int E>
__device__ __forceinline__ void sample_point(const T* __restrict__ img, int64_t C, int D, int H, int W, T cz, T cy,
                                             T cx, T* __restrict__ o, int nearest) {
    const bool inside = cz >= (T)0 && cz <= (T)(D - 1) && cy >= (T)0 && cy <= (T)(H - 1) && cx >= (T)0 &&
                        cx <= (T)(W - 1);
    const int64_t plane = (int64_t)D * H * W;
    if (!inside) {
        for (int64_t k = 0; k < C * E; k++) o[k] = (T)0;
        return;
    }
    if (nearest) {
        const int z = (int)nearbyint((double)cz), y = (int)nearbyint((double)cy), x = (int)nearbyint((double)cx);
        const int64_t vi = ((int64_t)z * H + y) * W + x;
        for (int64_t ch = 0; ch < C; ch++)
#pragma unroll
            for (int e = 0; e < E; e++) o[ch * E + e] = img[(ch * plane + vi) * E + e];
        return;
    }
    const T fz = floor(cz), fy = floor(cy), fx = floor(cx);
    const int z0 = (int)fz, y0 = (int)fy, x0 = (int)fx;
    const T az[2] = {(fz + (T)1) - cz, cz - fz};
    const T ay[2] = {(fy + (T)1) - cy, cy - fy};
    const T ax[2] = {(fx + (T)1) - cx, cx - fx};
    for (int64_t ch = 0; ch < C; ch++) {
        T acc[E];
#pragma unroll
        for (int e = 0; e < E; e++) acc[e] = (T)0;
#pragma unroll
        for (int k = 0; k < 8; k++) {
            const int bz = (k >> 2) & 1, by = (k >> 1) & 1, bx = k & 1;
            const int z = z0 + bz, y = y0 + by, x = x0 + bx;
            if (z >= D || y >= H || x >= W) continue;
            const T wgt = ax[bx] * ay[by] * az[bz];
            const int64_t vi = ch * plane + ((int64_t)z * H + y) * W + x;
#pragma unroll
            for (int e = 0; e < E; e++) acc[e] += img[vi * E + e] * wgt;
        }
#pragma unroll
        for (int e = 0; e < E; e++) o[ch * E + e] = acc[e];
    }
}

template <typename T, int E>
__global__ void sample3d_kernel(const T* __restrict__ img, int64_t C, int D, int H, int W,
                                const T* __restrict__ coords, int64_t n, T* __restrict__ out, int nearest) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    sample_point<T, E>(img, C, D, H, W, coords[i * 3 + 0], coords[i * 3 + 1], coords[i * 3 + 2], out + i * C * E,
                       nearest);
}

// Backward of sample3d_kernel: d/dimage (ACCUMULATED, atomics) and
// d/dcoordinates (overwritten), PyTorch's complex-gradient convention.
// Trilinear: the same corners and weights; the coordinate gradient per axis is
// Re(conj(G) dS/dc) summed over the channels, zero where grid_sample's border
// clip stops it (a source index of exactly 0 or n-1 on that axis).  Nearest:
// the gradient goes to the sampled voxel; coordinates get none.
template <typename T>
__device__ __forceinline__ bool coord_grad_passes(T c, int n) {
    // grid_sample's round trip of the coordinate: c -> c / (0.5 n - 0.5) - 1 -> ((g + 1) / 2) (n - 1)
    const T half = (T)0.5 * (T)n - (T)0.5;
    const T raw = ((c / half - (T)1 + (T)1) * (T)0.5) * (T)(n - 1);
    return raw > (T)0 && raw < (T)(n - 1);
}

template <typename T, int E>
__global__ void sample3d_bwd_kernel(const T* __restrict__ img, int64_t C, int D, int H, int W,
                                    const T* __restrict__ coords, int64_t n, const T* __restrict__ grad,
                                    T* __restrict__ gimg, T* __restrict__ gcoord, int nearest) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const T cz = coords[i * 3 + 0], cy = coords[i * 3 + 1], cx = coords[i * 3 + 2];
    const T* gi = grad + i * C * E;
    T dz = (T)0, dy = (T)0, dx = (T)0;
    const bool inside = cz >= (T)0 && cz <= (T)(D - 1) && cy >= (T)0 && cy <= (T)(H - 1) && cx >= (T)0 &&
                        cx <= (T)(W - 1);
    const int64_t plane = (int64_t)D * H * W;
    if (inside && nearest) {
        if (gimg) {
            const int z = (int)nearbyint((double)cz), y = (int)nearbyint((double)cy), x = (int)nearbyint((double)cx);
            const int64_t vi = ((int64_t)z * H + y) * W + x;
            for (int64_t ch = 0; ch < C; ch++)
#pragma unroll
                for (int e = 0; e < E; e++) atomicAdd(gimg + (ch * plane + vi) * E + e, gi[ch * E + e]);
        }
    } else if (inside) {
        const T fz = floor(cz), fy = floor(cy), fx = floor(cx);
        const int z0 = (int)fz, y0 = (int)fy, x0 = (int)fx;
        const T az[2] = {(fz + (T)1) - cz, cz - fz};
        const T ay[2] = {(fy + (T)1) - cy, cy - fy};
        const T ax[2] = {(fx + (T)1) - cx, cx - fx};
        const T sgn[2] = {(T)-1, (T)1};
        for (int64_t ch = 0; ch < C; ch++) {
#pragma unroll
            for (int k = 0; k < 8; k++) {
                const int bz = (k >> 2) & 1, by = (k >> 1) & 1, bx = k & 1;
                const int z = z0 + bz, y = y0 + by, x = x0 + bx;
                if (z >= D || y >= H || x >= W) continue;
                const int64_t vi = ch * plane + ((int64_t)z * H + y) * W + x;
                if (gimg) {
                    const T wgt = ax[bx] * ay[by] * az[bz];
#pragma unroll
                    for (int e = 0; e < E; e++) atomicAdd(gimg + vi * E + e, gi[ch * E + e] * wgt);
                }
                if (gcoord) {
                    T gv = (T)0;  // Re(conj(G) v)
#pragma unroll
                    for (int e = 0; e < E; e++) gv += gi[ch * E + e] * img[vi * E + e];
                    dz += gv * sgn[bz] * ay[by] * ax[bx];
                    dy += gv * az[bz] * sgn[by] * ax[bx];
                    dx += gv * az[bz] * ay[by] * sgn[bx];
                }
            }
        }
        if (!coord_grad_passes(cz, D)) dz = (T)0;
        if (!coord_grad_passes(cy, H)) dy = (T)0;
        if (!coord_grad_passes(cx, W)) dx = (T)0;
    }
    if (gcoord) {
        gcoord[i * 3 + 0] = dz;
        gcoord[i * 3 + 1] = dy;
        gcoord[i * 3 + 2] = dx;
    }
}

// affine_transform_image_3d (torch_transform_image/transforms_3d.py:10-40):
// output voxel (z, y, x) of matrix m samples the image at M_m (z, y, x, 1),
// M in zyx order, computed in float32 with the reference's operation order
// (((m0 z + m1 y) + m2 x) + m3 1, each product rounded) so that nearest
// sampling picks the same voxels.  One thread per (matrix, output voxel).
template <typename T, int E>
__global__ void affine3d_kernel(const T* __restrict__ img, int64_t C, int D, int H, int W,
                                const float* __restrict__ mats, int64_t nm, int od, int oh, int ow,
                                T* __restrict__ out, int nearest) {
    const int64_t vox = (int64_t)od * oh * ow;
    const int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= nm * vox) return;
    const int64_t mi = idx / vox, r = idx - mi * vox;
    const float z = (float)(r / ((int64_t)oh * ow)), y = (float)((r / ow) % oh), x = (float)(r % ow);
    const float* M = mats + mi * 16;
    float c[3];
#pragma unroll
    for (int i = 0; i < 3; i++)
        c[i] = __fadd_rn(__fadd_rn(__fadd_rn(__fmul_rn(M[i * 4 + 0], z), __fmul_rn(M[i * 4 + 1], y)),
                                   __fmul_rn(M[i * 4 + 2], x)),
                         __fmul_rn(M[i * 4 + 3], 1.0f));
    sample_point<T, E>(img, C, D, H, W, (T)c[0], (T)c[1], (T)c[2], out + idx * C * E, nearest);
}

template <typename T, int E, typename WT>
__global__ void insert3d_kernel(const T* __restrict__ vals, const float* __restrict__ coords, int64_t n,
                                T* __restrict__ img, int64_t C, int D, int H, int W, WT* __restrict__ wts,
                                int nearest) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float cz = coords[i * 3 + 0], cy = coords[i * 3 + 1], cx = coords[i * 3 + 2];
    if (!(cz >= 0.0f && cz <= (float)D - 1.0f && cy >= 0.0f && cy <= (float)H - 1.0f && cx >= 0.0f &&
          cx <= (float)W - 1.0f))
        return;
    const int64_t plane = (int64_t)D * H * W;
    const T* v = vals + i * C * E;
    if (nearest) {
        const int64_t vi = ((int64_t)rintf(cz) * H + (int64_t)rintf(cy)) * W + (int64_t)rintf(cx);
        for (int64_t ch = 0; ch < C; ch++)
#pragma unroll
            for (int e = 0; e < E; e++) atomic_add_real(img + (ch * plane + vi) * E + e, v[ch * E + e]);
        atomic_add_real(wts + vi, (WT)1);
        return;
    }
    const float z0 = floorf(cz), y0 = floorf(cy), x0 = floorf(cx);
    const int iz[2] = {(int)z0, (int)ceilf(cz)}, iy[2] = {(int)y0, (int)ceilf(cy)}, ix[2] = {(int)x0, (int)ceilf(cx)};
    const float tz = cz - z0, ty = cy - y0, tx = cx - x0;
#pragma unroll
    for (int k = 0; k < 8; k++) {
        const int bz = (k >> 2) & 1, by = (k >> 1) & 1, bx = k & 1;
        const float w = ((bz ? tz : 1.0f - tz) * (by ? ty : 1.0f - ty)) * (bx ? tx : 1.0f - tx);
        if (w == 0.0f) continue;
        const int64_t vi = ((int64_t)iz[bz] * H + iy[by]) * W + ix[bx];
        const WT ww = (WT)w;
        const T wv = (T)ww;
        for (int64_t ch = 0; ch < C; ch++)
#pragma unroll
            for (int e = 0; e < E; e++) atomic_add_real(img + (ch * plane + vi) * E + e, v[ch * E + e] * wv);
        atomic_add_real(wts + vi, ww);
    }
}

// Backward of insert3d_kernel w.r.t. the values: each point gathers the
// upstream image gradient at the voxels it was added to, with the same float32
// weights (grad_values (n, channels) overwritten; zero for dropped points).
template <typename T, int E>
__global__ void insert3d_bwd_kernel(const T* __restrict__ gimg, const float* __restrict__ coords, int64_t n,
                                    int64_t C, int D, int H, int W, T* __restrict__ gvals, int nearest) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float cz = coords[i * 3 + 0], cy = coords[i * 3 + 1], cx = coords[i * 3 + 2];
    T* o = gvals + i * C * E;
    for (int64_t k = 0; k < C * E; k++) o[k] = (T)0;
    if (!(cz >= 0.0f && cz <= (float)D - 1.0f && cy >= 0.0f && cy <= (float)H - 1.0f && cx >= 0.0f &&
          cx <= (float)W - 1.0f))
        return;
    const int64_t plane = (int64_t)D * H * W;
    if (nearest) {
        const int64_t vi = ((int64_t)rintf(cz) * H + (int64_t)rintf(cy)) * W + (int64_t)rintf(cx);
        for (int64_t ch = 0; ch < C; ch++)
#pragma unroll
            for (int e = 0; e < E; e++) o[ch * E + e] = gimg[(ch * plane + vi) * E + e];
        return;
    }
    const float z0 = floorf(cz), y0 = floorf(cy), x0 = floorf(cx);
    const int iz[2] = {(int)z0, (int)ceilf(cz)}, iy[2] = {(int)y0, (int)ceilf(cy)}, ix[2] = {(int)x0, (int)ceilf(cx)};
    const float tz = cz - z0, ty = cy - y0, tx = cx - x0;
#pragma unroll
    for (int k = 0; k < 8; k++) {
        const int bz = (k >> 2) & 1, by = (k >> 1) & 1, bx = k & 1;
        const float w = ((bz ? tz : 1.0f - tz) * (by ? ty : 1.0f - ty)) * (bx ? tx : 1.0f - tx);
        if (w == 0.0f) continue;
        const int64_t vi = ((int64_t)iz[bz] * H + iy[by]) * W + ix[bx];
        for (int64_t ch = 0; ch < C; ch++)
#pragma unroll
            for (int e = 0; e < E; e++) o[ch * E + e] += gimg[(ch * plane + vi) * E + e] * (T)w;
    }
}

// Single-precision trilinear kernels.
//
// The generic kernels spend their time in scalar float atomics, one per corner
// and component, that each reach L2 as a request of their own, and in 64-bit
// index arithmetic per corner.  Here one voxel index and three strides (32-bit
// where the image allows it: IDX) address a cell, complex values travel as one
// 8-byte load or reduction, and the lanes 2j and 2j + 1 of a warp reduce the
// x-low and the x-high voxel of one point in the same instruction: adjacent
// voxels, so one L2 request serves both (the L2 takes 197 G requests/s whether
// one or two such lanes share them).
//
// Cell of an inside coordinate: low corner, fractions, strides to the high
// corners.  A high corner past the last index has fraction 0 and stride 0.
template <typename IDX>
struct Cell {
    IDX base, sz, sy, sx;
    float tz, ty, tx;
};

template <typename IDX>
__device__ __forceinline__ Cell<IDX> cell_of(float cz, float cy, float cx, int D, int H, int W) {
    const float fz = floorf(cz), fy = floorf(cy), fx = floorf(cx);
    const int z0 = (int)fz, y0 = (int)fy, x0 = (int)fx;
    Cell<IDX> k;
    k.base = ((IDX)z0 * H + y0) * W + x0;
    k.sz = z0 + 1 < D ? (IDX)H * W : 0;
    k.sy = y0 + 1 < H ? (IDX)W : 0;
    k.sx = x0 + 1 < W ? 1 : 0;
    k.tz = cz - fz;
    k.ty = cy - fy;
    k.tx = cx - fx;
    return k;
}

__device__ __forceinline__ bool inside3(float cz, float cy, float cx, int D, int H, int W) {
    return cz >= 0.0f && cz <= (float)(D - 1) && cy >= 0.0f && cy <= (float)(H - 1) && cx >= 0.0f &&
           cx <= (float)(W - 1);
}

template <int E>
struct Vec;
template <>
struct Vec<1> {
    using T = float;
};
template <>
struct Vec<2> {
    using T = float2;
};
__device__ __forceinline__ void vec_fma(float& a, float v, float w) { a = fmaf(v, w, a); }
__device__ __forceinline__ void vec_fma(float2& a, float2 v, float w) {
    a.x = fmaf(v.x, w, a.x);
    a.y = fmaf(v.y, w, a.y);
}
__device__ __forceinline__ float vec_mul(float v, float w) { return v * w; }
__device__ __forceinline__ float2 vec_mul(float2 v, float w) { return make_float2(v.x * w, v.y * w); }
__device__ __forceinline__ float vec_dot(float a, float b) { return a * b; }
__device__ __forceinline__ float vec_dot(float2 a, float2 b) { return fmaf(a.x, b.x, a.y * b.y); }
__device__ __forceinline__ float vec_shfl(float v, int src) { return __shfl_sync(0xffffffffu, v, src); }
__device__ __forceinline__ float2 vec_shfl(float2 v, int src) {
    return make_float2(vec_shfl(v.x, src), vec_shfl(v.y, src));
}

// Weights ((fraction or its complement) products) of corner k: bit 2 z, bit 1 y, bit 0 x.
template <typename IDX>
__device__ __forceinline__ IDX corner_offset(const Cell<IDX>& c, int k) {
    return ((k & 4) ? c.sz : 0) + ((k & 2) ? c.sy : 0) + ((k & 1) ? c.sx : 0);
}

template <int E, typename IDX>
__global__ void __launch_bounds__(256)
sample3d_f32_kernel(const typename Vec<E>::T* __restrict__ img, int C, int D, int H, int W,
                    const float* __restrict__ coords, int64_t n, typename Vec<E>::T* __restrict__ out) {
    using V = typename Vec<E>::T;
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float cz = __ldcs(coords + i * 3), cy = __ldcs(coords + i * 3 + 1), cx = __ldcs(coords + i * 3 + 2);
    V* o = out + i * C;
    if (!inside3(cz, cy, cx, D, H, W)) {
        for (int ch = 0; ch < C; ch++) o[ch] = V{};
        return;
    }
    const Cell<IDX> k = cell_of<IDX>(cz, cy, cx, D, H, W);
    const float z0 = 1.0f - k.tz, y0 = 1.0f - k.ty, x0 = 1.0f - k.tx;
    const IDX plane = (IDX)D * H * W;
    for (int ch = 0; ch < C; ch++) {
        const V* p = img + ch * plane + k.base;
        V v[8];
#pragma unroll
        for (int c = 0; c < 8; c++) v[c] = __ldg(p + corner_offset(k, c));
        V acc{};
#pragma unroll
        for (int c = 0; c < 8; c++) {
            // a corner past the end adds nothing, whatever the voxel its zero stride points at holds
            const bool there = (!(c & 4) || k.sz) && (!(c & 2) || k.sy) && (!(c & 1) || k.sx);
            const float w = (((c & 1) ? k.tx : x0) * ((c & 2) ? k.ty : y0)) * ((c & 4) ? k.tz : z0);
            if (there) vec_fma(acc, v[c], w);
        }
        o[ch] = acc;
    }
}

template <int E, typename IDX>
__global__ void __launch_bounds__(256)
sample3d_f32_bwd_kernel(const typename Vec<E>::T* __restrict__ img, int C, int D, int H, int W,
                        const float* __restrict__ coords, int64_t n, const typename Vec<E>::T* __restrict__ grad,
                        typename Vec<E>::T* __restrict__ gimg, float* __restrict__ gcoord) {
    using V = typename Vec<E>::T;
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const bool live = i < n;
    float cz = -1.0f, cy = 0.0f, cx = 0.0f;
    if (live) {
        cz = __ldcs(coords + i * 3);
        cy = __ldcs(coords + i * 3 + 1);
        cx = __ldcs(coords + i * 3 + 2);
    }
    const bool in = live && inside3(cz, cy, cx, D, H, W);
    if (!in) cz = -1.0f;  // no scatter
    const IDX plane = (IDX)D * H * W;
    if (gcoord) {
        float dz = 0.0f, dy = 0.0f, dx = 0.0f;
        if (in) {
            const Cell<IDX> k = cell_of<IDX>(cz, cy, cx, D, H, W);
            const float z0 = 1.0f - k.tz, y0 = 1.0f - k.ty, x0 = 1.0f - k.tx;
            for (int ch = 0; ch < C; ch++) {
                const V g = __ldg(grad + i * C + ch);
                const V* p = img + ch * plane + k.base;
                V v[8];
#pragma unroll
                for (int c = 0; c < 8; c++) v[c] = __ldg(p + corner_offset(k, c));
                float d[8];  // Re(conj(G) v), zero past the end
#pragma unroll
                for (int c = 0; c < 8; c++) {
                    const bool there = (!(c & 4) || k.sz) && (!(c & 2) || k.sy) && (!(c & 1) || k.sx);
                    d[c] = there ? vec_dot(g, v[c]) : 0.0f;
                }
#pragma unroll
                for (int b = 0; b < 4; b++) {  // the other two axes' corners
                    const int zy = (b & 2) * 2 + (b & 1) * 2, zx = (b & 2) * 2 + (b & 1), yx = b;
                    dx = fmaf(((b & 2) ? k.tz : z0) * ((b & 1) ? k.ty : y0), d[zy + 1] - d[zy], dx);
                    dy = fmaf(((b & 2) ? k.tz : z0) * ((b & 1) ? k.tx : x0), d[zx + 2] - d[zx], dy);
                    dz = fmaf(((b & 2) ? k.ty : y0) * ((b & 1) ? k.tx : x0), d[yx + 4] - d[yx], dz);
                }
            }
            if (!coord_grad_passes(cz, D)) dz = 0.0f;
            if (!coord_grad_passes(cy, H)) dy = 0.0f;
            if (!coord_grad_passes(cx, W)) dx = 0.0f;
        }
        if (live) {
            __stcs(gcoord + i * 3, dz);
            __stcs(gcoord + i * 3 + 1, dy);
            __stcs(gcoord + i * 3 + 2, dx);
        }
    }
    if (!gimg) return;  // the same in every lane
    const int lane = threadIdx.x & 31, bx = lane & 1;
#pragma unroll
    for (int half = 0; half < 2; half++) {
        const int src = (lane >> 1) + 16 * half;
        const float pz = vec_shfl(cz, src), py = vec_shfl(cy, src), px = vec_shfl(cx, src);
        const bool on = pz >= 0.0f;
        const Cell<IDX> k = cell_of<IDX>(pz, py, px, D, H, W);
        const float wx = bx ? k.tx : 1.0f - k.tx;
        for (int ch = 0; ch < C; ch++) {
            const V g0 = in ? __ldg(grad + i * C + ch) : V{};
            const V g = vec_shfl(g0, src);
            V* p = gimg + ch * plane + k.base + bx * k.sx;
#pragma unroll
            for (int r = 0; r < 4; r++) {
                const float w = (wx * ((r & 1) ? k.ty : 1.0f - k.ty)) * ((r & 2) ? k.tz : 1.0f - k.tz);
                const bool there = (!(r & 2) || k.sz) && (!(r & 1) || k.sy) && (!bx || k.sx);
                if (on && there) atomicAdd(p + (((r & 2) ? k.sz : 0) + ((r & 1) ? k.sy : 0)), vec_mul(g, w));
            }
        }
    }
}

template <int E, typename WT, typename IDX>
__global__ void __launch_bounds__(256)
insert3d_f32_kernel(const typename Vec<E>::T* __restrict__ vals, const float* __restrict__ coords, int64_t n,
                    typename Vec<E>::T* __restrict__ img, int C, int D, int H, int W, WT* __restrict__ wts) {
    using V = typename Vec<E>::T;
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    float cz = -1.0f, cy = 0.0f, cx = 0.0f;
    if (i < n) {
        cz = __ldcs(coords + i * 3);
        cy = __ldcs(coords + i * 3 + 1);
        cx = __ldcs(coords + i * 3 + 2);
    }
    const bool in = i < n && inside3(cz, cy, cx, D, H, W);
    if (!in) cz = -1.0f;
    const IDX plane = (IDX)D * H * W;
    const int lane = threadIdx.x & 31, bx = lane & 1;
#pragma unroll
    for (int half = 0; half < 2; half++) {
        const int src = (lane >> 1) + 16 * half;
        const float pz = vec_shfl(cz, src), py = vec_shfl(cy, src), px = vec_shfl(cx, src);
        const bool on = pz >= 0.0f;
        const Cell<IDX> k = cell_of<IDX>(pz, py, px, D, H, W);
        const IDX at = k.base + bx * k.sx;
        const float wx = bx ? k.tx : 1.0f - k.tx;
        float w[4];
        IDX o[4];
#pragma unroll
        for (int r = 0; r < 4; r++) {
            w[r] = (((r & 2) ? k.tz : 1.0f - k.tz) * ((r & 1) ? k.ty : 1.0f - k.ty)) * wx;
            o[r] = at + (((r & 2) ? k.sz : 0) + ((r & 1) ? k.sy : 0));
            if (on && w[r] != 0.0f) atomicAdd(wts + o[r], (WT)w[r]);
        }
        for (int ch = 0; ch < C; ch++) {
            const V v0 = in ? __ldg(vals + i * C + ch) : V{};
            const V v = vec_shfl(v0, src);
#pragma unroll
            for (int r = 0; r < 4; r++)
                if (on && w[r] != 0.0f) atomicAdd(img + ch * plane + o[r], vec_mul(v, (float)(WT)w[r]));
        }
    }
}

// The splat of many points through a bricked accumulator: one (re, im, weight,
// 0) float4 per corner by the slice insertion's lane octets
// (insert_point_octet: corners that neighbouring points share are added up
// before the reduction) instead of two reductions per corner into image and
// weights, then one pass that adds the accumulator to both.
template <int E>
__global__ void __launch_bounds__(256, 6)
splat_bricked_kernel(const typename Vec<E>::T* __restrict__ vals, const float* __restrict__ coords, int64_t n,
                     float4* __restrict__ acc, SliceGeom g) {
    __shared__ SplatTable tab[8];
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    float c[3] = {-1.0f, 0.0f, 0.0f}, re = 0.0f, im = 0.0f;
    if (i < n) {
        const float cz = __ldcs(coords + i * 3), cy = __ldcs(coords + i * 3 + 1), cx = __ldcs(coords + i * 3 + 2);
        if (inside3(cz, cy, cx, g.D, g.H, g.W)) {
            c[0] = cz;
            c[1] = cy;
            c[2] = cx;
            if constexpr (E == 2) {
                const float2 v = __ldcs(vals + i);
                re = v.x;
                im = v.y;
            } else {
                re = __ldcs(vals + i);
            }
        }
    }
    insert_point_octet(acc, g, re, im, 1.0f, c, tab[threadIdx.x >> 5], false);  // every lane takes part
}

// image += values, weights += weights of the bricked accumulator; one warp per
// brick row.
template <int E>
__global__ void __launch_bounds__(256)
splat_finish_kernel(const float4* __restrict__ acc, typename Vec<E>::T* __restrict__ img, float* __restrict__ wts,
                    SliceGeom g) {
    const int bh = (g.H + 1) >> 1, bw = (g.W + 1) >> 1;
    const int64_t rowi = (int64_t)blockIdx.x * 8 + (threadIdx.x >> 5);
    const int bz = (int)(rowi / bh), by = (int)(rowi - (int64_t)bz * bh);
    if (2 * bz >= g.D) return;
    const float4* row = acc + rowi * bw * 8;
    for (int t = threadIdx.x & 31; t < bw * 8; t += 32) {
        const int z = 2 * bz + ((t >> 2) & 1), y = 2 * by + ((t >> 1) & 1), x = 2 * (t >> 3) + (t & 1);
        if (z >= g.D || y >= g.H || x >= g.W) continue;
        const float4 a = __ldcs(row + t);
        if (a.x == 0.0f && a.y == 0.0f && a.z == 0.0f) continue;
        const int64_t o = ((int64_t)z * g.H + y) * g.W + x;
        if constexpr (E == 2) {
            const float2 v = img[o];
            img[o] = make_float2(v.x + a.x, v.y + a.y);
        } else {
            img[o] += a.x;
        }
        wts[o] += a.z;
    }
}

inline unsigned nblocks(int64_t n, int t) { return (unsigned)((n + t - 1) / t); }

// The single-precision trilinear kernels take up to 4096 channels; 8-byte
// aligned complex images, as torch allocates them.
inline bool f32_path(int32_t dtype, int32_t nearest, int64_t channels, const void* a, const void* b, const void* c) {
    const uintptr_t mask = dtype == 2 ? 7 : 3;
    return (dtype == 0 || dtype == 2) && !nearest && channels <= 4096 &&
           (((uintptr_t)a | (uintptr_t)b | (uintptr_t)c) & mask) == 0;
}

// Bytes of the bricked accumulator, or 0 where the direct splat is used: the
// accumulator's zeroing and the last pass cost about 12 ps a voxel, the splat
// 22 ps a point against 39 (measured at 192^3 / 2, 9.3 M points: 256 against 361
// us), so from one point per voxel.
inline size_t splat_bytes(int32_t dtype, int64_t n, int64_t channels, int64_t d, int64_t h, int64_t w,
                          int32_t weights_f64, int32_t nearest) {
    if ((dtype != 0 && dtype != 2) || nearest || weights_f64 || channels != 1 || d < 1 || h < 1 || w < 1) return 0;
    if (d > (1 << 20) || h > (1 << 20) || w > (1 << 20)) return 0;
    const int64_t slots = ((d + 1) / 2) * ((h + 1) / 2) * ((w + 1) / 2) * 8;
    return n >= 200000 && n >= d * h * w && slots < (1LL << 31) ? (size_t)slots * sizeof(float4) : 0;
}
inline bool idx32(int64_t channels, int64_t d, int64_t h, int64_t w) { return channels * d * h * w < (1LL << 31); }

}  // namespace tt

using namespace tt;

extern "C" int tt_sample_image_3d(const void* image, int32_t dtype, int64_t channels, int64_t d, int64_t h,
                                  int64_t w, const void* coordinates, int64_t n, void* out, int32_t nearest,
                                  void* stream) {
    if (n == 0) return TT_OK;
    if (!image || !coordinates || !out || channels < 1 || d < 1 || h < 1 || w < 1 || n < 0)
        return fail(TT_ERR_INVALID, "sample_image_3d: bad arguments");
    cudaStream_t st = as_stream(stream);
    const unsigned b = nblocks(n, 256);
    if (f32_path(dtype, nearest, channels, image, out, nullptr)) {
#define TT_SAMPLE(E, V, IDX)                                                                                       \
    sample3d_f32_kernel<E, IDX><<<b, 256, 0, st>>>((const V*)image, (int)channels, (int)d, (int)h, (int)w,        \
                                                   (const float*)coordinates, n, (V*)out)
        const bool small = idx32(channels, d, h, w);
        if (dtype == 0 && small) TT_SAMPLE(1, float, int32_t);
        else if (dtype == 0) TT_SAMPLE(1, float, int64_t);
        else if (small) TT_SAMPLE(2, float2, int32_t);
        else TT_SAMPLE(2, float2, int64_t);
#undef TT_SAMPLE
        return check_launch("sample3d_f32_kernel");
    }
    switch (dtype) {
        case 0:
            sample3d_kernel<float, 1><<<b, 256, 0, st>>>((const float*)image, channels, (int)d, (int)h, (int)w,
                                                          (const float*)coordinates, n, (float*)out, nearest);
            break;
        case 1:
            sample3d_kernel<double, 1><<<b, 256, 0, st>>>((const double*)image, channels, (int)d, (int)h, (int)w,
                                                           (const double*)coordinates, n, (double*)out, nearest);
            break;
        case 2:
            sample3d_kernel<float, 2><<<b, 256, 0, st>>>((const float*)image, channels, (int)d, (int)h, (int)w,
                                                          (const float*)coordinates, n, (float*)out, nearest);
            break;
        case 3:
            sample3d_kernel<double, 2><<<b, 256, 0, st>>>((const double*)image, channels, (int)d, (int)h, (int)w,
                                                           (const double*)coordinates, n, (double*)out, nearest);
            break;
        default:
            return fail(TT_ERR_INVALID, "sample_image_3d: unknown dtype code %d", dtype);
    }
    return check_launch("sample3d_kernel");
}

extern "C" int tt_insert_into_image_3d(const void* values, int32_t dtype, const float* coordinates, int64_t n,
                                       void* image, int64_t channels, int64_t d, int64_t h, int64_t w,
                                       void* weights, int32_t weights_f64, int32_t nearest, void* stream) {
    if (n == 0) return TT_OK;
    if (!values || !coordinates || !image || !weights || channels < 1 || d < 1 || h < 1 || w < 1 || n < 0)
        return fail(TT_ERR_INVALID, "insert_into_image_3d: bad arguments");
    cudaStream_t st = as_stream(stream);
    const unsigned b = nblocks(n, 256);
    if (f32_path(dtype, nearest, channels, values, image, nullptr)) {
#define TT_INSERT(E, V, WT, IDX)                                                                                  \
    insert3d_f32_kernel<E, WT, IDX><<<b, 256, 0, st>>>((const V*)values, coordinates, n, (V*)image, (int)channels, \
                                                       (int)d, (int)h, (int)w, (WT*)weights)
#define TT_INSERT_W(E, V)                                       \
    if (idx32(channels, d, h, w)) {                             \
        if (weights_f64) TT_INSERT(E, V, double, int32_t);      \
        else TT_INSERT(E, V, float, int32_t);                   \
    } else if (weights_f64) {                                   \
        TT_INSERT(E, V, double, int64_t);                       \
    } else {                                                    \
        TT_INSERT(E, V, float, int64_t);                        \
    }
        if (dtype == 0) {
            TT_INSERT_W(1, float)
        } else {
            TT_INSERT_W(2, float2)
        }
#undef TT_INSERT_W
#undef TT_INSERT
        return check_launch("insert3d_f32_kernel");
    }
#define TT_INSERT_CASE(T, E)                                                                                  \
    if (weights_f64)                                                                                          \
        insert3d_kernel<T, E, double><<<b, 256, 0, st>>>((const T*)values, coordinates, n, (T*)image, channels, \
                                                         (int)d, (int)h, (int)w, (double*)weights, nearest);  \
    else                                                                                                      \
        insert3d_kernel<T, E, float><<<b, 256, 0, st>>>((const T*)values, coordinates, n, (T*)image, channels,  \
                                                        (int)d, (int)h, (int)w, (float*)weights, nearest);
    switch (dtype) {
        case 0: TT_INSERT_CASE(float, 1) break;
        case 1: TT_INSERT_CASE(double, 1) break;
        case 2: TT_INSERT_CASE(float, 2) break;
        case 3: TT_INSERT_CASE(double, 2) break;
        default:
            return fail(TT_ERR_INVALID, "insert_into_image_3d: unknown dtype code %d", dtype);
    }
#undef TT_INSERT_CASE
    return check_launch("insert3d_kernel");
}

extern "C" size_t tt_insert_into_image_3d_workspace_bytes(int32_t dtype, int64_t n, int64_t channels, int64_t d,
                                                          int64_t h, int64_t w, int32_t weights_f64,
                                                          int32_t nearest) {
    return splat_bytes(dtype, n, channels, d, h, w, weights_f64, nearest);
}

extern "C" int tt_insert_into_image_3d_workspace(const void* values, int32_t dtype, const float* coordinates,
                                                 int64_t n, void* image, int64_t channels, int64_t d, int64_t h,
                                                 int64_t w, void* weights, int32_t weights_f64, int32_t nearest,
                                                 void* workspace, size_t workspace_bytes, void* stream) {
    const size_t need = splat_bytes(dtype, n, channels, d, h, w, weights_f64, nearest);
    if (!need || !f32_path(dtype, nearest, channels, values, image, nullptr))
        return tt_insert_into_image_3d(values, dtype, coordinates, n, image, channels, d, h, w, weights, weights_f64,
                                       nearest, stream);
    if (!values || !coordinates || !image || !weights)
        return fail(TT_ERR_INVALID, "insert_into_image_3d: bad arguments");
    if (!workspace || workspace_bytes < need)
        return fail(TT_ERR_WORKSPACE, "insert_into_image_3d: workspace of %zu bytes needed, got %zu", need,
                    workspace_bytes);
    if ((n + 255) / 256 > 0x7fffffffLL) return fail(TT_ERR_INVALID, "insert_into_image_3d: too many points");
    cudaStream_t st = as_stream(stream);
    cudaError_t e = cudaMemsetAsync(workspace, 0, need, st);
    if (e != cudaSuccess) return fail(TT_ERR_CUDA, "insert_into_image_3d: memset: %s", cudaGetErrorString(e));
    SliceGeom g{};  // the splat and its last pass read the image dims only
    g.D = (int)d;
    g.H = (int)h;
    g.W = (int)w;
    float4* acc = (float4*)workspace;
    const unsigned rows = nblocks(((d + 1) / 2) * ((h + 1) / 2), 8);
    if (dtype == 2) {
        splat_bricked_kernel<2><<<nblocks(n, 256), 256, 0, st>>>((const float2*)values, coordinates, n, acc, g);
        splat_finish_kernel<2><<<rows, 256, 0, st>>>(acc, (float2*)image, (float*)weights, g);
    } else {
        splat_bricked_kernel<1><<<nblocks(n, 256), 256, 0, st>>>((const float*)values, coordinates, n, acc, g);
        splat_finish_kernel<1><<<rows, 256, 0, st>>>(acc, (float*)image, (float*)weights, g);
    }
    return check_launch("splat_bricked_kernel");
}

extern "C" int tt_affine_transform_image_3d(const void* image, int32_t dtype, int64_t channels, int64_t d, int64_t h,
                                            int64_t w, const float* matrices_zyx, int64_t n_matrices, int64_t od,
                                            int64_t oh, int64_t ow, int32_t nearest, void* out, void* stream) {
    if (n_matrices == 0 || od * oh * ow == 0) return TT_OK;
    if (!image || !matrices_zyx || !out || channels < 1 || d < 1 || h < 1 || w < 1 || n_matrices < 0 || od < 0 ||
        oh < 0 || ow < 0)
        return fail(TT_ERR_INVALID, "affine_transform_image_3d: bad arguments");
    if (dtype < 0 || dtype > 3) return fail(TT_ERR_INVALID, "affine_transform_image_3d: dtype must be 0-3");
    const int64_t total = n_matrices * od * oh * ow;
    const unsigned b = nblocks(total, 256);
    cudaStream_t st = as_stream(stream);
    switch (dtype) {
        case 0:
            affine3d_kernel<float, 1><<<b, 256, 0, st>>>((const float*)image, channels, (int)d, (int)h, (int)w,
                                                         matrices_zyx, n_matrices, (int)od, (int)oh, (int)ow,
                                                         (float*)out, nearest);
            break;
        case 1:
            affine3d_kernel<double, 1><<<b, 256, 0, st>>>((const double*)image, channels, (int)d, (int)h, (int)w,
                                                          matrices_zyx, n_matrices, (int)od, (int)oh, (int)ow,
                                                          (double*)out, nearest);
            break;
        case 2:
            affine3d_kernel<float, 2><<<b, 256, 0, st>>>((const float*)image, channels, (int)d, (int)h, (int)w,
                                                         matrices_zyx, n_matrices, (int)od, (int)oh, (int)ow,
                                                         (float*)out, nearest);
            break;
        default:
            affine3d_kernel<double, 2><<<b, 256, 0, st>>>((const double*)image, channels, (int)d, (int)h, (int)w,
                                                          matrices_zyx, n_matrices, (int)od, (int)oh, (int)ow,
                                                          (double*)out, nearest);
    }
    return check_launch("affine3d_kernel");
}

extern "C" int tt_sample_image_3d_backward(const void* image, int32_t dtype, int64_t channels, int64_t d, int64_t h,
                                           int64_t w, const void* coordinates, int64_t n, const void* grad_out,
                                           void* grad_image, void* grad_coordinates, int32_t nearest, void* stream) {
    if (n == 0) return TT_OK;
    if (!image || !coordinates || !grad_out || channels < 1 || d < 1 || h < 1 || w < 1 || n < 0)
        return fail(TT_ERR_INVALID, "sample_image_3d backward: bad arguments");
    if (dtype < 0 || dtype > 3) return fail(TT_ERR_INVALID, "sample_image_3d backward: dtype must be 0-3");
    if (!grad_image && !grad_coordinates) return TT_OK;
    const unsigned b = nblocks(n, 256);
    cudaStream_t st = as_stream(stream);
    if (f32_path(dtype, nearest, channels, image, grad_out, grad_image)) {
#define TT_SAMPLE_BWD(E, V, IDX)                                                                                    \
    sample3d_f32_bwd_kernel<E, IDX><<<b, 256, 0, st>>>((const V*)image, (int)channels, (int)d, (int)h, (int)w,     \
                                                       (const float*)coordinates, n, (const V*)grad_out,           \
                                                       (V*)grad_image, (float*)grad_coordinates)
        const bool small = idx32(channels, d, h, w);
        if (dtype == 0 && small) TT_SAMPLE_BWD(1, float, int32_t);
        else if (dtype == 0) TT_SAMPLE_BWD(1, float, int64_t);
        else if (small) TT_SAMPLE_BWD(2, float2, int32_t);
        else TT_SAMPLE_BWD(2, float2, int64_t);
#undef TT_SAMPLE_BWD
        return check_launch("sample3d_f32_bwd_kernel");
    }
    switch (dtype) {
        case 0:
            sample3d_bwd_kernel<float, 1><<<b, 256, 0, st>>>((const float*)image, channels, (int)d, (int)h, (int)w,
                                                             (const float*)coordinates, n, (const float*)grad_out,
                                                             (float*)grad_image, (float*)grad_coordinates, nearest);
            break;
        case 1:
            sample3d_bwd_kernel<double, 1><<<b, 256, 0, st>>>((const double*)image, channels, (int)d, (int)h,
                                                              (int)w, (const double*)coordinates, n,
                                                              (const double*)grad_out, (double*)grad_image,
                                                              (double*)grad_coordinates, nearest);
            break;
        case 2:
            sample3d_bwd_kernel<float, 2><<<b, 256, 0, st>>>((const float*)image, channels, (int)d, (int)h, (int)w,
                                                             (const float*)coordinates, n, (const float*)grad_out,
                                                             (float*)grad_image, (float*)grad_coordinates, nearest);
            break;
        default:
            sample3d_bwd_kernel<double, 2><<<b, 256, 0, st>>>((const double*)image, channels, (int)d, (int)h,
                                                              (int)w, (const double*)coordinates, n,
                                                              (const double*)grad_out, (double*)grad_image,
                                                              (double*)grad_coordinates, nearest);
    }
    return check_launch("sample3d_bwd_kernel");
}

extern "C" int tt_insert_into_image_3d_backward(const void* grad_image, int32_t dtype, const float* coordinates,
                                                int64_t n, int64_t channels, int64_t d, int64_t h, int64_t w,
                                                int32_t nearest, void* grad_values, void* stream) {
    if (n == 0) return TT_OK;
    if (!grad_image || !coordinates || !grad_values || channels < 1 || d < 1 || h < 1 || w < 1 || n < 0)
        return fail(TT_ERR_INVALID, "insert_into_image_3d backward: bad arguments");
    if (dtype < 0 || dtype > 3) return fail(TT_ERR_INVALID, "insert_into_image_3d backward: dtype must be 0-3");
    const unsigned b = nblocks(n, 256);
    cudaStream_t st = as_stream(stream);
    switch (dtype) {
        case 0:
            insert3d_bwd_kernel<float, 1><<<b, 256, 0, st>>>((const float*)grad_image, coordinates, n, channels,
                                                             (int)d, (int)h, (int)w, (float*)grad_values, nearest);
            break;
        case 1:
            insert3d_bwd_kernel<double, 1><<<b, 256, 0, st>>>((const double*)grad_image, coordinates, n, channels,
                                                              (int)d, (int)h, (int)w, (double*)grad_values, nearest);
            break;
        case 2:
            insert3d_bwd_kernel<float, 2><<<b, 256, 0, st>>>((const float*)grad_image, coordinates, n, channels,
                                                             (int)d, (int)h, (int)w, (float*)grad_values, nearest);
            break;
        default:
            insert3d_bwd_kernel<double, 2><<<b, 256, 0, st>>>((const double*)grad_image, coordinates, n, channels,
                                                              (int)d, (int)h, (int)w, (double*)grad_values, nearest);
    }
    return check_launch("insert3d_bwd_kernel");
}
