// The transforms of project_3d_to_2d (torch_fourier_slice/project.py:48-92) and
// backproject_2d_to_3d (torch_fourier_slice/backproject.py:48-92), with their
// padding, shifts, weights, cropping and layouts in the kernels' loads and
// stores (the transform itself is in fft.cuh).
//
// Padded box e = d + 2 p, half spectrum wr = e/2 + 1, and L = 2 (wr - 1) the
// length of the inverse real transform (the reference runs irfftn without an
// output size, so L = e - 1 for odd e).
//
//   projection       volume (d, d, d) -> x transforms of its d^2 rows, weighted by
//                    sinc^2 -> y transforms of d planes -> z transforms, stored as
//                    the bricked copy the gathers read (tt_pack_volume_bricks)
//                    -> per slice and eight columns: central-slice samples into
//                    shared memory, their inverse y transforms, the d kept rows
//                    stored -> inverse x transforms, the kept columns stored
//   its adjoint      the same passes backwards around the extraction's backward
//   reconstruction   images (d, d) -> x transforms of d rows -> y transforms:
//                    fftshifted slices; after the insertion, the accumulator is
//                    completed (Friedel), divided by max(weights, 1) and
//                    transformed along z, y and x, keeping d planes, rows and
//                    columns, the last divided by sinc^2
//
// A library transform of the padded arrays moves the zeros and the cropped
// samples through HBM in every pass and needs separate passes for the padding,
// the scaling and the layouts.  Every kernel here is bound by HBM or L2 traffic
// at large sizes and by launch and barrier latency at small ones.
#include <cuda_runtime.h>

#include "capi_util.cuh"
#include "fft.cuh"
#include "real_space.cuh"
#include "slice_common.cuh"
#include "slice_ops.cuh"

namespace tt {

constexpr int kFftMaxThreads = 512;

// sinc^2 weight of rows (.., y, z) of a (d, d, *) block that starts at `pad` on
// every axis of an (n0, n1, n2) array.
enum class RowWeight { kNone, kSinc2, kOverSinc2 };
struct RowWeights {
    int d, pad, n0, n1, n2;
    float i0, i1, i2;
};
static RowWeights make_weights(int64_t d, int64_t pad, int64_t n0, int64_t n1, int64_t n2) {
    return RowWeights{(int)d,  (int)pad, (int)n0, (int)n1, (int)n2, (float)(1.0 / (double)n0), (float)(1.0 / (double)n1),
                      (float)(1.0 / (double)n2)};
}
__device__ __forceinline__ float row_f01(const RowWeights& w, int64_t row) {
    const int r = (int)(row % ((int64_t)w.d * w.d));
    const float f0 = shifted_fftfreq(r / w.d + w.pad, w.n0, w.i0);
    const float f1 = shifted_fftfreq(r % w.d + w.pad, w.n1, w.i1);
    return __fadd_rn(__fmul_rn(f0, f0), __fmul_rn(f1, f1));
}

// Real rows (rows, len) -> half spectra (rows, n/2 + 1): sample x of a row sits
// at position (x + off) mod n of a zero row of n.  Two rows per complex
// transform.  Bins are scaled by `edge` (0 and n/2) and `inner` (the others).
template <RowWeight W>
__global__ void __launch_bounds__(kFftMaxThreads)
rows_r2c_kernel(const float* __restrict__ in, float2* __restrict__ out, int64_t rows, int len, int off, float edge,
                float inner, const __grid_constant__ FftPlan p, RowWeights rw) {
    extern __shared__ float2 fft_smem[];
    const int n = p.n, wr = n / 2 + 1;
    float2 *a = fft_smem, *b = a + n * kFftBatch, *tw = b + n * kFftBatch;
    fft_roots(tw, n);
    const int64_t first = (int64_t)blockIdx.x * (2 * kFftBatch);
    const int span = (n + 31) & ~31;  // whole warps along a row
    for (int i = threadIdx.x; i < span * kFftBatch; i += blockDim.x) {
        const int c = i / span, k = i - c * span;
        if (k >= n) continue;
        int x = k - off;
        if (x < 0) x += n;
        const int64_t r0 = first + 2 * c;
        float2 v = make_float2(0.f, 0.f);
        if (x < len && r0 < rows) {
            v.x = __ldg(in + r0 * len + x);
            if (r0 + 1 < rows) v.y = __ldg(in + (r0 + 1) * len + x);
            if (W == RowWeight::kSinc2) {
                const float f2 = shifted_fftfreq(x + rw.pad, rw.n2, rw.i2);
                v.x *= sinc2_from(row_f01(rw, r0), f2);
                v.y *= sinc2_from(row_f01(rw, r0 + 1), f2);
            }
        }
        a[fft_at<true>(k, c)] = v;
    }
    __syncthreads();
    const float2* z = fft_run<false, true>(a, b, tw, p);
    const int ospan = (wr + 31) & ~31;
    for (int i = threadIdx.x; i < ospan * kFftBatch; i += blockDim.x) {
        const int c = i / ospan, k = i - c * ospan;
        const int64_t r0 = first + 2 * c;
        if (k >= wr || r0 >= rows) continue;
        const float2 u = z[fft_at<true>(k, c)], m = z[fft_at<true>(k ? n - k : 0, c)];
        const float f = 0.5f * (k == 0 || 2 * k == n ? edge : inner);
        // Z = X1 + i X2: X1 = (Z[k] + conj Z[n-k]) / 2, X2 = (Z[k] - conj Z[n-k]) / 2i
        out[r0 * wr + k] = make_float2(f * (u.x + m.x), f * (u.y - m.y));
        if (r0 + 1 < rows) out[(r0 + 1) * wr + k] = make_float2(f * (u.y + m.y), f * (m.x - u.x));
    }
}

// Half spectra (rows, n/2 + 1) -> real rows: samples (x + off) mod n, x < len,
// of the inverse real transform (unscaled, times `scale` and the weight).  The
// imaginary parts of bins 0 and n/2 are ignored; the other bins are scaled by
// `inner` (1: the inverse of a real transform; 1/2: its adjoint).
template <RowWeight W>
__global__ void __launch_bounds__(kFftMaxThreads)
rows_c2r_kernel(const float2* __restrict__ in, float* __restrict__ out, int64_t rows, int len, int off, float inner,
                float scale, const __grid_constant__ FftPlan p, RowWeights rw) {
    extern __shared__ float2 fft_smem[];
    const int n = p.n, wr = n / 2 + 1;
    float2 *a = fft_smem, *b = a + n * kFftBatch, *tw = b + n * kFftBatch;
    fft_roots(tw, n);
    const int64_t first = (int64_t)blockIdx.x * (2 * kFftBatch);
    const int span = (wr + 31) & ~31;
    for (int i = threadIdx.x; i < span * kFftBatch; i += blockDim.x) {
        const int c = i / span, k = i - c * span;
        if (k >= wr) continue;
        const int64_t r0 = first + 2 * c;
        float2 u = make_float2(0.f, 0.f), v = u;
        if (r0 < rows) u = __ldcs(in + r0 * wr + k);
        if (r0 + 1 < rows) v = __ldcs(in + (r0 + 1) * wr + k);
        if (k == 0 || 2 * k == n) {
            a[fft_at<true>(k, c)] = make_float2(u.x, v.x);
        } else {  // Z[k] = X1 + i X2, Z[n-k] = conj X1 + i conj X2
            u.x *= inner;
            u.y *= inner;
            v.x *= inner;
            v.y *= inner;
            a[fft_at<true>(k, c)] = make_float2(u.x - v.y, u.y + v.x);
            a[fft_at<true>(n - k, c)] = make_float2(u.x + v.y, v.x - u.y);
        }
    }
    __syncthreads();
    const float2* z = fft_run<true, true>(a, b, tw, p);
    const int ospan = (len + 31) & ~31;
    for (int i = threadIdx.x; i < ospan * kFftBatch; i += blockDim.x) {
        const int c = i / ospan, x = i - c * ospan;
        const int64_t r0 = first + 2 * c;
        if (x >= len || r0 >= rows) continue;
        int k = x + off;
        if (k >= n) k -= n;
        float2 v = z[fft_at<true>(k, c)];
        v.x *= scale;
        v.y *= scale;
        if (W != RowWeight::kNone) {
            const float f2 = shifted_fftfreq(x + rw.pad, rw.n2, rw.i2);
            const float s0 = sinc2_from(row_f01(rw, r0), f2), s1 = sinc2_from(row_f01(rw, r0 + 1), f2);
            v.x = W == RowWeight::kSinc2 ? v.x * s0 : v.x / s0;
            v.y = W == RowWeight::kSinc2 ? v.y * s1 : v.y / s1;
        }
        out[r0 * len + x] = v.x;
        if (r0 + 1 < rows) out[(r0 + 1) * len + x] = v.y;
    }
}

// Columns of `cols` complex samples: row r of batch b at base + b * batch + r * row.
// Input rows r sit at (r + off) mod n of a zero column; output rows r are the
// transform's samples (r + off) mod n.
struct Columns {
    int64_t batch, row;
    int rows, off;
};

template <bool INV>
__global__ void __launch_bounds__(kFftMaxThreads)
columns_kernel(const float2* __restrict__ in, Columns ci, float2* __restrict__ out, Columns co, int cols, int xtiles,
               const __grid_constant__ FftPlan p) {
    extern __shared__ float2 fft_smem[];
    const int n = p.n;
    float2 *a = fft_smem, *b = a + n * kFftBatch, *tw = b + n * kFftBatch;
    fft_roots(tw, n);
    const int64_t bi = blockIdx.x / xtiles;
    const int x0 = (int)(blockIdx.x - bi * xtiles) * kFftBatch;
    const int c = threadIdx.x & (kFftBatch - 1), x = x0 + c;  // blockDim is a multiple of 8: one column per thread
    const float2* src = in + bi * ci.batch + x;
    for (int k = threadIdx.x >> 3; k < n; k += blockDim.x >> 3) {
        int r = k - ci.off;
        if (r < 0) r += n;
        a[k * kFftBatch + c] = (r < ci.rows && x < cols) ? __ldcs(src + r * ci.row) : make_float2(0.f, 0.f);
    }
    __syncthreads();
    const float2* z = fft_run<INV, false>(a, b, tw, p);
    if (x >= cols) return;
    float2* dst = out + bi * co.batch + x;
    for (int r = threadIdx.x >> 3; r < co.rows; r += blockDim.x >> 3) {
        int k = r + co.off;
        if (k >= n) k -= n;
        dst[r * co.row] = z[k * kFftBatch + c];
    }
}

// z transforms of (d, e, wr) half spectra (y fftshifted) into the bricked copy
// of the fftshifted (e, e, wr) volume.  A block takes two rows y and four
// columns x, so it stores whole pairs of bricks (128-byte lines); slots past an
// odd e are zero.
__global__ void __launch_bounds__(kFftMaxThreads)
columns_to_bricks_kernel(const float2* __restrict__ in, int rows, int off, float2* __restrict__ bricks, int wr,
                         int xtiles, const __grid_constant__ FftPlan p) {
    extern __shared__ float2 fft_smem[];
    const int n = p.n, bh = (n + 1) >> 1, bw = (wr + 1) >> 1;
    float2 *a = fft_smem, *b = a + n * kFftBatch, *tw = b + n * kFftBatch;
    fft_roots(tw, n);
    const int by = blockIdx.x / xtiles, xt = blockIdx.x - by * xtiles;
    const int c = threadIdx.x & (kFftBatch - 1);
    const int y = 2 * by + (c >> 2), x = 4 * xt + (c & 3);
    const bool live = y < n && x < wr;
    const float2* src = in + (int64_t)y * wr + x;
    for (int k = threadIdx.x >> 3; k < n; k += blockDim.x >> 3) {
        int r = k - off;
        if (r < 0) r += n;
        a[k * kFftBatch + c] = (r < rows && live) ? __ldcs(src + (int64_t)r * n * wr) : make_float2(0.f, 0.f);
    }
    __syncthreads();
    const float2* f = fft_run<false, false>(a, b, tw, p);
    // slot s of brick t of the pair: z = 2 zb + bit 2, y bit 1, x = 2 t + bit 0
    const int shift = n - n / 2;  // z (fftshifted) is sample (z + shift) mod n
    for (int i = threadIdx.x; i < bh * 16; i += blockDim.x) {
        const int zb = i >> 4, t = (i >> 3) & 1, s = i & 7;
        if (2 * xt + t >= bw) continue;
        const int z = 2 * zb + (s >> 2);
        int k = z + shift;
        if (k >= n) k -= n;
        const int q = ((s >> 1) & 1) * 4 + 2 * t + (s & 1);
        bricks[(((int64_t)zb * bh + by) * bw + 2 * xt + t) * 8 + s] =
            z < n ? f[k * kFftBatch + q] : make_float2(0.f, 0.f);
    }
}

// Insertion accumulators (float4 slots, fftshifted; BRICKED: accumulator_slot
// order) -> Friedel completion, division by max(weights, 1), inverse z
// transforms, planes (z + off) mod n of them: (rows, e, wr) with y fftshifted.
// One block per two rows y and four columns x of a channel (grid y); the
// weights are channel 0's.
template <bool BRICKED>
__global__ void __launch_bounds__(kFftMaxThreads)
normalize_columns_kernel(const float4* __restrict__ acc, int64_t stride, float2* __restrict__ out, int rows, int off,
                         int wr, int xtiles, const __grid_constant__ FftPlan p) {
    extern __shared__ float2 fft_smem[];
    const int n = p.n;
    float2 *a = fft_smem, *b = a + n * kFftBatch, *tw = b + n * kFftBatch;
    fft_roots(tw, n);
    SliceGeom g{};  // accumulator_slot reads the volume dims only
    g.D = n;
    g.H = n;
    g.W = wr;
    const int by = blockIdx.x / xtiles, xt = blockIdx.x - by * xtiles;
    const int c = threadIdx.x & (kFftBatch - 1);
    const int y = 2 * by + (c >> 2), x = 4 * xt + (c & 3);
    const bool live = y < n && x < wr;
    const float4* ch = acc + blockIdx.y * stride;
    const int shift = n - n / 2;
    auto slot = [&](int z, int yy, int xx) -> int64_t {
        return BRICKED ? accumulator_slot(g, z, yy, xx) : ((int64_t)z * n + yy) * wr + xx;
    };
    for (int z = threadIdx.x >> 3; z < n; z += blockDim.x >> 3) {
        float2 v = make_float2(0.f, 0.f);
        if (live) {
            const int64_t s = slot(z, y, x);
            const float4 q = ch[s];
            float re = q.x, im = q.y, w = blockIdx.y ? acc[s].z : q.z;
            if (x == 0) {
                const int zm = z ? n - z : 0, ym = y ? n - y : 0;
                if (!(zm == n / 2 && ym == n / 2)) {
                    const int64_t sm = slot(zm, ym, 0);
                    const float4 u = ch[sm];
                    re += u.x;
                    im -= u.y;
                    w += acc[sm].z;
                }
            }
            const float den = w < 1.0f ? 1.0f : w;
            v = make_float2(re / den, im / den);
        }
        int k = z + shift;
        if (k >= n) k -= n;
        a[k * kFftBatch + c] = v;
    }
    __syncthreads();
    const float2* f = fft_run<true, false>(a, b, tw, p);
    if (!live) return;
    float2* dst = out + ((int64_t)blockIdx.y * rows * n + y) * wr + x;
    for (int r = threadIdx.x >> 3; r < rows; r += blockDim.x >> 3) {
        int k = r + off;
        if (k >= n) k -= n;
        dst[(int64_t)r * n * wr] = f[k * kFftBatch + c];
    }
}

// Central slices from the bricked copy and their inverse y transforms in one
// kernel: a block samples eight columns of one slice (a warp's 8 x 4 patch of
// pixels as in extract_fwd_kernel, the same geometry, values and rounding),
// transforms them and stores rows (r + off) mod e, r < rows, of
// (n, channels, rows, wr).  The slices never reach HBM.
__global__ void __launch_bounds__(kFftMaxThreads)
slice_columns_kernel(const VoxBrick2* __restrict__ bricks, int64_t vstride, int channels, const void* __restrict__ rot,
                     float2* __restrict__ out, int rows, int off, int xtiles, SliceGeom g,
                     const __grid_constant__ FftPlan p) {
    extern __shared__ float2 fft_smem[];
    __shared__ float m[9];
    const int n = p.n;
    float2 *a = fft_smem, *b = a + n * kFftBatch, *tw = b + n * kFftBatch;
    const int64_t sc = blockIdx.x / xtiles;  // slice and channel
    const int xt = (int)(blockIdx.x - sc * xtiles);
    const int64_t s = sc / channels;
    if (threadIdx.x < 9) m[threadIdx.x] = prep_rotation_elem(rot, g.rot_f64, s, threadIdx.x, g, true);
    fft_roots(tw, n);
    __syncthreads();
    const VoxBrick2* vol = bricks + (sc - s * channels) * vstride;
    const int c = threadIdx.x & (kFftBatch - 1), ix = xt * kFftBatch + c;
    const int shift = n - n / 2;
    // the column part of the geometry (slice_row_geom's counterpart), rounded
    // as rotate_slice_point rounds it
    const float qx = __fmul_rn((float)ix, g.inv_w), qx2 = __fmul_rn(qx, qx);
    float mx[3];
#pragma unroll
    for (int i = 0; i < 3; i++) mx[i] = __fmul_rn(m[i * 3 + 2], qx);
#pragma unroll 4
    for (int iy = threadIdx.x >> 3; iy < n; iy += blockDim.x >> 3) {
        float2 r = make_float2(0.f, 0.f);
        const float qy = shifted_freq(iy, n, g.inv_h);
        if (ix < g.wr && (!g.has_fmax || __fsqrt_rn(__fadd_rn(__fmul_rn(qy, qy), qx2)) <= g.fmax)) {
            float q[3], cc[3];
#pragma unroll
            for (int i = 0; i < 3; i++) q[i] = __fadd_rn(__fmul_rn(m[i * 3 + 1], qy), mx[i]);
            const bool cj = extract_conj(g, m, q[2]);
            if (cj) {
                q[0] = -q[0];
                q[1] = -q[1];
                q[2] = -q[2];
            }
            to_dft_coords(g, q, cc);
            if (inside_volume(g, cc)) {
                r = sample_trilinear(vol, g, make_corners(g, cc));
                if (cj) r.y = -r.y;
            }
        }
        int k = iy + shift;
        if (k >= n) k -= n;
        a[k * kFftBatch + c] = r;
    }
    __syncthreads();
    const float2* f = fft_run<true, false>(a, b, tw, p);
    if (ix >= g.wr) return;
    float2* dst = out + sc * rows * (int64_t)g.wr + ix;
    for (int r = threadIdx.x >> 3; r < rows; r += blockDim.x >> 3) {
        int k = r + off;
        if (k >= n) k -= n;
        dst[(int64_t)r * g.wr] = f[k * kFftBatch + c];
    }
}

// ------------------------------------------------------------------ launches

template <typename K>
static int fft_smem(K kernel, const FftPlan& p, size_t& bytes) {
    bytes = fft_smem_bytes(p.n);
    if (bytes > 48 * 1024) {
        cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
        if (e != cudaSuccess) return fail(TT_ERR_CUDA, "transform: shared memory: %s", cudaGetErrorString(e));
    }
    return TT_OK;
}

static int row_blocks(int64_t rows, unsigned& blocks) {
    const int64_t b = (rows + 2 * kFftBatch - 1) / (2 * kFftBatch);
    if (b > 0x7fffffffLL) return fail(TT_ERR_INVALID, "transform: too many rows");
    blocks = (unsigned)b;
    return TT_OK;
}

template <RowWeight W>
static int launch_r2c(const float* in, float2* out, int64_t rows, int64_t len, int64_t off, float edge, float inner,
                      const FftPlan& p, const RowWeights& rw, cudaStream_t st) {
    size_t sm;
    unsigned blocks;
    if (int e = fft_smem(rows_r2c_kernel<W>, p, sm)) return e;
    if (int e = row_blocks(rows, blocks)) return e;
    rows_r2c_kernel<W><<<blocks, fft_threads(p.n), sm, st>>>(in, out, rows, (int)len, (int)(off % p.n), edge, inner, p,
                                                             rw);
    return check_launch("rows_r2c_kernel");
}

template <RowWeight W>
static int launch_c2r(const float2* in, float* out, int64_t rows, int64_t len, int64_t off, float inner, float scale,
                      const FftPlan& p, const RowWeights& rw, cudaStream_t st) {
    size_t sm;
    unsigned blocks;
    if (int e = fft_smem(rows_c2r_kernel<W>, p, sm)) return e;
    if (int e = row_blocks(rows, blocks)) return e;
    rows_c2r_kernel<W><<<blocks, fft_threads(p.n), sm, st>>>(in, out, rows, (int)len, (int)(off % p.n), inner, scale, p,
                                                             rw);
    return check_launch("rows_c2r_kernel");
}

template <bool INV>
static int launch_columns(const float2* in, Columns ci, float2* out, Columns co, int64_t batches, int cols,
                          const FftPlan& p, cudaStream_t st) {
    size_t sm;
    if (int e = fft_smem(columns_kernel<INV>, p, sm)) return e;
    const int xtiles = (cols + kFftBatch - 1) / kFftBatch;
    if (batches * xtiles > 0x7fffffffLL) return fail(TT_ERR_INVALID, "transform: too many columns");
    ci.off %= p.n;
    co.off %= p.n;
    columns_kernel<INV><<<(unsigned)(batches * xtiles), fft_threads(p.n), sm, st>>>(in, ci, out, co, cols, xtiles, p);
    return check_launch("columns_kernel");
}

// Plans of a padded box: e and, for the inverse real transforms, L = 2 (wr - 1).
struct BoxPlans {
    int64_t d, p, e, wr, l, crop;  // crop = L - 2 p, the width of the cropped output
    FftPlan pe, pl;
};
static int make_box(int64_t d, int64_t pad, BoxPlans& b) {
    if (d < 1 || pad < 0 || d > kFftMaxLength || pad > kFftMaxLength)
        return fail(TT_ERR_INVALID, "transform: bad box");
    b.d = d;
    b.p = pad;
    b.e = d + 2 * pad;
    b.wr = b.e / 2 + 1;
    b.l = 2 * (b.wr - 1);
    b.crop = b.l - 2 * pad;
    if (!make_fft_plan(b.e, b.pe) || !make_fft_plan(b.l, b.pl) || b.crop < 1)
        return fail(TT_ERR_INVALID, "transform: box %lld padded to %lld is not supported", (long long)d,
                    (long long)b.e);
    return TT_OK;
}

}  // namespace tt

using namespace tt;

extern "C" int32_t tt_transform_supported(int64_t d, int64_t pad) {
    BoxPlans b;
    return make_box(d, pad, b) == TT_OK;
}

extern "C" size_t tt_transform_workspace_bytes(int32_t volumes, int64_t count, int64_t d, int64_t pad) {
    if (count < 0 || d < 1 || pad < 0) return 0;
    const int64_t e = d + 2 * pad, wr = e / 2 + 1;
    // volumes: x spectra of d^2 rows beside the (d, e, wr) planes; images: d rows each
    return (size_t)(count * d * wr * (volumes ? d + e : 1)) * sizeof(float2);
}

static int check_transform(const void* in, const void* out, const void* workspace, size_t workspace_bytes,
                           int32_t volumes, int64_t count, int64_t d, int64_t pad, BoxPlans& b, const char* what) {
    if (int e = make_box(d, pad, b)) return e;
    if (count < 0) return fail(TT_ERR_INVALID, "%s: negative count", what);
    if (!in || !out) return fail(TT_ERR_INVALID, "%s: NULL pointer argument", what);
    const size_t need = tt_transform_workspace_bytes(volumes, count, d, pad);
    if (need && (!workspace || workspace_bytes < need))
        return fail(TT_ERR_WORKSPACE, "%s: workspace of %zu bytes needed, got %zu", what, need, workspace_bytes);
    return TT_OK;
}

extern "C" int tt_project_volume_bricks(const float* volumes, int64_t channels, int64_t d, int64_t pad, void* bricks,
                                        void* workspace, size_t workspace_bytes, void* stream) {
    BoxPlans b;
    if (int e = check_transform(volumes, bricks, workspace, workspace_bytes, 1, channels, d, pad, b,
                                "project_volume_bricks"))
        return e;
    if (channels == 0) return TT_OK;
    cudaStream_t st = as_stream(stream);
    float2* xs = (float2*)workspace;                        // (c, d, d, wr)
    float2* ys = xs + channels * d * d * b.wr;              // (c, d, e, wr)
    const int64_t at = pad + b.e / 2;                       // fftshift(pad(v)): sample x at (x + at) mod e
    const int64_t shift = b.e - b.e / 2;                    // fftshifted row r is bin (r + shift) mod e
    if (int e = launch_r2c<RowWeight::kSinc2>(volumes, xs, channels * d * d, d, at, 1.f, 1.f, b.pe,
                                              make_weights(d, pad, b.e, b.e, b.e), st))
        return e;
    if (int e = launch_columns<false>(xs, Columns{d * b.wr, b.wr, (int)d, (int)at}, ys,
                                      Columns{b.e * b.wr, b.wr, (int)b.e, (int)shift}, channels * d, (int)b.wr, b.pe,
                                      st))
        return e;
    size_t sm;
    if (int e = fft_smem(columns_to_bricks_kernel, b.pe, sm)) return e;
    const int xtiles = (int)((b.wr + 3) / 4), bh = (int)((b.e + 1) / 2);
    const int64_t slots = (int64_t)bh * bh * ((b.wr + 1) / 2) * 8;
    for (int64_t ch = 0; ch < channels; ch++) {
        columns_to_bricks_kernel<<<(unsigned)(bh * xtiles), fft_threads(b.pe.n), sm, st>>>(
            ys + ch * d * b.e * b.wr, (int)d, (int)(at % b.e), (float2*)bricks + ch * slots, (int)b.wr, xtiles, b.pe);
        if (int e = check_launch("columns_to_bricks_kernel")) return e;
    }
    return TT_OK;
}

extern "C" int tt_project_slices(const void* bricks, int64_t channels, const void* rotation_matrices, int64_t d,
                                 int64_t pad, float* images, void* workspace, size_t workspace_bytes,
                                 const tt_slice_params* p, void* stream) {
    if (int e = validate_params(p, true)) return e;
    BoxPlans b;
    if (int e = check_transform(bricks, images, workspace, workspace_bytes, 0, p->n * channels, d, pad, b,
                                "project_slices"))
        return e;
    if (channels < 1 || channels > 4096) return fail(TT_ERR_INVALID, "project_slices: channels must be in [1, 4096]");
    if (p->img_d != b.e || p->img_h != b.e || p->img_w != b.e || p->vol_d != b.e || p->vol_h != b.e ||
        p->vol_w != b.wr || p->volume_layout != TT_VOLUME_BRICKS)
        return fail(TT_ERR_INVALID, "project_slices: the params are not those of a bricked padded box");
    if (p->n == 0) return TT_OK;
    if (!rotation_matrices) return fail(TT_ERR_INVALID, "project_slices: NULL pointer argument");
    SliceGeom g = make_geom(*p);
    cudaStream_t st = as_stream(stream);
    float2* cs = (float2*)workspace;  // (n, c, d, wr)
    size_t sm;
    if (int e = fft_smem(slice_columns_kernel, b.pe, sm)) return e;
    const int xtiles = (int)((b.wr + kFftBatch - 1) / kFftBatch);
    const int64_t blocks = p->n * channels * xtiles;
    if (blocks > 0x7fffffffLL) return fail(TT_ERR_INVALID, "project_slices: too many blocks");
    const int64_t half = (b.e + 1) / 2;
    slice_columns_kernel<<<(unsigned)blocks, fft_threads(b.pe.n), sm, st>>>(
        (const VoxBrick2*)bricks, half * half * ((b.wr + 1) / 2) * 8, (int)channels, rotation_matrices, cs, (int)d,
        (int)((pad + b.e / 2) % b.e), xtiles, g, b.pe);
    if (int e = check_launch("slice_columns_kernel")) return e;
    return launch_c2r<RowWeight::kNone>(cs, images, p->n * channels * d, b.crop, pad + b.l / 2, 1.f,
                                        (float)(1.0 / ((double)b.e * (double)b.l)), b.pl, RowWeights{}, st);
}

extern "C" int tt_project_slices_backward(const float* grad_images, int64_t count, int64_t d, int64_t pad,
                                          void* grad_slices, void* workspace, size_t workspace_bytes, void* stream) {
    BoxPlans b;
    if (int e = check_transform(grad_images, grad_slices, workspace, workspace_bytes, 0, count, d, pad, b,
                                "project_slices_backward"))
        return e;
    if (count == 0) return TT_OK;
    cudaStream_t st = as_stream(stream);
    float2* cs = (float2*)workspace;
    // adjoint of the inverse real transform: bins 0 and L/2 once, the others twice
    const float f = (float)(1.0 / ((double)b.e * (double)b.l));
    if (int e = launch_r2c<RowWeight::kNone>(grad_images, cs, count * d, b.crop, pad + b.l / 2, f, 2.f * f, b.pl,
                                             RowWeights{}, st))
        return e;
    return launch_columns<false>(cs, Columns{d * b.wr, b.wr, (int)d, (int)(pad + b.e / 2)}, (float2*)grad_slices,
                                 Columns{b.e * b.wr, b.wr, (int)b.e, (int)(b.e - b.e / 2)}, count, (int)b.wr, b.pe, st);
}

extern "C" int tt_project_volume_backward(const void* grad_dft, int64_t channels, int64_t d, int64_t pad,
                                          float* grad_volumes, void* workspace, size_t workspace_bytes, void* stream) {
    BoxPlans b;
    if (int e = check_transform(grad_dft, grad_volumes, workspace, workspace_bytes, 1, channels, d, pad, b,
                                "project_volume_backward"))
        return e;
    if (channels == 0) return TT_OK;
    cudaStream_t st = as_stream(stream);
    float2* xs = (float2*)workspace;            // (c, d, d, wr)
    float2* zs = xs + channels * d * d * b.wr;  // (c, d, e, wr)
    const int64_t at = pad + b.e / 2, shift = b.e - b.e / 2, plane = b.e * b.wr;
    for (int64_t ch = 0; ch < channels; ch++)  // along z, one batch per row y
        if (int e = launch_columns<true>((const float2*)grad_dft + ch * b.e * plane,
                                         Columns{b.wr, plane, (int)b.e, (int)shift}, zs + ch * d * plane,
                                         Columns{b.wr, plane, (int)d, (int)at}, b.e, (int)b.wr, b.pe, st))
            return e;
    if (int e = launch_columns<true>(zs, Columns{plane, b.wr, (int)b.e, (int)shift}, xs,
                                     Columns{d * b.wr, b.wr, (int)d, (int)at}, channels * d, (int)b.wr, b.pe, st))
        return e;
    // adjoint of the real transform: the real part of the half spectrum's inverse, mates not doubled
    return launch_c2r<RowWeight::kSinc2>(xs, grad_volumes, channels * d * d, d, at, 0.5f, 1.f, b.pe,
                                         make_weights(d, pad, b.e, b.e, b.e), st);
}

extern "C" int tt_backproject_spectra(const float* images, int64_t count, int64_t d, int64_t pad, void* slices,
                                      void* workspace, size_t workspace_bytes, void* stream) {
    BoxPlans b;
    if (int e = check_transform(images, slices, workspace, workspace_bytes, 0, count, d, pad, b, "backproject_spectra"))
        return e;
    if (count == 0) return TT_OK;
    cudaStream_t st = as_stream(stream);
    float2* xs = (float2*)workspace;
    const int64_t at = pad + b.e / 2;
    if (int e = launch_r2c<RowWeight::kNone>(images, xs, count * d, d, at, 1.f, 1.f, b.pe, RowWeights{}, st)) return e;
    return launch_columns<false>(xs, Columns{d * b.wr, b.wr, (int)d, (int)at}, (float2*)slices,
                                 Columns{b.e * b.wr, b.wr, (int)b.e, (int)(b.e - b.e / 2)}, count, (int)b.wr, b.pe, st);
}

extern "C" int tt_backproject_volume(const void* accumulator, int32_t bricked, int64_t channels, int64_t d, int64_t pad,
                                     float* volumes, void* workspace, size_t workspace_bytes, void* stream) {
    BoxPlans b;
    if (int e = check_transform(accumulator, volumes, workspace, workspace_bytes, 1, channels, d, pad, b,
                                "backproject_volume"))
        return e;
    if (channels < 1 || channels > 4096)
        return fail(TT_ERR_INVALID, "backproject_volume: channels must be in [1, 4096]");
    cudaStream_t st = as_stream(stream);
    float2* xs = (float2*)workspace;            // (c, d, d, wr)
    float2* zs = xs + channels * d * d * b.wr;  // (c, d, e, wr)
    const int64_t at = pad + b.e / 2, plane = b.e * b.wr, half = (b.e + 1) / 2;
    const int xtiles = (int)((b.wr + 3) / 4);
    const dim3 grid((unsigned)(half * xtiles), (unsigned)channels);
    size_t sm;
    if (bricked) {
        if (int e = fft_smem(normalize_columns_kernel<true>, b.pe, sm)) return e;
        normalize_columns_kernel<true><<<grid, fft_threads(b.pe.n), sm, st>>>(
            (const float4*)accumulator, half * half * ((b.wr + 1) / 2) * 8, zs, (int)d, (int)(at % b.e), (int)b.wr,
            xtiles, b.pe);
    } else {
        if (int e = fft_smem(normalize_columns_kernel<false>, b.pe, sm)) return e;
        normalize_columns_kernel<false><<<grid, fft_threads(b.pe.n), sm, st>>>(
            (const float4*)accumulator, b.e * plane, zs, (int)d, (int)(at % b.e), (int)b.wr, xtiles, b.pe);
    }
    if (int e = check_launch("normalize_columns_kernel")) return e;
    if (int e = launch_columns<true>(zs, Columns{plane, b.wr, (int)b.e, (int)(b.e - b.e / 2)}, xs,
                                     Columns{d * b.wr, b.wr, (int)d, (int)at}, channels * d, (int)b.wr, b.pe, st))
        return e;
    const double scale = 1.0 / ((double)b.e * (double)b.e * (double)b.l);
    return launch_c2r<RowWeight::kOverSinc2>(xs, volumes, channels * d * d, b.crop, pad + b.l / 2, 1.f, (float)scale,
                                             b.pl, make_weights(d, pad, b.e, b.e, b.l), st);
}
