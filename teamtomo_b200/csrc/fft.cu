// The transforms of project_3d_to_2d (torch_fourier_slice/project.py:48-92) and
// backproject_2d_to_3d (torch_fourier_slice/backproject.py:48-92), with their
// padding, shifts, weights, cropping and layouts in the kernels' loads and
// stores (the transform itself is in fft.cuh).
//
// Padded box e = d + 2 p, half spectrum wr = e/2 + 1, and L = 2 (wr - 1) the
// length of the inverse real transform (the reference runs irfftn without an
// output size, so L = e - 1 for odd e).
//
//   projection       volume (d, d, d) times sinc^2 -> x transforms of its d^2 rows
//                    -> y transforms of d planes -> z transforms, stored as the
//                    bricked copy the gathers read (tt_pack_volume_bricks)
//                    -> central slices -> inverse y transforms, the d kept rows
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
// the scaling and the layouts.  Measured on a B200, whole calls with the
// library transforms / here: 64^3 x 100 projections 102 / 59 us, 90^3 x 256
// with both gradients 1021 / 343 us, two 160^3 maps x 400 2684 / 883 us,
// 10,000 images of 128^2 (the insertion takes 7.1 ms of it) 13.4 / 9.1 to 9.5 ms.
// Passes of radix 8, 4, 2 and odd primes through shared memory with a barrier
// each took 1.58 (rows) and 2.16 ms (columns) of the last, the passes in
// registers 0.63 and 1.00 ms, at floors of 0.30 and 0.61 ms of HBM traffic:
// the kernels are bound by instruction issue (about 50 per sample) at four
// blocks' registers per SM.  Sampling the slices in the column kernel took
// longer than the extraction and the transform one after the other (990 / 800
// against 460 + 150 us for 2 x 400 slices of 320): the gathers want more
// resident threads than a transform's registers leave.
#include <cuda_runtime.h>

#include "capi_util.cuh"
#include "fft.cuh"
#include "real_space.cuh"
#include "slice_common.cuh"
#include "slice_ops.cuh"

namespace tt {

// Maps (rows / d^2, d, d, len) that start at `pad` on every axis of an
// (n, n, n2) array, times (DIV: over) the array's sinc(|f|)^2.  One warp per
// row: its two leading frequencies are formed once.  A pass of its own because
// the weight costs more than a transform's step per sample and the transform
// kernels hold their samples in registers.  `out` may be `in`.
template <bool DIV>
__global__ void __launch_bounds__(256)
sinc2_kernel(const float* in, float* out, int64_t rows, int d, int len, int pad, int n, int n2, float inv_n,
             float inv_n2) {
    const int64_t row = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    if (row >= rows) return;
    const int r = (int)(row % ((int64_t)d * d));
    const float f0 = shifted_fftfreq(r / d + pad, n, inv_n), f1 = shifted_fftfreq(r % d + pad, n, inv_n);
    const float f01 = __fadd_rn(__fmul_rn(f0, f0), __fmul_rn(f1, f1));
    for (int x = threadIdx.x & 31; x < len; x += 32) {
        const float w = sinc2_from(f01, shifted_fftfreq(x + pad, n2, inv_n2)), v = in[row * len + x];
        out[row * len + x] = DIV ? v / w : v * w;
    }
}

// The tile that the last pass does not read (staged results).
__device__ __forceinline__ float2* fft_free_tile(float2* a, float2* b, const FftPlan& p) {
    return (p.passes & 1) ? a : b;
}

// Real rows are transformed two at a time, as the real and imaginary part of
// one complex row, which mixes their rounding errors and spreads a NaN or an
// infinity of one over the other: a pair never holds rows of two images (maps,
// channels, orientations), so an image comes out as it would alone.  ODD: the
// images have an odd number of rows, each one's last row goes with zeros, and a
// tile's pairs may belong to several images.  With an even number (and for one
// image) consecutive rows never straddle.  Row transforms, pairs of the launch /
// pairs of an image: 4000 images of 33^2 33.0 / 34.8 us (3 % more transforms),
// of 45^2 29.5 / 31.5, 600 of 113^2 40.3 / 36.2; inverse ones of 8000 images of
// 33^2 34.6 / 34.9, of 45^2 47.0 / 49.3, 1200 of 113^2 60.5 / 60.9.
struct RowPairs {
    int64_t count;  // rows; pairs when ODD
    uint32_t per;   // ODD: pairs of an image
    uint32_t inv;   // ODD: floor((2^32 - 1) / per)
};
inline RowPairs make_row_pairs(int64_t images, int64_t rows, bool& odd) {
    odd = images > 1 && (rows & 1);
    if (!odd) return RowPairs{images * rows, 1, 0};
    const uint32_t per = (uint32_t)((rows + 1) / 2);
    return RowPairs{images * per, per, 0xffffffffu / per};
}

// A transform's rows, `at` and a row length further: the offset from the tile's
// first row (RowTile::first) and which exist.
struct RowPair {
    int at;
    bool one, two;
};

// The rows of a tile's transforms.  of(c, len) is what a butterfly keeps of
// transform c: its index, or (ODD) its pair, which formed again for each sample
// costs 5 % there; kept, it costs even tiles 2 to 4 %.
template <bool ODD>
struct RowTile {
    int left;  // rows left
    static __device__ __forceinline__ int64_t first(const RowPairs&, int64_t t) { return t * (2 * kFftBatch); }
    __device__ __forceinline__ RowTile(const RowPairs& p, int64_t t)
        : left((int)min((int64_t)(2 * kFftBatch), p.count - t * (2 * kFftBatch))) {}
    __device__ __forceinline__ int of(int c, int) const { return c; }
    __device__ __forceinline__ RowPair pair(int c, int len) const {
        return RowPair{2 * c * len, 2 * c < left, 2 * c + 1 < left};
    }
};
template <>
struct RowTile<true> {
    int left;        // pairs left
    uint32_t table;  // four bits a transform: images that end before it, whether one ends with it
    // Image of the tile's first pair (of fewer than 2^32) and the pair's place in it.
    static __device__ __forceinline__ uint32_t image(const RowPairs& p, int64_t t, uint32_t& k) {
        const uint32_t pair = (uint32_t)t * kFftBatch;
        uint32_t i = __umulhi(pair, p.inv);  // at most one too low
        k = pair - i * p.per;
        if (k >= p.per) {
            i++;
            k -= p.per;
        }
        return i;
    }
    static __device__ __forceinline__ int64_t first(const RowPairs& p, int64_t t) {
        uint32_t k;
        return 2 * kFftBatch * t - image(p, t, k);
    }
    __device__ __forceinline__ RowTile(const RowPairs& p, int64_t t)
        : left((int)min((int64_t)kFftBatch, p.count - t * kFftBatch)), table(0) {
        uint32_t k;
        image(p, t, k);
        // the pairs that end an image: one at most from eight pairs an image up
        for (uint32_t end = p.per - k; end <= kFftBatch; end += p.per)
            table += ((0x11111111u << (4 * (end - 1))) << 4) + (8u << (4 * (end - 1)));
    }
    __device__ __forceinline__ RowPair of(int c, int len) const {
        const int t = (int)(table >> (4 * c));
        return RowPair{(2 * c - (t & 7)) * len, c < left, c < left && !(t & 8)};
    }
    __device__ __forceinline__ RowPair pair(const RowPair& r, int) const { return r; }
    __device__ __forceinline__ RowPair pair(int c, int len) const { return of(c, len); }
};

template <bool ODD>
struct RealRows {
    const float* src;
    int len;
    RowTile<ODD> rows;
    __device__ __forceinline__ auto of(int c) const { return rows.of(c, len); }
    template <class C>
    __device__ __forceinline__ float2 get(int x, const C& c) const {
        float2 v = make_float2(0.f, 0.f);
        if (x < len) {
            const RowPair r = rows.pair(c, len);
            const int at = r.at + x;
            if (r.one) v.x = __ldcs(src + at);
            if (r.two) v.y = __ldcs(src + at + len);
        }
        return v;
    }
};
template <bool ODD>
struct RealRowsOut {
    float* dst;
    int len;
    RowTile<ODD> rows;
    float scale;
    __device__ __forceinline__ auto of(int c) const { return rows.of(c, len); }
    template <class C>
    __device__ __forceinline__ void put(int x, const C& c, float2 v) const {
        if (x >= len) return;
        const RowPair r = rows.pair(c, len);
        const int at = r.at + x;
        if (r.one) dst[at] = v.x * scale;
        if (r.two) dst[at + len] = v.y * scale;
    }
};

// Half spectra X1, X2 of the same rows as the spectrum X1 + i X2, of which bins
// past n / 2 are the conjugates of their mates n - k.  Only the real parts of bins
// 0 and n/2 count, times `edge`.
// Which side of n/2 a butterfly's sample r falls on is known from r and the
// radix R (but for the middle sample of odd ones), which leaves one address and
// no selects: 128,000 rows of 320 120 -> 100 us.
template <bool ODD>
struct HalfSpectra {
    const float2* src;
    int stride, n;
    float edge;
    RowTile<ODD> rows;
    struct Cursor {
        const float2 *lo, *hi;  // bin j and bin n - j of X1
        int j, nb, n, stride;
        float edge;
        bool one, two;
        __device__ __forceinline__ float2 get(int r, int R) const {
            const int i = j + r * nb;
            const bool mate = (2 * r == R - 1) ? 2 * i > n : 2 * r >= R;
            const float2* at = mate ? hi - r * nb : lo + r * nb;
            float2 u = make_float2(0.f, 0.f), v = u;
            if (one) u = __ldg(at);
            if (two) v = __ldg(at + stride);
            float2 z = mate ? make_float2(u.x + v.y, v.x - u.y) : make_float2(u.x - v.y, v.x + u.y);
            if ((r == 0 && j == 0) || ((2 * r == R || 2 * r == R - 1) && 2 * i == n))
                z = make_float2(edge * u.x, edge * v.x);
            return z;
        }
    };
    __device__ __forceinline__ Cursor from(int j, int c, int nb, const FftPlan&) const {
        const RowPair r = rows.pair(c, stride);
        const float2* row = src + r.at;
        return Cursor{row + j, row + n - j, j, nb, n, stride, edge, r.one, r.two};
    }
};

// Rows of the tile's complex columns, of which `cols` exist.
struct ColumnRows {
    const float2* src;
    int64_t row;
    int rows, cols;
    __device__ __forceinline__ int of(int c) const { return c; }
    __device__ __forceinline__ float2 get(int r, int c) const {
        return (r < rows && c < cols) ? __ldcs(src + r * row + c) : make_float2(0.f, 0.f);
    }
};
struct ColumnRowsOut {
    float2* dst;
    int64_t row;
    int rows, cols;
    __device__ __forceinline__ int of(int c) const { return c; }
    __device__ __forceinline__ void put(int r, int c, float2 v) const {
        if (r < rows && c < cols) dst[r * row + c] = v;
    }
};

// Real rows (rows, len) -> half spectra (n/2 + 1 bins at `stride`): sample x of
// a row sits at position (x + off) mod n of a zero row of n.  Two rows per
// complex transform (RowPairs).  Bins are scaled by `edge` (0 and n/2) and
// `inner` (the others).
template <bool ODD>
__global__ void __launch_bounds__(kFftMaxThreads, 4)
rows_r2c_kernel(const float* __restrict__ in, float2* __restrict__ out, RowPairs pairs, int len, int off, int stride,
                float edge, float inner, const __grid_constant__ FftPlan p, int64_t tiles) {
    extern __shared__ float2 fft_smem[];
    const int n = p.n, wr = n / 2 + 1, tile = fft_tile_size(p);
    float2 *a = fft_smem, *b = a + tile, *tw = b + tile;
    fft_roots<false>(tw, n);
    const PlainTile<false> z{fft_free_tile(a, b, p), n};
    for (int64_t t = blockIdx.x; t < tiles; t += gridDim.x) {
        const RowTile<ODD> rows(pairs, t);
        const int64_t first = RowTile<ODD>::first(pairs, t);
        const RealRows<ODD> rows_in{in + first * len, len, rows};
        fft_run<false, false>(Outside<RealRows<ODD>>{rows_in, off, n}, z, a, b, tw, p);
        __syncthreads();
        float2* dst = out + first * stride;
        // a warp takes 32 bins of a transform (no division by the row length: 10,000
        // images of 128^2 657 -> 631 us)
        for (int w = threadIdx.x >> 5; w < (wr + 31) / 32 * kFftBatch; w += blockDim.x >> 5) {
            const int c = w & (kFftBatch - 1), k = w / kFftBatch * 32 + (threadIdx.x & 31);
            const RowPair r = rows.pair(c, stride);
            if (k >= wr || !r.one) continue;
            const float2 u = z.at(k, c), m = z.at(k ? n - k : 0, c);
            const float f = 0.5f * (k == 0 || 2 * k == n ? edge : inner);
            // Z = X1 + i X2: X1 = (Z[k] + conj Z[n-k]) / 2, X2 = (Z[k] - conj Z[n-k]) / 2i
            const int at = r.at + k;
            dst[at] = make_float2(f * (u.x + m.x), f * (u.y - m.y));
            if (r.two) dst[at + stride] = make_float2(f * (u.y + m.y), f * (m.x - u.x));
        }
        __syncthreads();
    }
}

// Half spectra (n/2 + 1 bins at `stride`) -> real rows: samples (x + off) mod n,
// x < len, of the inverse real transform (unscaled, times `scale`).  The
// imaginary parts of bins 0 and n/2 are ignored; the other bins are scaled by
// `inner` (1: the inverse of a real transform; 1/2: its adjoint; a power of two).
template <bool ODD>
__global__ void __launch_bounds__(kFftMaxThreads, 4)
rows_c2r_kernel(const float2* __restrict__ in, float* __restrict__ out, RowPairs pairs, int len, int off, int stride,
                float inner, float scale, const __grid_constant__ FftPlan p, int64_t tiles, int smem_tiles) {
    extern __shared__ float2 fft_smem[];
    const int n = p.n, tile = fft_tile_size(p);
    float2 *a = fft_smem, *b = a + tile, *tw = a + tile * smem_tiles;
    fft_roots<true>(tw, n);
    for (int64_t t = blockIdx.x; t < tiles; t += gridDim.x) {
        const RowTile<ODD> rows(pairs, t);
        const int64_t first = RowTile<ODD>::first(pairs, t);
        const HalfSpectra<ODD> spectra{in + first * stride, stride, n, 1.0f / inner, rows};
        const RealRowsOut<ODD> rows_out{out + first * len, len, rows, scale * inner};
        fft_run<true, false>(spectra, Outside<RealRowsOut<ODD>>{rows_out, off, n}, a, b, tw, p);
        __syncthreads();
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
__global__ void __launch_bounds__(kFftMaxThreads, 4)
columns_kernel(const float2* __restrict__ in, Columns ci, float2* __restrict__ out, Columns co, int cols, int xtiles,
               const __grid_constant__ FftPlan p, int64_t tiles, int smem_tiles) {
    extern __shared__ float2 fft_smem[];
    const int n = p.n, tile = fft_tile_size(p);
    float2 *a = fft_smem, *b = a + tile, *tw = a + tile * smem_tiles;
    fft_roots<INV>(tw, n);
    for (int64_t t = blockIdx.x; t < tiles; t += gridDim.x) {
        const int64_t bi = t / xtiles;
        const int x0 = (int)(t - bi * xtiles) * kFftBatch;
        const ColumnRows rows_in{in + bi * ci.batch + x0, ci.row, ci.rows, cols - x0};
        const ColumnRowsOut rows_out{out + bi * co.batch + x0, co.row, co.rows, cols - x0};
        fft_run<INV, true>(Outside<ColumnRows>{rows_in, ci.off, n}, Outside<ColumnRowsOut>{rows_out, co.off, n}, a, b,
                           tw, p);
        __syncthreads();
    }
}

// Columns of a tile of two rows y (transform bit 2) and four columns x, of
// which `ys` and `xs` exist, in (z, y, x) planes `row` apart.
struct BrickColumns {
    const float2* src;
    int64_t row;
    int rows, stride, ys, xs;
    __device__ __forceinline__ int of(int c) const { return c; }
    __device__ __forceinline__ float2 get(int r, int c) const {
        return (r < rows && (c >> 2) < ys && (c & 3) < xs) ? __ldcs(src + r * row + (c >> 2) * stride + (c & 3))
                                                          : make_float2(0.f, 0.f);
    }
};
struct BrickColumnsOut {
    float2* dst;
    int64_t row;
    int rows, stride, ys, xs;
    __device__ __forceinline__ int of(int c) const { return c; }
    __device__ __forceinline__ void put(int r, int c, float2 v) const {
        if (r < rows && (c >> 2) < ys && (c & 3) < xs) dst[r * row + (c >> 2) * stride + (c & 3)] = v;
    }
};

// Bricks of the same columns: transform c's fftshifted sample z goes to slot
// (z & 1, c >> 2, c & 1) of brick (c >> 1) & 1 of the tile's pair, so the eight
// transforms of a sample fill two whole 32-byte sectors.  Bricks past the row's
// end are skipped; slots past an odd e get the zeros that absent columns load.
struct BricksOut {
    float2* dst;  // slot 0 of the pair's first brick at z = 0
    int plane, n, bricks;
    __device__ __forceinline__ int of(int c) const { return c; }
    __device__ __forceinline__ void put(int z, int c, float2 v) const {
        const int t = (c >> 1) & 1;
        if (t >= bricks) return;
        float2* o = dst + (int64_t)(z >> 1) * plane + t * 8 + (z & 1) * 4 + (c >> 2) * 2 + (c & 1);
        *o = v;
        if (z == n - 1 && !(z & 1)) o[4] = make_float2(0.f, 0.f);
    }
};

// z transforms of (d, e, stride) half spectra (y fftshifted) into the bricked copy
// of the fftshifted (e, e, wr) volume.  A tile is two rows y and four columns
// x.  Storing from the last pass instead of staging the results for 128-byte
// stores: 320^3 from 160 planes 99 -> 65 us.
__global__ void __launch_bounds__(kFftMaxThreads, 4)
columns_to_bricks_kernel(const float2* __restrict__ in, int rows, int off, float2* __restrict__ bricks, int wr,
                         int stride, int xtiles, const __grid_constant__ FftPlan p, int smem_tiles) {
    extern __shared__ float2 fft_smem[];
    const int n = p.n, bh = (n + 1) >> 1, bw = (wr + 1) >> 1, tile = fft_tile_size(p);
    float2 *a = fft_smem, *b = a + tile, *tw = a + tile * smem_tiles;
    fft_roots<false>(tw, n);
    const int by = blockIdx.x / xtiles, xt = blockIdx.x - by * xtiles;
    const BrickColumns cols{in + (int64_t)(2 * by) * stride + 4 * xt, (int64_t)n * stride, rows, stride, n - 2 * by,
                            wr - 4 * xt};
    const BricksOut out{bricks + ((int64_t)by * bw + 2 * xt) * 8, bh * bw * 8, n, bw - 2 * xt};
    // z (fftshifted) is sample (z + n - n / 2) mod n
    fft_run<false, true>(Outside<BrickColumns>{cols, off, n}, Outside<BricksOut>{out, n - n / 2, n}, a, b, tw, p);
}

// Insertion accumulators (float4 slots, fftshifted; BRICKED: accumulator_slot
// order) -> Friedel completion, division by max(weights, 1), inverse z
// transforms, planes (z + off) mod n of them: (rows, e, stride) with y fftshifted.
// One block per two rows y and four columns x of a channel (grid y); the
// weights are channel 0's.
template <bool BRICKED>
__global__ void __launch_bounds__(kFftMaxThreads, 4)
normalize_columns_kernel(const float4* __restrict__ acc, int64_t channel, float2* __restrict__ out, int rows, int off,
                         int wr, int stride, int xtiles, const __grid_constant__ FftPlan p) {
    extern __shared__ float2 fft_smem[];
    const int n = p.n, tile = fft_tile_size(p);
    float2 *a = fft_smem, *b = a + tile, *tw = b + tile;
    fft_roots<true>(tw, n);
    SliceGeom g{};  // accumulator_slot reads the volume dims only
    g.D = n;
    g.H = n;
    g.W = wr;
    const int by = blockIdx.x / xtiles, xt = blockIdx.x - by * xtiles;
    const float4* ch = acc + blockIdx.y * channel;
    const int shift = n - n / 2;
    const PlainTile<true> staged{b, n};
    {
        const int c = threadIdx.x & (kFftBatch - 1);
        const int y = 2 * by + (c >> 2), x = 4 * xt + (c & 3);
        auto slot = [&](int z, int yy, int xx) -> int64_t {
            return BRICKED ? accumulator_slot(g, z, yy, xx) : ((int64_t)z * n + yy) * wr + xx;
        };
        for (int z = threadIdx.x >> 3; z < n; z += blockDim.x >> 3) {
            float2 v = make_float2(0.f, 0.f);
            if (y < n && x < wr) {
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
            staged.at(k, c) = v;
        }
    }
    __syncthreads();
    const int64_t plane = (int64_t)n * stride;
    const BrickColumnsOut cols{out + blockIdx.y * rows * plane + (int64_t)(2 * by) * stride + 4 * xt, plane, rows, stride,
                               n - 2 * by, wr - 4 * xt};
    fft_run<true, true>(staged, Outside<BrickColumnsOut>{cols, off, n}, a, b, tw, p);
}

// ------------------------------------------------------------------ launches

// Shared memory of a kernel with `tiles` tiles (two where a pass, or a third
// factor, needs a second one).
static int fft_tiles(const FftPlan& p, bool staged) { return staged || p.passes > 2 ? 2 : 1; }

template <typename K>
static int fft_smem(K kernel, const FftPlan& p, int tiles, size_t& bytes) {
    bytes = fft_smem_bytes(p, tiles);
    if (bytes > 48 * 1024) {
        // always the same limit: a thread must not lower it between another one's call and launch
        cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kFftSmemLimit);
        if (e != cudaSuccess) return fail(TT_ERR_CUDA, "transform: shared memory: %s", cudaGetErrorString(e));
    }
    return TT_OK;
}

// Blocks for `tiles` tiles: up to four tiles a block, which share its roots of
// unity, as long as every SM keeps eight blocks.
static unsigned fft_blocks(int64_t tiles) {
    int64_t per = tiles / (148 * 8);
    per = per < 1 ? 1 : (per > 4 ? 4 : per);
    return (unsigned)((tiles + per - 1) / per);
}

static int row_tiles(const RowPairs& pairs, bool odd, int64_t& tiles) {
    const int64_t per = odd ? kFftBatch : 2 * kFftBatch;
    tiles = (pairs.count + per - 1) / per;
    if (tiles > 0x7fffffffLL || (odd && pairs.count > 0xffffffffLL))
        return fail(TT_ERR_INVALID, "transform: too many rows");
    return TT_OK;
}

// `images` times `rows` real rows of `len` samples.
static int launch_r2c(const float* in, float2* out, int64_t images, int64_t rows, int64_t len, int64_t off,
                      int64_t stride, float edge, float inner, const FftPlan& p, cudaStream_t st) {
    size_t sm;
    int64_t tiles;
    bool odd;
    const RowPairs pairs = make_row_pairs(images, rows, odd);
    const auto kernel = odd ? rows_r2c_kernel<true> : rows_r2c_kernel<false>;
    if (int e = fft_smem(kernel, p, 2, sm)) return e;
    if (int e = row_tiles(pairs, odd, tiles)) return e;
    kernel<<<fft_blocks(tiles), p.threads, sm, st>>>(in, out, pairs, (int)len, (int)(off % p.n), (int)stride, edge, inner,
                                                     p, tiles);
    return check_launch("rows_r2c_kernel");
}

static int launch_c2r(const float2* in, float* out, int64_t images, int64_t rows, int64_t len, int64_t off,
                      int64_t stride, float inner, float scale, const FftPlan& p, cudaStream_t st) {
    size_t sm;
    int64_t tiles;
    bool odd;
    const RowPairs pairs = make_row_pairs(images, rows, odd);
    const auto kernel = odd ? rows_c2r_kernel<true> : rows_c2r_kernel<false>;
    const int smem_tiles = fft_tiles(p, false);
    if (int e = fft_smem(kernel, p, smem_tiles, sm)) return e;
    if (int e = row_tiles(pairs, odd, tiles)) return e;
    kernel<<<fft_blocks(tiles), p.threads, sm, st>>>(in, out, pairs, (int)len, (int)(off % p.n), (int)stride, inner,
                                                     scale, p, tiles, smem_tiles);
    return check_launch("rows_c2r_kernel");
}

// Maps (channels, d, d, len) inside an (n, n, n2) array, times or over sinc^2.
template <bool DIV>
static int launch_sinc2(const float* in, float* out, int64_t channels, int64_t d, int64_t len, int64_t pad, int64_t n,
                        int64_t n2, cudaStream_t st) {
    const int64_t rows = channels * d * d, blocks = (rows + 7) / 8;
    if (blocks > 0x7fffffffLL) return fail(TT_ERR_INVALID, "transform: too many rows");
    sinc2_kernel<DIV><<<(unsigned)blocks, 256, 0, st>>>(in, out, rows, (int)d, (int)len, (int)pad, (int)n, (int)n2,
                                                       (float)(1.0 / (double)n), (float)(1.0 / (double)n2));
    return check_launch("sinc2_kernel");
}

template <bool INV>
static int launch_columns(const float2* in, Columns ci, float2* out, Columns co, int64_t batches, int cols,
                          const FftPlan& p, cudaStream_t st) {
    size_t sm;
    const int smem_tiles = fft_tiles(p, false);
    if (int e = fft_smem(columns_kernel<INV>, p, smem_tiles, sm)) return e;
    const int xtiles = (cols + kFftBatch - 1) / kFftBatch;
    const int64_t tiles = batches * xtiles;
    if (tiles > 0x7fffffffLL) return fail(TT_ERR_INVALID, "transform: too many columns");
    ci.off %= p.n;
    co.off %= p.n;
    columns_kernel<INV><<<fft_blocks(tiles), p.threads, sm, st>>>(in, ci, out, co, cols, xtiles, p, tiles, smem_tiles);
    return check_launch("columns_kernel");
}

// Plans of a padded box: e and, for the inverse real transforms, L = 2 (wr - 1).
// Half spectra that stay inside a call have rows of `row` >= wr bins, a
// multiple of eight: the 64-byte segments that the column kernels move then
// start on sector boundaries.
struct BoxPlans {
    int64_t d, p, e, wr, row, l, crop;  // crop = L - 2 p, the width of the cropped output
    FftPlan pe, pl;
};
static int64_t spectrum_row(int64_t wr) { return (wr + 7) / 8 * 8; }
static int make_box(int64_t d, int64_t pad, BoxPlans& b) {
    if (d < 1 || pad < 0 || d > kFftMaxLength || pad > kFftMaxLength)
        return fail(TT_ERR_INVALID, "transform: bad box");
    b.d = d;
    b.p = pad;
    b.e = d + 2 * pad;
    b.wr = b.e / 2 + 1;
    b.row = spectrum_row(b.wr);
    b.l = 2 * (b.wr - 1);
    b.crop = b.l - 2 * pad;
    if (!make_fft_plan(b.e, b.pe) || !make_fft_plan(b.l, b.pl) || b.crop < 1)
        return fail(TT_ERR_INVALID, "transform: box %lld padded to %lld is not supported", (long long)d,
                    (long long)b.e);
    return TT_OK;
}

int launch_extract_bricks(const void* bricks, int64_t channels, int64_t slots, const void* rot, float2* out,
                          const SliceGeom& g, cudaStream_t st);

}  // namespace tt

using namespace tt;

extern "C" int32_t tt_transform_supported(int64_t d, int64_t pad) {
    BoxPlans b;
    return make_box(d, pad, b) == TT_OK;
}

extern "C" int64_t tt_transform_row(int64_t d, int64_t pad) {
    return d < 1 || pad < 0 ? 0 : spectrum_row((d + 2 * pad) / 2 + 1);
}

extern "C" size_t tt_transform_workspace_bytes(int32_t kind, int64_t count, int64_t d, int64_t pad) {
    if (count < 0 || d < 1 || pad < 0) return 0;
    const int64_t e = d + 2 * pad, wr = e / 2 + 1, row = spectrum_row(wr);
    int64_t per = d * row;                       // images: the x spectra of d rows
    if (kind == 1) per = d * row * (d + e);      // volumes: x spectra of d^2 rows beside (d, e) rows
    if (kind == 2) per = (d + e) * row;          // projections: slices beside their d kept rows
    return (size_t)(count * per) * sizeof(float2);
}

static int check_transform(const void* in, const void* out, const void* workspace, size_t workspace_bytes,
                           int32_t kind, int64_t count, int64_t d, int64_t pad, BoxPlans& b, const char* what) {
    if (int e = make_box(d, pad, b)) return e;
    if (count < 0) return fail(TT_ERR_INVALID, "%s: negative count", what);
    if (!in || !out) return fail(TT_ERR_INVALID, "%s: NULL pointer argument", what);
    const size_t need = tt_transform_workspace_bytes(kind, count, d, pad);
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
    float2* xs = (float2*)workspace;               // (c, d, d, row)
    float2* ys = xs + channels * d * d * b.row;    // (c, d, e, row), first the weighted maps
    const int64_t at = pad + b.e / 2;              // fftshift(pad(v)): sample x at (x + at) mod e
    const int64_t shift = b.e - b.e / 2;           // fftshifted row r is bin (r + shift) mod e
    if (int e = launch_sinc2<false>(volumes, (float*)ys, channels, d, d, pad, b.e, b.e, st)) return e;
    if (int e = launch_r2c((const float*)ys, xs, channels, d * d, d, at, b.row, 1.f, 1.f, b.pe, st)) return e;
    if (int e = launch_columns<false>(xs, Columns{d * b.row, b.row, (int)d, (int)at}, ys,
                                      Columns{b.e * b.row, b.row, (int)b.e, (int)shift}, channels * d, (int)b.wr, b.pe,
                                      st))
        return e;
    size_t sm;
    const int smem_tiles = fft_tiles(b.pe, false);
    if (int e = fft_smem(columns_to_bricks_kernel, b.pe, smem_tiles, sm)) return e;
    const int xtiles = (int)((b.wr + 3) / 4), bh = (int)((b.e + 1) / 2);
    const int64_t slots = (int64_t)bh * bh * ((b.wr + 1) / 2) * 8;
    for (int64_t ch = 0; ch < channels; ch++) {
        columns_to_bricks_kernel<<<(unsigned)(bh * xtiles), b.pe.threads, sm, st>>>(
            ys + ch * d * b.e * b.row, (int)d, (int)(at % b.e), (float2*)bricks + ch * slots, (int)b.wr, (int)b.row,
            xtiles, b.pe, smem_tiles);
        if (int e = check_launch("columns_to_bricks_kernel")) return e;
    }
    return TT_OK;
}

extern "C" int tt_project_slices(const void* bricks, int64_t channels, const void* rotation_matrices, int64_t d,
                                 int64_t pad, float* images, void* workspace, size_t workspace_bytes,
                                 const tt_slice_params* p, void* stream) {
    if (int e = validate_params(p, true)) return e;
    if (channels < 1 || channels > 4096) return fail(TT_ERR_INVALID, "project_slices: channels must be in [1, 4096]");
    BoxPlans b;
    if (int e = check_transform(bricks, images, workspace, workspace_bytes, 2, p->n * channels, d, pad, b,
                                "project_slices"))
        return e;
    if (p->img_d != b.e || p->img_h != b.e || p->img_w != b.e || p->vol_d != b.e || p->vol_h != b.e ||
        p->vol_w != b.wr || p->volume_layout != TT_VOLUME_BRICKS || p->volume_unshifted || p->slices_unshifted)
        return fail(TT_ERR_INVALID, "project_slices: the params are not those of a bricked padded box");
    if (p->n == 0) return TT_OK;
    if (!rotation_matrices) return fail(TT_ERR_INVALID, "project_slices: NULL pointer argument");
    SliceGeom g = make_geom(*p);
    g.slice_rows = (int)(channels * b.e);
    g.slice_pitch = (int)b.row;
    cudaStream_t st = as_stream(stream);
    const int64_t count = p->n * channels, half = (b.e + 1) / 2, slots = half * half * ((b.wr + 1) / 2) * 8;
    float2* cs = (float2*)workspace;          // (n, c, d, row)
    float2* slices = cs + count * d * b.row;  // (n, c, e, row)
    if (int e = launch_extract_bricks(bricks, channels, slots, rotation_matrices, slices, g, st)) return e;
    if (int e = launch_columns<true>(slices, Columns{b.e * b.row, b.row, (int)b.e, (int)(b.e - b.e / 2)}, cs,
                                     Columns{d * b.row, b.row, (int)d, (int)(pad + b.e / 2)}, count, (int)b.wr, b.pe,
                                     st))
        return e;
    return launch_c2r(cs, images, count, d, b.crop, pad + b.l / 2, b.row, 1.f,
                      (float)(1.0 / ((double)b.e * (double)b.l)), b.pl, st);
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
    if (int e = launch_r2c(grad_images, cs, count, d, b.crop, pad + b.l / 2, b.row, f, 2.f * f, b.pl, st)) return e;
    return launch_columns<false>(cs, Columns{d * b.row, b.row, (int)d, (int)(pad + b.e / 2)}, (float2*)grad_slices,
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
    float2* xs = (float2*)workspace;             // (c, d, d, row)
    float2* zs = xs + channels * d * d * b.row;  // (c, d, e, row)
    const int64_t at = pad + b.e / 2, shift = b.e - b.e / 2, plane = b.e * b.wr, zplane = b.e * b.row;
    for (int64_t ch = 0; ch < channels; ch++)  // along z, one batch per row y
        if (int e = launch_columns<true>((const float2*)grad_dft + ch * b.e * plane,
                                         Columns{b.wr, plane, (int)b.e, (int)shift}, zs + ch * d * zplane,
                                         Columns{b.row, zplane, (int)d, (int)at}, b.e, (int)b.wr, b.pe, st))
            return e;
    if (int e = launch_columns<true>(zs, Columns{zplane, b.row, (int)b.e, (int)shift}, xs,
                                     Columns{d * b.row, b.row, (int)d, (int)at}, channels * d, (int)b.wr, b.pe, st))
        return e;
    // adjoint of the real transform: the real part of the half spectrum's inverse, mates not doubled
    if (int e = launch_c2r(xs, grad_volumes, channels, d * d, d, at, b.row, 0.5f, 1.f, b.pe, st)) return e;
    return launch_sinc2<false>(grad_volumes, grad_volumes, channels, d, d, pad, b.e, b.e, st);
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
    if (int e = launch_r2c(images, xs, count, d, d, at, b.row, 1.f, 1.f, b.pe, st)) return e;
    return launch_columns<false>(xs, Columns{d * b.row, b.row, (int)d, (int)at}, (float2*)slices,
                                 Columns{b.e * b.row, b.row, (int)b.e, (int)(b.e - b.e / 2)}, count, (int)b.wr, b.pe, st);
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
    float2* xs = (float2*)workspace;             // (c, d, d, row)
    float2* zs = xs + channels * d * d * b.row;  // (c, d, e, row)
    const int64_t at = pad + b.e / 2, zplane = b.e * b.row, half = (b.e + 1) / 2;
    const int xtiles = (int)((b.wr + 3) / 4);
    const dim3 grid((unsigned)(half * xtiles), (unsigned)channels);
    size_t sm;
    if (bricked) {
        if (int e = fft_smem(normalize_columns_kernel<true>, b.pe, 2, sm)) return e;
        normalize_columns_kernel<true><<<grid, b.pe.threads, sm, st>>>(
            (const float4*)accumulator, half * half * ((b.wr + 1) / 2) * 8, zs, (int)d, (int)(at % b.e), (int)b.wr,
            (int)b.row, xtiles, b.pe);
    } else {
        if (int e = fft_smem(normalize_columns_kernel<false>, b.pe, 2, sm)) return e;
        normalize_columns_kernel<false><<<grid, b.pe.threads, sm, st>>>((const float4*)accumulator, b.e * b.e * b.wr, zs,
                                                                        (int)d, (int)(at % b.e), (int)b.wr,
                                                                        (int)b.row, xtiles, b.pe);
    }
    if (int e = check_launch("normalize_columns_kernel")) return e;
    if (int e = launch_columns<true>(zs, Columns{zplane, b.row, (int)b.e, (int)(b.e - b.e / 2)}, xs,
                                     Columns{d * b.row, b.row, (int)d, (int)at}, channels * d, (int)b.wr, b.pe, st))
        return e;
    const double scale = 1.0 / ((double)b.e * (double)b.e * (double)b.l);
    if (int e = launch_c2r(xs, volumes, channels, d * d, b.crop, pad + b.l / 2, b.row, 1.f, (float)scale, b.pl, st))
        return e;
    return launch_sinc2<true>(volumes, volumes, channels, d, b.crop, pad, b.e, b.l, st);
}
