// Batched 1D Fourier transforms in shared memory, eight at a time per block.
//
// The real-space wrappers pad their inputs to about twice the size and crop
// their outputs, and every pass of a library transform over the padded arrays
// moves the zeros and the cropped samples through HBM, with separate passes
// for the padding, the shifts, the scaling and the layout.  The kernels built
// on this file (fft.cu) read only the rows that hold data, write only the rows
// that are kept, and apply shifts, weights, the slice sampling and the volume
// layout in their loads and stores.
//
// A block holds eight transforms of length n in a [sample][transform] tile
// (64-byte rows) and its ping-pong copy: Stockham passes, radix 8, 4, 2, then
// 3, 5, 7, 11, 13, one butterfly of one transform per thread and step.
// Consecutive threads take the eight transforms of one sample, so the tile's
// loads are contiguous; the twiddles are a table of the n-th roots of unity
// computed once per block.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace tt {

constexpr int kFftBatch = 8;          // transforms per block
constexpr int kFftMaxLength = 1024;   // two tiles of 64 KB
constexpr int kFftMaxPasses = 10;

struct FftPlan {
    int n;
    int passes;
    int radix[kFftMaxPasses];
    int ns[kFftMaxPasses];           // product of the earlier radices
    uint32_t inv_ns[kFftMaxPasses];  // floor(2^20 / ns) + 1: j / ns = j * inv_ns >> 20 for j * ns < 2^20
    int step[kFftMaxPasses];         // n / (ns * radix): root stride of the pass
};

// Plan of length n; false when n has a prime factor above 13 or is out of range.
inline bool make_fft_plan(int64_t n, FftPlan& p) {
    if (n < 2 || n > kFftMaxLength) return false;
    p.n = (int)n;
    p.passes = 0;
    int m = (int)n, twos = 0, ns = 1;
    auto add = [&](int r) {
        const int i = p.passes++;
        p.radix[i] = r;
        p.ns[i] = ns;
        p.inv_ns[i] = (1u << 20) / (uint32_t)ns + 1;
        p.step[i] = (int)n / (ns * r);
        ns *= r;
    };
    while (m % 2 == 0) {
        m /= 2;
        twos++;
    }
    int fours = twos % 3 == 0 ? 0 : (twos % 3 == 2 ? 1 : (twos >= 4 ? 2 : 0));
    for (int k = 0; k < (twos - 2 * fours) / 3; k++) add(8);
    for (int k = 0; k < fours; k++) add(4);
    if (twos == 1) add(2);
    for (int r : {13, 11, 7, 5, 3})
        while (m % r == 0) {
            add(r);
            m /= r;
        }
    return m == 1;
}

inline size_t fft_smem_bytes(int n) { return (size_t)n * (2 * kFftBatch + 1) * sizeof(float2); }

// One thread per sample of a transform, in whole warps.
inline int fft_threads(int n) {
    const int t = (n + 31) / 32 * 32;
    return t < 64 ? 64 : (t > 512 ? 512 : t);
}

__device__ __forceinline__ float2 cadd(float2 a, float2 b) { return make_float2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ float2 csub(float2 a, float2 b) { return make_float2(a.x - b.x, a.y - b.y); }
__device__ __forceinline__ float2 cmul(float2 a, float2 b) {
    return make_float2(fmaf(a.x, b.x, -a.y * b.y), fmaf(a.x, b.y, a.y * b.x));
}

// exp(-2 pi i t / n), 0 <= t < n: reduced to the first octant in integers, so
// the angle handed to sincospi is small and accurate.
__device__ __forceinline__ float2 unit_root(int t, int n) {
    const int q = (4 * t) / n, r = 4 * t - q * n;  // quarter turns and the rest, r / (4 n) of a turn
    const bool far = 2 * r > n;
    float s, c;
    sincospif((float)(far ? n - r : r) / (float)(2 * n), &s, &c);
    if (far) {
        const float x = s;
        s = c;
        c = x;
    }
    // (c, s) at angle q * pi / 2 + the rest, conjugated
    switch (q) {
        case 0: return make_float2(c, -s);
        case 1: return make_float2(-s, -c);
        case 2: return make_float2(-c, s);
        default: return make_float2(s, c);
    }
}

__device__ __forceinline__ void fft_roots(float2* tw, int n) {
    for (int t = threadIdx.x; t < n; t += blockDim.x) tw[t] = unit_root(t, n);
}

// Tile address of sample k of transform c.  SWZ (tiles that are filled or read
// along k): the transforms of a sample are permuted so that sixteen
// consecutive samples of one transform lie in different banks.
template <bool SWZ>
__device__ __forceinline__ int fft_at(int k, int c) {
    return k * kFftBatch + (SWZ ? (c ^ ((k >> 1) & 7)) : c);
}

// cos and sin of 2 pi k / R, 0 < k <= R / 2 (k folds to a constant in unrolled code).
template <int R>
__device__ __forceinline__ float root_cos(int k) {
    switch (R) {
        case 3: return -0.5f;
        case 5: return k == 1 ? 0.30901699437494745f : -0.80901699437494734f;
        case 7: return k == 1 ? 0.62348980185873359f : (k == 2 ? -0.22252093395631434f : -0.90096886790241903f);
        case 11:
            return k == 1   ? 0.84125353283118121f
                   : k == 2 ? 0.41541501300188644f
                   : k == 3 ? -0.142314838273285f
                   : k == 4 ? -0.65486073394528499f
                            : -0.95949297361449737f;
        default:
            return k == 1   ? 0.88545602565320991f
                   : k == 2 ? 0.56806474673115592f
                   : k == 3 ? 0.12053668025532301f
                   : k == 4 ? -0.35460488704253545f
                   : k == 5 ? -0.74851074817110119f
                            : -0.97094181742605201f;
    }
}
template <int R>
__device__ __forceinline__ float root_sin(int k) {
    switch (R) {
        case 3: return 0.86602540378443865f;
        case 5: return k == 1 ? 0.95105651629515353f : 0.58778525229247325f;
        case 7: return k == 1 ? 0.7818314824680298f : (k == 2 ? 0.97492791218182362f : 0.43388373911755823f);
        case 11:
            return k == 1   ? 0.54064081745559756f
                   : k == 2 ? 0.90963199535451833f
                   : k == 3 ? 0.9898214418809328f
                   : k == 4 ? 0.75574957435425827f
                            : 0.28173255684142967f;
        default:
            return k == 1   ? 0.46472317204376851f
                   : k == 2 ? 0.82298386589365635f
                   : k == 3 ? 0.99270887409805397f
                   : k == 4 ? 0.93501624268541483f
                   : k == 5 ? 0.66312265824079519f
                            : 0.23931566428755768f;
    }
}

// Multiplication by -i (forward) or +i (inverse).
template <bool INV>
__device__ __forceinline__ float2 turn(float2 a) {
    return INV ? make_float2(-a.y, a.x) : make_float2(a.y, -a.x);
}

// In-register transform of R samples, R odd: pairs (m, R - m) by their sums
// and differences.
template <int R, bool INV>
struct Dft {
    static __device__ __forceinline__ void run(float2 v[R]) {
        constexpr int H = (R - 1) / 2;
        float2 t[H], u[H], x0 = v[0];
#pragma unroll
        for (int m = 1; m <= H; m++) {
            t[m - 1] = cadd(v[m], v[R - m]);
            u[m - 1] = csub(v[m], v[R - m]);
            x0 = cadd(x0, t[m - 1]);
        }
        float2 y[R];
        y[0] = x0;
#pragma unroll
        for (int q = 1; q <= H; q++) {
            float2 a = v[0], b = make_float2(0.f, 0.f);
#pragma unroll
            for (int m = 1; m <= H; m++) {
                const int k = (q * m) % R, f = k <= H ? k : R - k;
                const float c = root_cos<R>(f), s = k <= H ? root_sin<R>(f) : -root_sin<R>(f);
                a.x = fmaf(c, t[m - 1].x, a.x);
                a.y = fmaf(c, t[m - 1].y, a.y);
                b.x = fmaf(s, u[m - 1].x, b.x);
                b.y = fmaf(s, u[m - 1].y, b.y);
            }
            const float2 w = turn<INV>(b);
            y[q] = cadd(a, w);
            y[R - q] = csub(a, w);
        }
#pragma unroll
        for (int q = 0; q < R; q++) v[q] = y[q];
    }
};
template <bool INV>
struct Dft<2, INV> {
    static __device__ __forceinline__ void run(float2 v[2]) {
        const float2 a = v[0];
        v[0] = cadd(a, v[1]);
        v[1] = csub(a, v[1]);
    }
};
template <bool INV>
struct Dft<4, INV> {
    static __device__ __forceinline__ void run(float2 v[4]) {
        const float2 a = cadd(v[0], v[2]), b = csub(v[0], v[2]), c = cadd(v[1], v[3]);
        const float2 d = turn<INV>(csub(v[1], v[3]));
        v[0] = cadd(a, c);
        v[1] = cadd(b, d);
        v[2] = csub(a, c);
        v[3] = csub(b, d);
    }
};
template <bool INV>
struct Dft<8, INV> {
    static __device__ __forceinline__ void run(float2 v[8]) {
        float2 e[4] = {v[0], v[2], v[4], v[6]}, o[4] = {v[1], v[3], v[5], v[7]};
        Dft<4, INV>::run(e);
        Dft<4, INV>::run(o);
        constexpr float h = 0.70710678118654752f;
        const float2 w1 = make_float2(h, INV ? h : -h), w3 = make_float2(-h, INV ? h : -h);
        o[1] = cmul(o[1], w1);
        o[2] = turn<INV>(o[2]);
        o[3] = cmul(o[3], w3);
#pragma unroll
        for (int k = 0; k < 4; k++) {
            v[k] = cadd(e[k], o[k]);
            v[k + 4] = csub(e[k], o[k]);
        }
    }
};

// One Stockham pass of radix R from tile a to tile b.
template <int R, bool INV, bool SWZ>
__device__ __forceinline__ void fft_pass(const float2* a, float2* b, const float2* tw, int n, int ns, uint32_t inv_ns,
                                         int step) {
    const int nb = n / R;
    for (int i = threadIdx.x; i < nb * kFftBatch; i += blockDim.x) {
        const int c = i & (kFftBatch - 1), j = i >> 3;
        const int k = j - (int)(((uint32_t)j * inv_ns) >> 20) * ns;
        float2 v[R];
#pragma unroll
        for (int r = 0; r < R; r++) v[r] = a[fft_at<SWZ>(j + r * nb, c)];
        if (ns > 1) {
#pragma unroll
            for (int r = 1; r < R; r++) {
                float2 w = tw[r * k * step];
                if (INV) w.y = -w.y;
                v[r] = cmul(v[r], w);
            }
        }
        Dft<R, INV>::run(v);
        const int o = (j - k) * R + k;
#pragma unroll
        for (int r = 0; r < R; r++) b[fft_at<SWZ>(o + r * ns, c)] = v[r];
    }
    __syncthreads();
}

// Transforms the tile (the block's eight transforms; a barrier precedes the
// call) with the exponent's sign - (+ when INV), unscaled; returns the tile
// that holds the result.
template <bool INV, bool SWZ>
__device__ __forceinline__ float2* fft_run(float2* a, float2* b, const float2* tw, const FftPlan& p) {
    for (int s = 0; s < p.passes; s++) {
        switch (p.radix[s]) {
            case 8: fft_pass<8, INV, SWZ>(a, b, tw, p.n, p.ns[s], p.inv_ns[s], p.step[s]); break;
            case 4: fft_pass<4, INV, SWZ>(a, b, tw, p.n, p.ns[s], p.inv_ns[s], p.step[s]); break;
            case 2: fft_pass<2, INV, SWZ>(a, b, tw, p.n, p.ns[s], p.inv_ns[s], p.step[s]); break;
            case 3: fft_pass<3, INV, SWZ>(a, b, tw, p.n, p.ns[s], p.inv_ns[s], p.step[s]); break;
            case 5: fft_pass<5, INV, SWZ>(a, b, tw, p.n, p.ns[s], p.inv_ns[s], p.step[s]); break;
            case 7: fft_pass<7, INV, SWZ>(a, b, tw, p.n, p.ns[s], p.inv_ns[s], p.step[s]); break;
            case 11: fft_pass<11, INV, SWZ>(a, b, tw, p.n, p.ns[s], p.inv_ns[s], p.step[s]); break;
            default: fft_pass<13, INV, SWZ>(a, b, tw, p.n, p.ns[s], p.inv_ns[s], p.step[s]); break;
        }
        float2* t = a;
        a = b;
        b = t;
    }
    return a;
}

}  // namespace tt
