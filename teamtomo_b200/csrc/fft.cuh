// Batched 1D Fourier transforms, eight per block, for the kernels of fft.cu.
//
// The real-space wrappers pad their inputs to about twice the size and crop
// their outputs, and every pass of a library transform over the padded arrays
// moves the zeros and the cropped samples through HBM, with separate passes
// for the padding, the shifts, the scaling and the layout.  The kernels built
// on this file read only the rows that hold data, write only the rows that are
// kept, and apply shifts, weights, the slice sampling and the volume layout in
// their loads and stores.
//
// A length n is split into two to four factors of at most 20 (256 = 16 x 16,
// 320 = 16 x 20, 180 = 12 x 15).  A thread transforms one factor's samples in
// registers (a Stockham pass); the passes exchange samples through shared
// memory, so a two-factor length crosses it once, and the first pass can load
// from and the last store to global memory directly (figures in fft.cu).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace tt {

constexpr int kFftBatch = 8;          // transforms per block
constexpr int kFftMaxLength = 1024;
constexpr int kFftMaxPasses = 4;
constexpr int kFftMaxThreads = 256;

struct FftPlan {
    int n;
    int passes;
    int threads;                     // block size: the widest pass's butterflies, in whole warps
    int radix[kFftMaxPasses];
    int ns[kFftMaxPasses];           // product of the earlier factors
    uint32_t inv_ns[kFftMaxPasses];  // floor(2^20 / ns) + 1: j / ns = j * inv_ns >> 20 for j * ns < 2^20
    uint32_t inv_nb[kFftMaxPasses];  // the same for n / radix, used for i < 8 n / radix: i * nb < 2^20
    int step[kFftMaxPasses];         // n / (ns * radix): root stride of the pass
    int pitched;                     // samples of one transform in the pitched order (padding included)
};

constexpr int kFftRadices[] = {20, 16, 15, 14, 13, 12, 11, 10, 9, 8, 7, 6, 5, 4, 3, 2};

// Fewest factors first, then the smallest largest factor; at least two.
inline bool split_length(int n, int passes, int cap, int* out) {
    if (passes == 0) return n == 1;
    for (int r : kFftRadices) {
        if (r > cap || n % r) continue;
        out[0] = r;
        if (split_length(n / r, passes - 1, r, out + 1)) return true;
    }
    return false;
}

// Plan of length n; false when n is not a product of two to four factors in
// range (a prime factor above 13, a prime, n > 1024).
inline bool make_fft_plan(int64_t n, FftPlan& p) {
    if (n < 4 || n > kFftMaxLength) return false;
    p.n = (int)n;
    p.passes = 0;
    int f[kFftMaxPasses];
    for (int k = 2; k <= kFftMaxPasses && !p.passes; k++)
        for (int cap = 2; cap <= 20; cap++)
            if (split_length((int)n, k, cap, f)) {
                p.passes = k;
                break;
            }
    if (!p.passes) return false;
    int ns = 1, widest = 0;
    for (int i = 0; i < p.passes; i++) {
        const int nb = (int)n / f[i];
        p.radix[i] = f[i];
        p.ns[i] = ns;
        p.inv_ns[i] = (1u << 20) / (uint32_t)ns + 1;
        p.inv_nb[i] = (1u << 20) / (uint32_t)nb + 1;
        p.step[i] = (int)n / (ns * f[i]);
        ns *= f[i];
        widest = nb > widest ? nb : widest;
    }
    p.pitched = (int)n / f[0] * (f[0] | 1);
    const int t = (widest * kFftBatch + 31) / 32 * 32;
    p.threads = t < 64 ? 64 : (t > kFftMaxThreads ? kFftMaxThreads : t);
    return true;
}

// Tiles hold eight transforms, [sample][transform] (COLUMNS) or
// [transform][sample].  Staged samples are in natural order; between passes
// sample i sits at (i / R) * (R | 1) + i % R, R the first factor, so that the
// first pass's stores, R apart, fall on different banks and every later access
// of a butterfly is one base and one stride.
__device__ __forceinline__ int fft_tile_size(const FftPlan& p) { return p.pitched * kFftBatch; }

// Shared memory: `tiles` tiles and the roots of unity.
inline size_t fft_smem_bytes(const FftPlan& p, int tiles) {
    return ((size_t)p.pitched * kFftBatch * tiles + p.n) * sizeof(float2);
}
constexpr int kFftSmemLimit = 227 * 1024;  // a block's most; two tiles of 1000 samples take 145 KB

// Both components in one instruction: the transforms are bound by issue slots
// (65 %).  With the column passes' twiddles from memory: columns of 800 x 320^2
// 138 -> 131 us, 320^3 from 160 planes 67 -> 65 us.
__device__ __forceinline__ float2 cadd(float2 a, float2 b) {
    float2 r;
    asm("{ .reg .b64 a, b, d; mov.b64 a, {%2, %3}; mov.b64 b, {%4, %5}; add.rn.f32x2 d, a, b; mov.b64 {%0, %1}, d; }"
        : "=f"(r.x), "=f"(r.y)
        : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
    return r;
}
__device__ __forceinline__ float2 csub(float2 a, float2 b) {
    float2 r;
    asm("{ .reg .b64 a, b, d; mov.b64 a, {%2, %3}; mov.b64 b, {%4, %5}; sub.rn.f32x2 d, a, b; mov.b64 {%0, %1}, d; }"
        : "=f"(r.x), "=f"(r.y)
        : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
    return r;
}
// a + t and a - t for a t whose components were swapped (turn): one by one, as a
// pair they would have to be moved first.
__device__ __forceinline__ float2 cadd1(float2 a, float2 t) { return make_float2(a.x + t.x, a.y + t.y); }
__device__ __forceinline__ float2 csub1(float2 a, float2 t) { return make_float2(a.x - t.x, a.y - t.y); }
__device__ __forceinline__ float2 cmul(float2 a, float2 b) {
    return make_float2(fmaf(a.x, b.x, -a.y * b.y), fmaf(a.x, b.y, a.y * b.x));
}

// exp(-2 pi i t / n) (+ when INV), 0 <= t < n: reduced to the first octant in
// integers, so the angle handed to sincospi is small and accurate.
template <bool INV>
__device__ __forceinline__ float2 unit_root(int t, int n) {
    const int q = (4 * t >= n) + (2 * t >= n) + (4 * t >= 3 * n);  // quarter turns
    const int r = 4 * t - q * n;                                   // and the rest, r / (4 n) of a turn
    const bool far = 2 * r > n;
    float s, c;
    sincospif((float)(far ? n - r : r) / (float)(2 * n), &s, &c);
    float2 w = far ? make_float2(s, c) : make_float2(c, s);
    if (q & 1) w = make_float2(-w.y, w.x);
    if (q & 2) w = make_float2(-w.x, -w.y);
    return INV ? w : make_float2(w.x, -w.y);
}

template <bool INV>
__device__ __forceinline__ void fft_roots(float2* tw, int n) {
    for (int t = threadIdx.x; t < n; t += blockDim.x) tw[t] = unit_root<INV>(t, n);
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

// ---- transforms of R samples in registers

// R an odd prime: pairs (m, R - m) by their sums and differences.
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
            y[q] = cadd1(a, w);
            y[R - q] = csub1(a, w);
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
        v[1] = cadd1(b, d);
        v[2] = csub(a, c);
        v[3] = csub1(b, d);
    }
};

// R = A * B: A transforms of B samples (stride A), twiddles W(a * q), B
// transforms of A samples.  W(k) multiplies by exp(-+2 pi i k / R).
template <int A, int B, bool INV, class W>
__device__ __forceinline__ void dft_split(float2 v[A * B], W twiddle) {
    float2 t[A][B];
#pragma unroll
    for (int a = 0; a < A; a++) {
#pragma unroll
        for (int b = 0; b < B; b++) t[a][b] = v[a + A * b];
        Dft<B, INV>::run(t[a]);
#pragma unroll
        for (int q = 1; q < B; q++)
            if (a) t[a][q] = twiddle(t[a][q], a * q);
    }
#pragma unroll
    for (int q = 0; q < B; q++) {
        float2 u[A];
#pragma unroll
        for (int a = 0; a < A; a++) u[a] = t[a][q];
        Dft<A, INV>::run(u);
#pragma unroll
        for (int a = 0; a < A; a++) v[q + B * a] = u[a];
    }
}
template <bool INV>
__device__ __forceinline__ float2 by_root(float2 x, float c, float s) {  // exp(-+i angle) from its cos and sin
    return cmul(x, make_float2(c, INV ? s : -s));
}
template <bool INV>
struct Dft<8, INV> {
    static __device__ __forceinline__ void run(float2 v[8]) {
        constexpr float h = 0.70710678118654752f;
        dft_split<2, 4, INV>(v, [](float2 x, int k) {
            return k == 1 ? by_root<INV>(x, h, h) : (k == 2 ? turn<INV>(x) : by_root<INV>(x, -h, h));
        });
    }
};
template <bool INV>
struct Dft<9, INV> {
    static __device__ __forceinline__ void run(float2 v[9]) {
        dft_split<3, 3, INV>(v, [](float2 x, int k) {
            return k == 1   ? by_root<INV>(x, 0.76604444311897804f, 0.64278760968653933f)
                   : k == 2 ? by_root<INV>(x, 0.17364817766693035f, 0.98480775301220806f)
                            : by_root<INV>(x, -0.93969262078590838f, 0.34202014332566873f);  // k == 4
        });
    }
};
template <bool INV>
struct Dft<16, INV> {
    static __device__ __forceinline__ void run(float2 v[16]) {
        constexpr float h = 0.70710678118654752f, c = 0.92387953251128674f, s = 0.38268343236508977f;
        dft_split<4, 4, INV>(v, [](float2 x, int k) {
            return k == 1   ? by_root<INV>(x, c, s)
                   : k == 2 ? by_root<INV>(x, h, h)
                   : k == 3 ? by_root<INV>(x, s, c)
                   : k == 4 ? turn<INV>(x)
                   : k == 6 ? by_root<INV>(x, -h, h)
                            : by_root<INV>(x, -c, -s);  // k == 9
        });
    }
};

// R = A * B, A and B coprime: sample (B a + A b) mod R, bin k with k = p mod A,
// k = q mod B; a two-dimensional transform without twiddles.
template <int A, int B, bool INV>
struct DftCoprime {
    static __host__ __device__ constexpr int inverse(int x, int m) {
        for (int i = 1; i < m; i++)
            if (x * i % m == 1) return i;
        return 0;
    }
    static __device__ __forceinline__ void run(float2 v[A * B]) {
        constexpr int R = A * B, PA = B * inverse(B % A, A), PB = A * inverse(A % B, B);
        float2 t[A][B];
#pragma unroll
        for (int a = 0; a < A; a++) {
#pragma unroll
            for (int b = 0; b < B; b++) t[a][b] = v[(B * a + A * b) % R];
            Dft<B, INV>::run(t[a]);
        }
#pragma unroll
        for (int q = 0; q < B; q++) {
            float2 u[A];
#pragma unroll
            for (int a = 0; a < A; a++) u[a] = t[a][q];
            Dft<A, INV>::run(u);
#pragma unroll
            for (int p = 0; p < A; p++) v[(PA * p + PB * q) % R] = u[p];
        }
    }
};
template <bool INV>
struct Dft<6, INV> : DftCoprime<2, 3, INV> {};
template <bool INV>
struct Dft<10, INV> : DftCoprime<2, 5, INV> {};
template <bool INV>
struct Dft<12, INV> : DftCoprime<4, 3, INV> {};
template <bool INV>
struct Dft<14, INV> : DftCoprime<2, 7, INV> {};
template <bool INV>
struct Dft<15, INV> : DftCoprime<3, 5, INV> {};
template <bool INV>
struct Dft<20, INV> : DftCoprime<4, 5, INV> {};

// ---- passes
//
// A pass reads butterfly j's samples j + r * nb (nb = n / R) from a source and
// writes results o + r * ns to a destination.  Sources and destinations give a
// cursor for one butterfly, then take r (and, to read, the radix).

// A tile in natural order.
template <bool COLUMNS>
struct PlainTile {
    float2* t;
    int n;
    __device__ __forceinline__ float2& at(int k, int c) const { return t[COLUMNS ? k * kFftBatch + c : c * n + k]; }
    struct Cursor {
        float2* t;
        int step;
        __device__ __forceinline__ float2 get(int r, int) const { return t[r * step]; }
        __device__ __forceinline__ void put(int r, float2 v) const { t[r * step] = v; }
    };
    __device__ __forceinline__ Cursor from(int j, int c, int nb, const FftPlan&) const {
        return Cursor{&at(j, c), COLUMNS ? nb * kFftBatch : nb};
    }
    __device__ __forceinline__ Cursor to(int j, int k, int c, int, const FftPlan& p, int s) const {
        return Cursor{&at((j - k) * p.radix[s] + k, c), COLUMNS ? p.ns[s] * kFftBatch : p.ns[s]};
    }
};

// A tile in the pitched order, between passes.
template <bool COLUMNS>
struct PitchedTile {
    float2* t;
    using Cursor = typename PlainTile<COLUMNS>::Cursor;
    __device__ __forceinline__ float2* at(int pos, int c, const FftPlan& p) const {
        return t + (COLUMNS ? pos * kFftBatch + c : c * p.pitched + pos);
    }
    // every pass after the first: nb and ns are multiples of the first factor
    __device__ __forceinline__ Cursor from(int j, int c, int nb, const FftPlan& p) const {
        const int R = p.radix[0], pitch = R | 1, q = (int)(((uint32_t)j * p.inv_ns[1]) >> 20);
        const int rows = (int)(((uint32_t)nb * p.inv_ns[1]) >> 20);
        return Cursor{at(q * pitch + j - q * R, c, p), rows * pitch * (COLUMNS ? kFftBatch : 1)};
    }
    __device__ __forceinline__ Cursor to(int j, int k, int c, int R, const FftPlan& p, int s) const {
        const int pitch = p.radix[0] | 1;
        if (s == 0) return Cursor{at(j * pitch, c, p), COLUMNS ? kFftBatch : 1};
        // results (j - k) * R + k + r * ns
        const int first = (j - k) * R + k, q = (int)(((uint32_t)first * p.inv_ns[1]) >> 20);
        const int rows = (int)(((uint32_t)p.ns[s] * p.inv_ns[1]) >> 20);
        return Cursor{at(q * pitch + first - q * p.radix[0], c, p), rows * pitch * (COLUMNS ? kFftBatch : 1)};
    }
};

// Global memory: f.get(x, f.of(c)) / f.put(x, f.of(c), v) with x = (sample -
// off) mod n, the row or column behind a sample; of(c) is what f keeps of a
// transform for a whole butterfly (its index, or more).
template <class F>
struct Outside {
    const F& f;
    int off, n;
    struct Cursor {
        const F& f;
        int x, step, n;
        decltype(f.of(0)) c;
        __device__ __forceinline__ int where(int r) const {
            const int y = x + r * step;  // in [0, 2 n)
            return (int)min((unsigned)y, (unsigned)(y - n));
        }
        __device__ __forceinline__ float2 get(int r, int) const { return f.get(where(r), c); }
        __device__ __forceinline__ void put(int r, float2 v) const { f.put(where(r), c, v); }
    };
    __device__ __forceinline__ int back(int k) const {
        const int x = k - off;
        return x < 0 ? x + n : x;
    }
    __device__ __forceinline__ Cursor from(int j, int c, int nb, const FftPlan&) const {
        return Cursor{f, back(j), nb, n, f.of(c)};
    }
    __device__ __forceinline__ Cursor to(int j, int k, int c, int R, const FftPlan& p, int s) const {
        return Cursor{f, back((j - k) * R + k), p.ns[s], n, f.of(c)};
    }
};

// One Stockham pass of radix R.  Consecutive threads take the eight transforms
// of one butterfly (COLUMNS) or consecutive butterflies of one transform.
// Twiddles are read by the column passes (four addresses a warp).  In the row
// passes, where they would conflict, the roots of powers r = 1, 2, 4, .. are read
// and the others are products of at most four of them.
template <int R, bool INV, bool COLUMNS, bool FIRST, class Src, class Dst>
__device__ __forceinline__ void fft_pass(const Src& src, const Dst& dst, const float2* tw, const FftPlan& p, int s) {
    const int nb = p.n / R, ns = FIRST ? 1 : p.ns[s];
    for (int i = threadIdx.x; i < nb * kFftBatch; i += blockDim.x) {
        const int c = COLUMNS ? i & (kFftBatch - 1) : (int)(((uint32_t)i * p.inv_nb[s]) >> 20);
        const int j = COLUMNS ? i >> 3 : i - c * nb;
        const int k = FIRST ? 0 : j - (int)(((uint32_t)j * p.inv_ns[s]) >> 20) * ns;
        float2 v[R];
        const auto in = src.from(j, c, nb, p);
#pragma unroll
        for (int r = 0; r < R; r++) v[r] = in.get(r, R);
        if constexpr (!FIRST) {
            float2 w[R];
            const int at = k * p.step[s];
#pragma unroll
            for (int r = 1; r < R; r++) {
                const int top = COLUMNS ? r : r >= 16 ? 16 : (r >= 8 ? 8 : (r >= 4 ? 4 : (r >= 2 ? 2 : 1)));
                w[r] = r == top ? tw[r * at] : cmul(w[top], w[r - top]);
                v[r] = cmul(v[r], w[r]);
            }
        }
        Dft<R, INV>::run(v);
        const auto out = dst.to(j, k, c, R, p, FIRST ? 0 : s);
#pragma unroll
        for (int r = 0; r < R; r++) out.put(r, v[r]);
    }
}

template <bool INV, bool COLUMNS, bool FIRST, class Src, class Dst>
__device__ __forceinline__ void fft_any_pass(const Src& src, const Dst& dst, const float2* tw, const FftPlan& p,
                                             int s) {
    switch (p.radix[s]) {
        case 20: fft_pass<20, INV, COLUMNS, FIRST>(src, dst, tw, p, s); break;
        case 16: fft_pass<16, INV, COLUMNS, FIRST>(src, dst, tw, p, s); break;
        case 15: fft_pass<15, INV, COLUMNS, FIRST>(src, dst, tw, p, s); break;
        case 14: fft_pass<14, INV, COLUMNS, FIRST>(src, dst, tw, p, s); break;
        case 13: fft_pass<13, INV, COLUMNS, FIRST>(src, dst, tw, p, s); break;
        case 12: fft_pass<12, INV, COLUMNS, FIRST>(src, dst, tw, p, s); break;
        case 11: fft_pass<11, INV, COLUMNS, FIRST>(src, dst, tw, p, s); break;
        case 10: fft_pass<10, INV, COLUMNS, FIRST>(src, dst, tw, p, s); break;
        case 9: fft_pass<9, INV, COLUMNS, FIRST>(src, dst, tw, p, s); break;
        case 8: fft_pass<8, INV, COLUMNS, FIRST>(src, dst, tw, p, s); break;
        case 7: fft_pass<7, INV, COLUMNS, FIRST>(src, dst, tw, p, s); break;
        case 6: fft_pass<6, INV, COLUMNS, FIRST>(src, dst, tw, p, s); break;
        case 5: fft_pass<5, INV, COLUMNS, FIRST>(src, dst, tw, p, s); break;
        case 4: fft_pass<4, INV, COLUMNS, FIRST>(src, dst, tw, p, s); break;
        case 3: fft_pass<3, INV, COLUMNS, FIRST>(src, dst, tw, p, s); break;
        default: fft_pass<2, INV, COLUMNS, FIRST>(src, dst, tw, p, s); break;
    }
}

// Transforms the block's eight transforms, exponent sign - (+ when INV),
// unscaled, from src to dst.  a and b are tiles; b is used from three factors
// up.  The roots are ready once a barrier has passed since fft_roots; the
// caller puts one between two calls (and between this call and readers of dst).
template <bool INV, bool COLUMNS, class Src, class Dst>
__device__ __forceinline__ void fft_run(const Src& src, const Dst& dst, float2* a, float2* b, const float2* tw,
                                        const FftPlan& p) {
    PitchedTile<COLUMNS> from{a}, to{b};
    fft_any_pass<INV, COLUMNS, true>(src, from, tw, p, 0);
    __syncthreads();
    for (int s = 1; s < p.passes - 1; s++) {
        fft_any_pass<INV, COLUMNS, false>(from, to, tw, p, s);
        __syncthreads();
        const PitchedTile<COLUMNS> x = from;
        from = to;
        to = x;
    }
    fft_any_pass<INV, COLUMNS, false>(from, dst, tw, p, p.passes - 1);
}

}  // namespace tt
