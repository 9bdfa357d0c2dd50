// Per-point operations shared by the single-volume and the batched kernels:
// grid_sample-style trilinear sampling of an rfft volume, the insertion splat,
// and the in-kernel CTF.
#pragma once
#include <cuda_runtime.h>

#include "slice_common.cuh"

namespace tt {

// ---------------------------------------------------------------- sampling

// grid_sample's source index of array coordinate c on an axis of n samples:
// c -> grid coordinate c / (0.5 n - 0.5) - 1 (grid_sample_utils.py:6-26) ->
// ((g + 1) / 2) * (n - 1) (align_corners=True), clipped to [0, n-1].
// grad_ok: the border clip passes a coordinate gradient — grid_sample's
// backward treats an index on the border itself (0 or n-1) as clipped.
__device__ __forceinline__ float source_index(float c, float half, float nm1, bool& grad_ok) {
    const float gc = __fsub_rn(__fdiv_rn(c, half), 1.0f);
    const float ix = __fmul_rn(__fmul_rn(__fadd_rn(gc, 1.0f), 0.5f), nm1);
    grad_ok = ix > 0.0f && ix < nm1;
    return fminf(fmaxf(ix, 0.0f), nm1);
}

// The same with the reciprocal of half (SliceGeom::half, rhalf).
__device__ __forceinline__ float source_index(float c, float half, float rhalf, float nm1, bool& grad_ok) {
    const float gc = __fsub_rn(divide_by(c, half, rhalf), 1.0f);
    const float ix = __fmul_rn(__fmul_rn(__fadd_rn(gc, 1.0f), 0.5f), nm1);
    grad_ok = ix > 0.0f && ix < nm1;
    return fminf(fmaxf(ix, 0.0f), nm1);
}

struct Corners {
    int z0, y0, x0;
    float ax0, ax1, ay0, ay1, az0, az1;  // per-axis weights of the low/high corner
    bool zin, yin, xin;                  // high corner inside the array
    bool gz, gy, gx;                     // the axis passes a coordinate gradient (not on the border)
};

// grid_sample source indices (z, y, x) of an inside array coordinate c, in
// [0, n-1], and whether each axis passes a coordinate gradient.
struct SourceIdx {
    float z, y, x;
    bool gz, gy, gx;
};

__device__ __forceinline__ SourceIdx source_indices(const SliceGeom& g, const float c[3]) {
    SourceIdx si;
    si.z = source_index(c[0], g.half[0], g.rhalf[0], g.ub0, si.gz);
    si.y = source_index(c[1], g.half[1], g.rhalf[1], g.ub1, si.gy);
    si.x = source_index(c[2], g.half[2], g.rhalf[2], g.ub2, si.gx);
    return si;
}

// Trilinear corner set of source indices (iz, iy, ix); gz, gy, gx are left
// false (make_corners sets them).
__device__ __forceinline__ Corners corners_at(const SliceGeom& g, float iz, float iy, float ix) {
    Corners k;
    k.gz = k.gy = k.gx = false;
    const float fz = floorf(iz), fy = floorf(iy), fx = floorf(ix);
    k.z0 = (int)fz;
    k.y0 = (int)fy;
    k.x0 = (int)fx;
    k.az0 = (fz + 1.0f) - iz;
    k.az1 = iz - fz;
    k.ay0 = (fy + 1.0f) - iy;
    k.ay1 = iy - fy;
    k.ax0 = (fx + 1.0f) - ix;
    k.ax1 = ix - fx;
    k.zin = k.z0 + 1 < g.D;
    k.yin = k.y0 + 1 < g.H;
    k.xin = k.x0 + 1 < g.W;
    return k;
}

// grid_sample trilinear corner set of an inside array coordinate c (the
// round trip decides the cell at integer kinks, where the derivative jumps).
__device__ __forceinline__ Corners make_corners(const SliceGeom& g, const float c[3]) {
    const SourceIdx si = source_indices(g, c);
    Corners k = corners_at(g, si.z, si.y, si.x);
    k.gz = si.gz;
    k.gy = si.gy;
    k.gx = si.gx;
    return k;
}

// Geometry of one extraction pixel: false when the pixel is outside
// fftfreq_max or its point outside the volume.
__device__ __forceinline__ bool extract_geometry(const SliceGeom& g, const float* m, int iy, int ix, float& qy,
                                                 float& qx, bool& cj, float c[3]) {
    qy = shifted_freq(iy, g.img_h, g.inv_h);
    qx = __fmul_rn((float)ix, g.inv_w);
    if (!in_fmax(g, qy, qx)) return false;
    float p[3];
    rotate_slice_point(m, qy, qx, p);
    cj = extract_conj(g, m, p[2]);
    if (cj) {
        p[0] = -p[0];
        p[1] = -p[1];
        p[2] = -p[2];
    }
    to_dft_coords(g, p, c);
    return inside_volume(g, c);
}

// The part of the extraction geometry that depends only on the slice row:
// its frequency qy, qy^2 for the fftfreq_max test, and the rotation's products
// m[i][1] * qy, each rounded as rotate_slice_point rounds it.  The slice
// kernels walk a row of tiles with a fixed row per thread, so these are formed
// once per thread instead of once per pixel.
struct SliceRow {
    float qy, qy2, my[3];
};

__device__ __forceinline__ SliceRow slice_row_geom(const SliceGeom& g, const float* m, int iy) {
    SliceRow r;
    r.qy = shifted_freq(iy, g.img_h, g.inv_h);
    r.qy2 = __fmul_rn(r.qy, r.qy);
#pragma unroll
    for (int i = 0; i < 3; i++) r.my[i] = __fmul_rn(m[i * 3 + 1], r.qy);
    return r;
}

// extract_geometry with the row part precomputed: the same operations and
// roundings, so the same flags and coordinates bit for bit.
__device__ __forceinline__ bool extract_geometry_row(const SliceGeom& g, const float* m, const SliceRow& row, int ix,
                                                     float& qx, bool& cj, float c[3]) {
    qx = __fmul_rn((float)ix, g.inv_w);
    if (g.has_fmax && !(__fsqrt_rn(__fadd_rn(row.qy2, __fmul_rn(qx, qx))) <= g.fmax)) return false;
    float p[3];
#pragma unroll
    for (int i = 0; i < 3; i++) p[i] = __fadd_rn(row.my[i], __fmul_rn(m[i * 3 + 2], qx));
    cj = extract_conj(g, m, p[2]);
    if (cj) {
        p[0] = -p[0];
        p[1] = -p[1];
        p[2] = -p[2];
    }
    to_dft_coords(g, p, c);
    return inside_volume(g, c);
}

// Element type of the bricked copy (brick_index addressing): one complex64 voxel.
struct VoxBrick2 {
    float x, y;
};

// The two x-corners (x0, x0 + 1) of volume row (z, y) (fftshifted
// coordinates): v0 when lo, v1 when hi (hi implies lo), zero otherwise.
// Plain layout: two 8-byte gathers.
__device__ __forceinline__ void load_xrow(const float2* __restrict__ vol, const SliceGeom& g, int z, int y, int x0,
                                          bool lo, bool hi, float2& v0, float2& v1) {
    const int64_t base = vox_index(g, z, y, x0);
    v0 = lo ? __ldg(vol + base) : make_float2(0.0f, 0.0f);
    v1 = hi ? __ldg(vol + base + 1) : make_float2(0.0f, 0.0f);
}

// x-paired layout (entry = (V[x], V[x + 1])): one 16-byte gather.
__device__ __forceinline__ void load_xrow(const float4* __restrict__ vol, const SliceGeom& g, int z, int y, int x0,
                                          bool lo, bool hi, float2& v0, float2& v1) {
    const float4 q = lo ? __ldg(vol + vox_index(g, z, y, x0)) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    v0 = make_float2(q.x, q.y);
    v1 = hi ? make_float2(q.z, q.w) : make_float2(0.0f, 0.0f);
}

// The four x-rows (z0 + bz, y0 + by) of a trilinear corner set k, addressed
// for layout VT: row (bz, by) gives v0 = V[.., x0] when lo and v1 =
// V[.., x0 + 1] when hi (hi implies lo), zero otherwise.
template <typename VT>
struct XRows {
    const VT* vol;
    int z0, y0, x0;
    __device__ __forceinline__ XRows(const VT* v, const SliceGeom&, const Corners& k)
        : vol(v), z0(k.z0), y0(k.y0), x0(k.x0) {}
    __device__ __forceinline__ void load(const SliceGeom& g, int bz, int by, bool lo, bool hi, float2& v0,
                                         float2& v1) const {
        load_xrow(vol, g, z0 + bz, y0 + by, x0, lo, hi, v0, v1);
    }
};

// Bricked layout (always fftshifted): the corner (z0, y0, x0) is addressed
// once; its +1 neighbours are the next slot of the brick along an even
// coordinate and the first slot of the next brick along an odd one (x: 1 or
// 7 slots, y: 2 or one brick row - 2, z: 4 or one brick plane - 4).  32-bit
// slot offsets: bricked copies hold fewer than 2^31 slots.
template <>
struct XRows<VoxBrick2> {
    const float2* p;
    uint32_t base, dz, dy, dx;
    __device__ __forceinline__ XRows(const VoxBrick2* v, const SliceGeom& g, const Corners& k)
        : p(reinterpret_cast<const float2*>(v)) {
        const uint32_t bh = (uint32_t)(g.H + 1) >> 1, bw = (uint32_t)(g.W + 1) >> 1;
        base = ((((uint32_t)k.z0 >> 1) * bh + ((uint32_t)k.y0 >> 1)) * bw + ((uint32_t)k.x0 >> 1)) * 8u +
               (((uint32_t)k.z0 & 1u) << 2) + (((uint32_t)k.y0 & 1u) << 1) + ((uint32_t)k.x0 & 1u);
        dx = (k.x0 & 1) ? 7u : 1u;
        dy = (k.y0 & 1) ? bw * 8u - 2u : 2u;
        dz = (k.z0 & 1) ? bh * bw * 8u - 4u : 4u;
    }
    __device__ __forceinline__ void load(const SliceGeom&, int bz, int by, bool lo, bool hi, float2& v0,
                                         float2& v1) const {
        const uint32_t i = base + (bz ? dz : 0u) + (by ? dy : 0u);
        v0 = lo ? __ldg(p + i) : make_float2(0.0f, 0.0f);
        v1 = hi ? __ldg(p + (i + dx)) : make_float2(0.0f, 0.0f);
    }
};

// Trilinear sample of the complex volume at corner set k; VT is float2 (plain
// layout), float4 (x-paired) or VoxBrick2 (bricked), with the same values and
// FMA order.
template <typename VT>
__device__ __forceinline__ float2 sample_trilinear(const VT* __restrict__ vol, const SliceGeom& g,
                                                   const Corners& k) {
    float2 r = make_float2(0.0f, 0.0f);
    const XRows<VT> rows(vol, g, k);
#pragma unroll
    for (int bz = 0; bz < 2; bz++) {
        if (bz && !k.zin) continue;
        const float wz = bz ? k.az1 : k.az0;
#pragma unroll
        for (int by = 0; by < 2; by++) {
            if (by && !k.yin) continue;
            const float wzy = (by ? k.ay1 : k.ay0) * wz;
            float2 v0, v1;
            rows.load(g, bz, by, true, k.xin, v0, v1);
            const float w0 = k.ax0 * wzy;
            r.x = fmaf(v0.x, w0, r.x);
            r.y = fmaf(v0.y, w0, r.y);
            if (k.xin) {
                const float w1 = k.ax1 * wzy;
                r.x = fmaf(v1.x, w1, r.x);
                r.y = fmaf(v1.y, w1, r.y);
            }
        }
    }
    return r;
}

// --------------------------------------------------------------------- CTF

// Per-image constants of the 2D CTF -sin(chi) of torch-ctf's calculate_ctf_2d
// (ctf_2d.py:12-131, ctf_utils.py:46-86, ctf_aberrations.py:42-81):
//   chi = k1 * s^2 * df(direction) + k2 * s^4 - phase_shift - atan(A / sqrt(1 - A^2))
//   k1 = -pi * lambda, k2 = pi / 2 * Cs * lambda^3 (Angstrom), s in cycles/Angstrom,
//   df = defocus - astig + 2 * (u . a)^2, u the unit frequency direction
//   (with float32 epsilon in its norm), a = sqrt(astig) * (sin theta, cos theta) (yx).
struct CtfConst {
    double k1, k2, phase;        // Angstrom units; phase includes the amplitude-contrast term
    double defocus, astig;       // micrometres (the astigmatism adjustment is done in um)
    double ay, ax;               // astigmatism vector sqrt(astig) * (sin, cos)
    double inv_px;               // 1 / pixel size (1/Angstrom)
};

// Constants of one image from its tt_ctf_params (double precision, once per
// image), in three parts of about equal length that different warps form side
// by side: part 0 the wavelength terms, 1 the phase terms, 2 the astigmatism.
__device__ inline void make_ctf_const(const tt_ctf_params& p, int part, CtfConst& k) {
    const double pi = 3.14159265358979323846;
    if (part == 0) {
        const double h = 6.62607015e-34, c = 299792458.0, m0 = 9.1093837015e-31, e = 1.602176634e-19;
        const double ev = e * (double)p.voltage_kv * 1e3;
        const double lambda = h * c / sqrt(ev * (2.0 * m0 * c * c + ev)) * 1e10;  // Angstrom
        const double cs = (double)p.spherical_aberration_mm * 1e7;
        k.k1 = -pi * lambda;
        k.k2 = pi / 2.0 * cs * lambda * lambda * lambda;
        k.inv_px = 1.0 / (double)p.pixel_size_a;
    } else if (part == 1) {
        const double ac = (double)p.amplitude_contrast;
        k.phase = (double)p.phase_shift_deg * pi / 180.0 + atan(ac / sqrt(1.0 - ac * ac));
        k.defocus = p.defocus_um;
    } else {
        k.astig = p.astigmatism_um;
        const double th = (double)p.astigmatism_angle_deg * pi / 180.0;
        const double sa = sqrt((double)(p.astigmatism_um > 0 ? p.astigmatism_um : 0.0f));
        double sn, cn;
        sincos(th, &sn, &cn);
        k.ay = sa * sn;
        k.ax = sa * cn;
    }
}

// CTF at slice frequency (qy, qx) in cycles/pixel.  The phase reaches hundreds
// of radians at high frequency, so it is evaluated in double.
__device__ __forceinline__ float ctf_value(const CtfConst& k, float qy, float qx) {
    const double y = (double)qy * k.inv_px, x = (double)qx * k.inv_px;
    const double s2 = y * y + x * x;
    double df = k.defocus * 1e4;  // um -> Angstrom
    if (k.astig != 0.0) {         // the same for every pixel of an image
        // (u . a)^2 with u = (y, x) / sqrt(s2 + eps), eps = torch.finfo(float32).eps:
        // one division instead of a square root and a reciprocal (both in
        // double: 256^3 x 4096 CTF slices, see batched.cu)
        const double t = y * k.ay + x * k.ax;
        df += (2.0 * (t * t) / (s2 + 1.1920928955078125e-07) - k.astig) * 1e4;
    }
    const double chi = k.k1 * s2 * df + k.k2 * s2 * s2 - k.phase;
    // the phase is reduced to half turns in [-1, 1] in double (error ~1e-12 at a
    // few thousand radians); the float sine of the reduced phase is then
    // accurate to ~1e-7, as the float result, at a fraction of a double sine's
    // cost, and sinpi needs no further reduction
    const double turns = chi * (1.0 / 6.283185307179586);
    return -sinpif((float)(2.0 * (turns - rint(turns))));
}

// ---------------------------------------------------------------- insertion

template <typename R>
struct Acc;
template <>
struct Acc<float> {
    using T = float4;
    using C = float2;
};
template <>
struct Acc<double> {
    using T = double4;
    using C = double2;
};

__device__ __forceinline__ void acc_add(float4* a, float re, float im, float w) {
    atomicAdd(a, make_float4(re, im, w, 0.0f));
}
__device__ __forceinline__ void acc_add(double4* a, double re, double im, double w) {
    atomicAdd(&a->x, re);
    atomicAdd(&a->y, im);
    atomicAdd(&a->z, w);
}

__device__ __forceinline__ float2 load_slice(const float2* p) { return __ldcs(p); }
__device__ __forceinline__ double2 load_slice(const double2* p) { return __ldcs(p); }

// Float accumulation target: one (re, im, w, 0) vector reduction per corner.
template <typename R>
struct FloatSplat {
    typename Acc<R>::T* acc;
    __device__ __forceinline__ void operator()(int64_t vi, R dre, R dim, R w, R wscale) const {
        acc_add(acc + vi, dre * w, dim * w, w * wscale);
    }
};

// Source pixels the insertion skips: outside fftfreq_max, and the
// Friedel-redundant half of the x = 0 column (x == 0, y < 0).
__device__ __forceinline__ bool insert_pixel_kept(const SliceGeom& g, float qy, float qx) {
    return in_fmax(g, qy, qx) && !(qx == 0.0f && qy < 0.0f);
}

// Floor / ceil cell of an insertion point and its fractional offsets.
struct InsertCell {
    int iz0, iy0, ix0, iz1, iy1, ix1;
    float tz, ty, tx;
};

// Insertion geometry of slice frequency (qy, qx): rotation, the strict x' < 0
// redirect (cj), array coordinates c and the whole-point bounds test.
__device__ __forceinline__ bool insert_coords(const SliceGeom& g, const float* m, float qy, float qx, bool& cj,
                                              float c[3]) {
    float p[3];
    rotate_slice_point(m, qy, qx, p);
    cj = p[2] < 0.0f;
    if (cj) {
        p[0] = -p[0];
        p[1] = -p[1];
        p[2] = -p[2];
    }
    to_dft_coords(g, p, c);
    return inside_volume(g, c);
}

// insert_coords with the row part of the geometry precomputed (slice_row_geom):
// the same operations and roundings.
__device__ __forceinline__ bool insert_coords_row(const SliceGeom& g, const float* m, const SliceRow& row, float qx,
                                                  bool& cj, float c[3]) {
    float p[3];
#pragma unroll
    for (int i = 0; i < 3; i++) p[i] = __fadd_rn(row.my[i], __fmul_rn(m[i * 3 + 2], qx));
    cj = p[2] < 0.0f;
    if (cj) {
        p[0] = -p[0];
        p[1] = -p[1];
        p[2] = -p[2];
    }
    to_dft_coords(g, p, c);
    return inside_volume(g, c);
}

// Floor / ceil cell of inside array coordinates c.
__device__ __forceinline__ void cell_at(const float c[3], InsertCell& k) {
    const float z0 = floorf(c[0]), y0 = floorf(c[1]), x0 = floorf(c[2]);
    k.tz = c[0] - z0;
    k.ty = c[1] - y0;
    k.tx = c[2] - x0;
    k.iz0 = (int)z0;
    k.iy0 = (int)y0;
    k.ix0 = (int)x0;
    k.iz1 = (int)ceilf(c[0]);
    k.iy1 = (int)ceilf(c[1]);
    k.ix1 = (int)ceilf(c[2]);
}

// z-phase of an insertion tile: the accumulator of a large volume is filled
// in nphase passes, pass k taking the tiles whose centre point (after the
// x' < 0 redirect) lies in the k-th z-slab, so each pass reduces into about
// 1/nphase of the accumulator and more of its lines stay in L2.  Only the
// order of the work changes: every tile belongs to exactly one pass.
// (cy, cx): the tile's centre pixel.
__device__ __forceinline__ int insert_tile_phase(const SliceGeom& g, const float* m, int cy, int cx, int nphase) {
    const float qy = shifted_freq(cy, g.img_h, g.inv_h);
    const float qx = __fmul_rn((float)cx, g.inv_w);
    float p[3];
    rotate_slice_point(m, qy, qx, p);
    const float z = p[2] < 0.0f ? -p[0] : p[0];
    const int ph = (int)floorf((z + 0.5f) * (float)nphase);
    return ph < 0 ? 0 : (ph >= nphase ? nphase - 1 : ph);
}

// Tiles first .. first + 31 of a row of `tiles` tiles (TX pixels wide, centre row
// cy) that belong to z-phase `phase`, as a bit mask: lane l answers for tile
// first + l, so a row costs one phase test instead of one per tile (320^3 in
// two phases: 9 % of the splat's instructions).  All lanes call it.
template <int TX>
__device__ __forceinline__ unsigned phase_tiles(const SliceGeom& g, const float* m, int cy, int first, int tiles,
                                                int phase, int nphase) {
    const int tx = first + (threadIdx.x & 31);
    const bool mine = tx < tiles &&
                      (nphase == 1 || insert_tile_phase(g, m, min(cy, g.img_h - 1), min(tx * TX + TX / 2, g.wr - 1),
                                                        nphase) == phase);
    return __ballot_sync(0xffffffffu, mine);
}

// Tiles first .. first + 31 of a row of tiles that hold, in the warp's ROWS rows
// from iy0 on, a pixel within fftfreq_max: the patch's nearest to the origin has
// the smallest frequencies, and the roundings are monotonic.  An empty patch costs
// the octets more than the lane pairs: up to 0.2 cycles per pixel the bricked
// splat of 2376 slices of 128^2 took 138 us (lane pairs 118) with a vote in every
// patch and takes 103, 1500 of 256^2 290 (270) and 172; without a limit nothing
// changes.  All lanes call it.
template <int TX, int ROWS>
__device__ __forceinline__ unsigned limit_tiles(const SliceGeom& g, int iy0, int first) {
    if (!g.has_fmax) return 0xffffffffu;
    const float qy = shifted_freq(min(max(g.img_h / 2, iy0), iy0 + ROWS - 1), g.img_h, g.inv_h);
    const float qx = __fmul_rn((float)((first + (int)(threadIdx.x & 31)) * TX), g.inv_w);
    return __ballot_sync(0xffffffffu, in_fmax(g, qy, qx));
}

// Insertion geometry and cell of slice frequency (qy, qx); false when the
// point is outside the volume.
__device__ __forceinline__ bool insert_cell(const SliceGeom& g, const float* m, float qy, float qx, bool& cj,
                                            InsertCell& k) {
    float c[3];
    if (!insert_coords(g, m, qy, qx, cj, c)) return false;
    cell_at(c, k);
    return true;
}

// Weight of corner `corner` (bit 2: z, bit 1: y, bit 0: x high) with the
// reference's float32 products, left to right.
__device__ __forceinline__ float insert_corner_weight(const InsertCell& k, int corner) {
    const int bz = (corner >> 2) & 1, by = (corner >> 1) & 1, bx = corner & 1;
    const float fz = bz ? k.tz : 1.0f - k.tz;
    const float fy = by ? k.ty : 1.0f - k.ty;
    const float fx = bx ? k.tx : 1.0f - k.tx;
    return (fz * fy) * fx;
}

__device__ __forceinline__ void insert_corner_zyx(const InsertCell& k, int corner, int& z, int& y, int& x) {
    z = (corner & 4) ? k.iz1 : k.iz0;
    y = (corner & 2) ? k.iy1 : k.iy0;
    x = (corner & 1) ? k.ix1 : k.ix0;
}

// Splat of one source pixel, following _insert_central_slices_rfft_3d.py:30-85
// and _insert_into_3d_dft_linear :289-346: each of the eight corners receives
// (data * w, w) through sink(voxel, re, im, w, weight scale).  With a CTF
// (ctf != nullptr) the data are weighted by the CTF and the interpolation
// weights by its square.
template <typename R, typename Sink>
__device__ __forceinline__ void insert_point_to(const typename Acc<R>::C* __restrict__ img, const float* m,
                                                const Sink& sink, const SliceGeom& g, int64_t s, int iy, int ix,
                                                const CtfConst* ctf = nullptr) {
    const float qy = shifted_freq(iy, g.img_h, g.inv_h);
    const float qx = __fmul_rn((float)ix, g.inv_w);
    if (!insert_pixel_kept(g, qy, qx)) return;
    // issued before the geometry so the load overlaps it
    const typename Acc<R>::C d = load_slice(img + (s * g.slice_rows + slice_row(g, iy)) * (int64_t)g.slice_pitch + ix);
    bool cj;
    InsertCell k;
    if (!insert_cell(g, m, qy, qx, cj, k)) return;
    R dre = d.x, dim = d.y, wscale = (R)1;
    if (ctf) {
        const float cv = ctf_value(*ctf, qy, qx);
        dre *= (R)cv;
        dim *= (R)cv;
        wscale = (R)(cv * cv);
    }
    if (cj) dim = -dim;
#pragma unroll
    for (int corner = 0; corner < 8; corner++) {
        const float w = insert_corner_weight(k, corner);
        if (w == 0.0f) continue;  // adds nothing (ceil == floor or zero fraction)
        int z, y, x;
        insert_corner_zyx(k, corner, z, y, x);
        sink(vox_index(g, z, y, x), dre, dim, (R)w, wscale);
    }
}

// Slot of voxel (z, y, x) (fftshifted) in a 2 x 2 x 2-bricked accumulator:
// bricks of 8 float4 slots (one 128-byte line) in (z, y, x) brick order, x
// fastest inside a brick; dims padded to even.
__device__ __forceinline__ int64_t accumulator_slot(const SliceGeom& g, int z, int y, int x) {
    const int64_t bh = (g.H + 1) >> 1, bw = (g.W + 1) >> 1;
    return ((((int64_t)(z >> 1) * bh + (y >> 1)) * bw + (x >> 1)) << 3) + ((z & 1) << 2) + ((y & 1) << 1) +
           (x & 1);
}

// The value a float splat adds for source pixel (iy, ix) of slice s: the
// (CTF-weighted, redirect-conjugated) data, the weight scale and the array
// coordinates c, with c[0] = -1 where the pixel adds nothing (no pixel,
// outside fftfreq_max, the redundant half of the x = 0 column, or a point
// outside the volume).
__device__ __forceinline__ void splat_source(const float2* __restrict__ img, const float* m, const SliceGeom& g,
                                             int64_t s, bool has_pixel, int iy, int ix, const CtfConst* ctf,
                                             float& dre, float& dim, float& wscale, float c[3]) {
    dre = 0.f;
    dim = 0.f;
    wscale = 1.f;
    c[0] = -1.f;
    c[1] = 0.f;
    c[2] = 0.f;
    if (!has_pixel) return;
    const float qy = shifted_freq(iy, g.img_h, g.inv_h);
    const float qx = __fmul_rn((float)ix, g.inv_w);
    if (!insert_pixel_kept(g, qy, qx)) return;
    const float2 d = load_slice(img + (s * g.slice_rows + slice_row(g, iy)) * (int64_t)g.slice_pitch + ix);
    bool cj;
    float ci[3];
    if (!insert_coords(g, m, qy, qx, cj, ci)) return;
    dre = d.x;
    dim = cj ? -d.y : d.y;
    if (ctf) {
        const float cv = ctf_value(*ctf, qy, qx);
        dre *= cv;
        dim *= cv;
        wscale = cv * cv;
    }
    c[0] = ci[0];
    c[1] = ci[1];
    c[2] = ci[2];
}

// splat_source without a CTF and with the row part of the geometry formed once
// per thread (slice_row_geom of the thread's slice row): the same operations
// and roundings.  irow: the storage row's first element.  256^3 x 4096: 2.92
// against 2.99 ms; the batched kernel, whose registers hold the CTF, loses 3 %
// with it.
__device__ __forceinline__ void splat_source_row(const float2* __restrict__ irow, const float* m, const SliceRow& row,
                                                 const SliceGeom& g, bool has_pixel, int ix, float& dre, float& dim,
                                                 float& wscale, float c[3]) {
    dre = 0.f;
    dim = 0.f;
    wscale = 1.f;
    c[0] = -1.f;
    c[1] = 0.f;
    c[2] = 0.f;
    const float qx = __fmul_rn((float)ix, g.inv_w);
    const bool kept = has_pixel && (!g.has_fmax || __fsqrt_rn(__fadd_rn(row.qy2, __fmul_rn(qx, qx))) <= g.fmax) &&
                      !(qx == 0.0f && row.qy < 0.0f);
    if (!kept) return;
    const float2 d = load_slice(irow + ix);
    bool cj;
    float ci[3];
    if (!insert_coords_row(g, m, row, qx, cj, ci)) return;
    dre = d.x;
    dim = cj ? -d.y : d.y;
    c[0] = ci[0];
    c[1] = ci[1];
    c[2] = ci[2];
}

// Float splat of one source pixel with x-paired lanes into the plain
// accumulator: lanes 2j and 2j+1 reduce the x-low and the x-high corner of
// the same pixel in the same instruction (adjacent voxels, usually one
// 32-byte L2 sector), serving pixels j and j + 16 in two rounds.  Only the
// pixel's value (and CTF weight) and its three array coordinates move by warp
// shuffles; each lane rebuilds the floor / ceil cell from them.  Same pixels,
// corners, weights ((fz * fy) * fx), CTF weighting and values as
// insert_point.  Must be called by all 32 lanes of the warp (has_pixel false
// where the tile overhangs the slice).
__device__ __forceinline__ void insert_point_paired(const float2* __restrict__ img, const float* m,
                                                    float4* __restrict__ acc, const SliceGeom& g, int64_t s,
                                                    bool has_pixel, int iy, int ix, const CtfConst* ctf = nullptr) {
    const unsigned full = 0xffffffffu;
    const int lane = threadIdx.x & 31, bx = lane & 1;
    float dre, dim, wscale, c[3];
    splat_source(img, m, g, s, has_pixel, iy, ix, ctf, dre, dim, wscale, c);
#pragma unroll
    for (int half = 0; half < 2; half++) {
        const int src = (lane >> 1) + 16 * half;
        // every lane runs every shuffle (full mask; ctf is the same for the warp)
        const float sre = __shfl_sync(full, dre, src), sim = __shfl_sync(full, dim, src);
        const float sws = ctf ? __shfl_sync(full, wscale, src) : 1.0f;
        float sc[3];
#pragma unroll
        for (int a = 0; a < 3; a++) sc[a] = __shfl_sync(full, c[a], src);
        if (sc[0] < 0.0f) continue;
        InsertCell k;
        cell_at(sc, k);
        const int x = bx ? k.ix1 : k.ix0;
        const float fx = bx ? k.tx : 1.0f - k.tx;
#pragma unroll
        for (int zy = 0; zy < 4; zy++) {
            const int bz = zy >> 1, by = zy & 1;
            const float w = ((bz ? k.tz : 1.0f - k.tz) * (by ? k.ty : 1.0f - k.ty)) * fx;
            if (w != 0.0f) {
                const int z = bz ? k.iz1 : k.iz0, y = by ? k.iy1 : k.iy0;
                acc_add(acc + vox_index(g, z, y, x), sre * w, sim * w, w * sws);
            }
        }
    }
}

// One warp's pixels on their way from the lane that formed them to the lanes
// that reduce their corners (insert_point_octet).
struct SplatTable {
    float4 data[32];  // re, im, bits of the low corner's slot, bits of the neighbour code
    float4 cell[32];  // fractions tz, ty, tx, weight scale (0: no pixel)
};

// Float splat of one source pixel into the 2 x 2 x 2-bricked accumulator
// (accumulator_slot, fewer than 2^32 slots) with lane octets: lanes 8j..8j+7
// reduce the eight corners of one pixel in the same instruction (corner =
// lane & 7: bit 2 z, bit 1 y, bit 0 x high), four neighbouring pixels of a
// slice row per instruction in eight rounds.  A cell's corners fall on (1.5)^3
// 128-byte lines on average, which leave the SM as one request each.
//
// The reductions are bound by the SM's request port to the L2 (82 % busy with
// one reduction per pixel and corner, at 60 % of the issue slots), so corners
// that two pixels share are added up first: the outer pixels of the four hand
// the corners that fall on their inner neighbour's cell to it (lanes 0 -> 1
// and 3 -> 2; the shared voxels follow from the two cells' offset, at most one
// voxel per axis).  256^3 x 2048 slices: 21 % fewer reduced sectors, 1.50 ms
// against 1.79; 128^3 x 4096: 0.77 against 0.88; 320^3 x 1024: 1.41 against
// 1.60.  The pixel records go through shared memory (two 16-byte broadcasts a
// round instead of seven shuffles).  Handing on from 1 to 2 as well takes
// another 15 % of the sectors but 22 more instructions a round, and the kernel
// is then bound by issue: 1.76 ms.
//
// dre, dim, wscale and c are the lane's pixel (splat_source; ctf: it may have a CTF);
// same corners and weights ((fz * fy) * fx) as insert_point.  All 32 lanes of
// the warp call it, with the warp's own table.
__device__ __forceinline__ void insert_point_octet(float4* __restrict__ acc, const SliceGeom& g, float dre, float dim,
                                                   float wscale, const float c[3], SplatTable& tab, bool ctf) {
    const unsigned full = 0xffffffffu;
    const int lane = threadIdx.x & 31, corner = lane & 7, p = lane >> 3;
    const uint32_t bh = (uint32_t)(g.H + 1) >> 1, bw = (uint32_t)(g.W + 1) >> 1;
    {
        const bool on = c[0] >= 0.0f;
        const float fz = floorf(c[0]), fy = floorf(c[1]), fx = floorf(c[2]);
        // a lane without a pixel: a cell far from every other, all of its corners zero
        const int z0 = on ? (int)fz : -0x10000, y0 = (int)fy, x0 = (int)fx;
        const uint32_t slot = (((uint32_t)z0 >> 1) * bh + ((uint32_t)y0 >> 1)) * bw * 8u + ((uint32_t)x0 >> 1) * 8u +
                              (((uint32_t)z0 & 1u) << 2) + (((uint32_t)y0 & 1u) << 1) + ((uint32_t)x0 & 1u);
        // neighbour code: corner k of this cell is corner k + D of the neighbour's;
        // bits 0-7 the corners for which it exists, bits 8-11 D + 8
        const int dz = z0 - __shfl_xor_sync(full, z0, 1), dy = y0 - __shfl_xor_sync(full, y0, 1),
                  dx = x0 - __shfl_xor_sync(full, x0, 1);
        const int pair_on = __shfl_xor_sync(full, (int)on, 1);  // every lane shuffles
        const bool both = on && pair_on;
        const int mz = dz == 0 ? 0xff : (dz == 1 ? 0x0f : (dz == -1 ? 0xf0 : 0));
        const int my = dy == 0 ? 0xff : (dy == 1 ? 0x33 : (dy == -1 ? 0xcc : 0));
        const int mx = dx == 0 ? 0xff : (dx == 1 ? 0x55 : (dx == -1 ? 0xaa : 0));
        const int code = (both ? mz & my & mx : 0) | (((dz * 4 + dy * 2 + dx + 8) & 15) << 8);
        // nothing to add (a patch outside fftfreq_max or the volume): 256^3 x 2048
        // up to 0.3 cycles per pixel 1060 -> 657 us
        if (!__any_sync(full, on)) return;
        __syncwarp();  // the previous call's reads
        tab.data[lane] = make_float4(dre, dim, __uint_as_float(on ? slot : 0u), __int_as_float(code));
        tab.cell[lane] = on ? make_float4(c[0] - fz, c[1] - fy, c[2] - fx, wscale) : make_float4(0.f, 0.f, 0.f, 0.f);
        __syncwarp();
    }
    // per axis: fraction t -> t (high corner) or 1 - t (low), both exact
    const float az = (corner & 4) ? 1.0f : -1.0f, bz = (corner & 4) ? 0.0f : 1.0f;
    const float ay = (corner & 2) ? 1.0f : -1.0f, by = (corner & 2) ? 0.0f : 1.0f;
    const float ax = (corner & 1) ? 1.0f : -1.0f, bx = (corner & 1) ? 0.0f : 1.0f;
    // slots from the low corner to this lane's, from an even / odd coordinate
    const uint32_t ez = (corner & 4) ? 4u : 0u, oz = (corner & 4) ? bh * bw * 8u - 4u : 0u;
    const uint32_t ey = (corner & 2) ? 2u : 0u, oy = (corner & 2) ? bw * 8u - 2u : 0u;
    const uint32_t ex = (corner & 1) ? 1u : 0u, ox = (corner & 1) ? 7u : 0u;
    const bool inner = p == 1 || p == 2;
    const int other = ((p ^ 1) << 3) + corner - 8;
#pragma unroll
    for (int r = 0; r < 8; r++) {
        const float4 d = tab.data[4 * r + p], f = tab.cell[4 * r + p];
        const uint32_t base = __float_as_uint(d.z);
        const int code = __float_as_int(d.w);
        const float w = (fmaf(f.x, az, bz) * fmaf(f.y, ay, by)) * fmaf(f.z, ax, bx);
        const uint32_t slot = base + ((base & 4u) ? oz : ez) + ((base & 2u) ? oy : ey) + ((base & 1u) ? ox : ex);
        // a corner of zero weight adds nothing, whatever the data and the CTF: past
        // the last index its slot is not its voxel's (0 * NaN would reduce into it;
        // without a CTF the scale is 0 or 1)
        float re = w != 0.0f ? d.x * w : 0.0f, im = w != 0.0f ? d.y * w : 0.0f;
        float wt = !ctf || w != 0.0f ? w * f.w : 0.0f;
        const bool shared = (code >> corner) & 1;
        const int from = other + ((code >> 8) & 15);
        const float ore = __shfl_sync(full, re, from), oim = __shfl_sync(full, im, from),
                    owt = __shfl_sync(full, wt, from);
        if (shared && inner) {
            re += ore;
            im += oim;
            wt += owt;
        }
        // with a CTF the weight can vanish where the data do not
        const bool any = ctf ? ((__float_as_uint(re) | __float_as_uint(im) | __float_as_uint(wt)) & 0x7fffffffu) != 0
                             : wt != 0.0f;
        if (any && (inner || !shared)) acc_add(acc + slot, re, im, wt);
    }
}

// dL/dacc at voxel (z, y, x) for upstream dL/dvolume G: the adjoint of the
// Friedel completion, G[v] + conj(G[m v]) on the x = 0 plane unless v is DC.
template <typename R>
__device__ __forceinline__ typename Acc<R>::C completed_grad(const typename Acc<R>::C* __restrict__ gvol,
                                                            const SliceGeom& g, int z, int y, int x) {
    typename Acc<R>::C a = gvol[vox_index(g, z, y, x)];
    if (x == 0 && !(z == g.D / 2 && y == g.H / 2)) {
        const typename Acc<R>::C b = gvol[vox_index(g, (g.D - z) % g.D, (g.H - y) % g.H, 0)];
        a.x += b.x;
        a.y -= b.y;
    }
    return a;
}

// Splat into the float (re, im, w, 0) accumulator.
template <typename R>
__device__ __forceinline__ void insert_point(const typename Acc<R>::C* __restrict__ img, const float* m,
                                             typename Acc<R>::T* __restrict__ acc, const SliceGeom& g, int64_t s,
                                             int iy, int ix, const CtfConst* ctf = nullptr) {
    insert_point_to<R>(img, m, FloatSplat<R>{acc}, g, s, iy, ix, ctf);
}

}  // namespace tt
