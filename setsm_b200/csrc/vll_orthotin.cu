// vll_orthotin.cu -- the TIN-triangle orthoimage height search of SETSM's
// blunder removal: VerticalLineLocus_Ortho (setsm_code.cpp:8234-8533) and the
// loop that drives it, Ortho_blunder (:8028-8232).
//
// For a triangle of matched points with two anchored vertices, the third
// (target) vertex's height is swept over its UGRID range; at each height the
// triangle's plane is rasterised over the grid cells of its bounding box, every
// cell inside the triangle is projected through the RPCs of the reference and
// each target image, and the Pearson correlation of the sampled intensities
// and magnitudes (Correlate, SubFunctions.cpp:974-1018) picks the height.
//
// GPU layout: one block per triangle, the triangles with two anchored
// vertices taken from a list.  The triangle's box and its inside cells do not
// depend on the swept height, so the inside cells are listed once.  All
// heights are screened, a thread each, with FP64 cubics in the height per
// cell; the few that can win are evaluated in the reference's own order:
// their cells are projected a thread each, the samples staged in shared
// memory for both of Correlate's passes, and every sum accumulated by one
// thread in the reference's cell order, so the FP64 results are the
// reference's bit for bit.  A triangle with more than 256 inside cells tests
// its box per height and recomputes the samples in the second pass.  The
// sequential "apply" pass of
// Ortho_blunder is restated in parallel with the same result: triangles that
// found a height are grouped by target point (stable radix sort), each
// point's triangles are walked in triangle order to find the record-breakers
// of the running maximum (the reference's com_count test), and the anchor
// counts of the second half of the pass use, per grid node, the first
// triangle index that anchored it.
#include <algorithm>
#include <cstdint>

#include <cub/device/device_radix_sort.cuh>
#include <cuda_runtime.h>

#include "vll_exact.cuh"
#include "vll_geo.cuh"
#include "vll_internal.h"

namespace vll {

namespace {

struct P3 {
    double x, y, z;
};

__device__ __forceinline__ double dmin(double a, double b) { return b < a ? b : a; }
__device__ __forceinline__ double dmax(double a, double b) { return a < b ? b : a; }

// One cell's samples (InterpolatePatch of both planes of both images at the
// plane height) are cell_sample's, for a cell that cell_inside accepts;
// setsm_code.cpp:8331-8451.
// Whether the cell lies in the triangle: the three edge tests (D3DPOINT
// differences; z unused, so the answer is the same at every height).
__device__ bool cell_inside(const DevLevel &P, const P3 &T1, const P3 &T2, const P3 &T3,
                            int64_t row, int64_t col) {
    const double gs = P.grid_res;
    const double cx = __dadd_rn(__dmul_rn((double)col, gs), P.boundary[0]);
    const double cy = __dadd_rn(__dmul_rn((double)row, gs), P.boundary[1]);
    int sum = 3;
    if (__dadd_rn(__dmul_rn(__dadd_rn(T2.x, -T1.x), __dadd_rn(cy, -T1.y)),
                  -__dmul_rn(__dadd_rn(T2.y, -T1.y), __dadd_rn(cx, -T1.x))) <= 0)
        --sum;
    if (__dadd_rn(__dmul_rn(__dadd_rn(T3.x, -T2.x), __dadd_rn(cy, -T2.y)),
                  -__dmul_rn(__dadd_rn(T3.y, -T2.y), __dadd_rn(cx, -T2.x))) <= 0)
        --sum;
    if (__dadd_rn(__dmul_rn(__dadd_rn(T1.x, -T3.x), __dadd_rn(cy, -T3.y)),
                  -__dmul_rn(__dadd_rn(T1.y, -T3.y), __dadd_rn(cx, -T3.x))) <= 0)
        --sum;
    return sum == 0 || sum == 3;
}

// The samples of a cell inside the triangle at the plane's height, or false
// when the plane is degenerate or a window corner leaves an image.
__device__ bool cell_sample(const DevLevel &P, const double2 *__restrict__ lonlat, int ti,
                            bool plane_ok, double A, double B, double C, double D, int64_t row,
                            int64_t col, double v[4]) {
    if (!plane_ok) return false;
    const double gs = P.grid_res;
    const double cx = __dadd_rn(__dmul_rn((double)col, gs), P.boundary[0]);
    const double cy = __dadd_rn(__dmul_rn((double)row, gs), P.boundary[1]);
    // Z = -1.0 * ((A x) + (B y) + D) / C
    const double z = __ddiv_rn(-__dadd_rn(__dadd_rn(__dmul_rn(A, cx), __dmul_rn(B, cy)), D), C);
    // the cell's longitude / latitude: from the grid-wide table when given
    // (the same function of the same coordinates), else computed here
    const double2 w = lonlat ? lonlat[row * P.grid_w + col] : ps2wgs_dev(P.param, cx, cy);
    const DevImage &ri = P.im[P.ref], &tI = P.im[ti];
    // the target image is projected with the reference image's adjustment,
    // as the reference does (temp_LIA, setsm_code.cpp:8392)
    const double2 rp = to_pyramid(rpc_project(ri.rpc, ri.adj, w.x, w.y, z), ri.sx, ri.sy, P.L);
    const double2 tp = to_pyramid(rpc_project(tI.rpc, ri.adj, w.x, w.y, z), tI.sx, tI.sy, P.L);
    if (!(tp.y >= 0 && __dadd_rn(tp.y, 1.0) < (double)tI.h && tp.x >= 0 &&
          __dadd_rn(tp.x, 1.0) < (double)tI.w && rp.y >= 0 && __dadd_rn(rp.y, 1.0) < (double)ri.h &&
          rp.x >= 0 && __dadd_rn(rp.x, 1.0) < (double)ri.w))
        return false;
    const double dx = __dadd_rn(rp.x, -(double)(int)rp.x), dy = __dadd_rn(rp.y, -(double)(int)rp.y);
    const int64_t pos = (int64_t)rp.x + (int64_t)rp.y * (int64_t)ri.w;
    const double dxr = __dadd_rn(tp.x, -(double)(int)tp.x), dyr = __dadd_rn(tp.y, -(double)(int)tp.y);
    const int64_t posr = (int64_t)tp.x + (int64_t)tp.y * (int64_t)tI.w;
    v[0] = interp(ri.img, pos, ri.w, dx, dy);
    v[1] = interp(tI.img, posr, tI.w, dxr, dyr);
    v[2] = interp(ri.mag, pos, ri.w, dx, dy);
    v[3] = interp(tI.mag, posr, tI.w, dxr, dyr);
    return true;
}

// Correlate's final step (SubFunctions.cpp:1000-1010).
__device__ __forceinline__ double corr_of(double slr, double sl2, double sr2) {
    if (sl2 > 1e-8 && sr2 > 1e-8) return __ddiv_rn(slr, sqrt(__dmul_rn(sl2, sr2)));
    return -99.0;
}

struct SearchOut {
    double f_height, f_sncc;
    int selected;
};

// A cell of the screening pass: the four RPC cubics of both images in the
// normalised height at the cell's longitude and latitude (im 0: reference),
// and the triangle's height there, z0 + z1 * (target vertex's height).
struct ScreenCell {
    double c[2][4][4];
    double z0, z1;
};

// The block's shared staging.  The triangle's bounding box and which of its
// cells lie inside do not depend on the swept height, so the inside cells are
// listed once per triangle (up to kCellCap).  The screening pass holds 32
// cells' cubics; an exact evaluation of one height keeps the listed cells'
// samples for both of Correlate's passes (a triangle with more inside cells
// tests its box, kCellCap cells at a time, and recomputes the samples in the
// second pass).
constexpr int kSearchThreads = 128;
constexpr int kSearchWarps = kSearchThreads / 32;
constexpr int kCellCap = 256;
struct CellStage {
    union {
        double v[4 * kCellCap];     // item i: img ref, img tgt, mag ref, mag tgt
        ScreenCell sc[32];
    };
    unsigned int valid[kCellCap / 32];
    int32_t cell[kCellCap];         // the box's cells inside the triangle, in cell order
    double sum[6];
    int count;
    int warp_n[kSearchWarps];
    float warp_best[kSearchWarps];
    unsigned int todo[kSearchWarps];
};

// One triangle's geometry shared by the passes.
struct TriBox {
    P3 r1, r2, tg;
    int row0, col0;
    int64_t ncol, ncell, n_in;
    bool listed;
};

// A screened correlation comes with a bound on its distance from the exact
// one.  The coordinates come from FP64 cubics (kCubicError pixel), the plane's
// height from the triangle's linear form, which the reference's plane equation
// differs from by its rounding at coordinates of 10^6 m over the plane's |C|
// (kept above kMinC; see plane_error).  What that is to the correlation follows
// from the steps between the texels against the samples' spread
// (ScreenAcc::corr): little for ordinary texture, 1e-5 and more for a steep
// triangle's few samples beside a bright texel.  kScreenBand covers the rest:
// one FP64 pass of sums over samples shifted by the first, and the float.
constexpr double kScreenBand = 1e-6;
constexpr float kMinC = 1e-2f;
constexpr float kCubicError = 2e-9f;
constexpr float kMaxError = 1e-6f;   // larger plane errors, in texels: the exact pass

// 1 / v from an FP32 seed and two Newton steps; `edge` is set where the seed
// is no finite non-zero float.
__device__ __forceinline__ double screen_rcp(double v, bool &edge) {
    const float f = __frcp_rn((float)v);
    if (!(fabsf(f) > 0.f && fabsf(f) < 3.0e38f)) edge = true;
    double r = (double)f;
    r = fma(r, fma(-v, r, 1.0), r);
    return fma(r, fma(-v, r, 1.0), r);
}

// Cubics j0 and j0 + 1 (a ratio's numerator and denominator) of one image at
// (lon, lat), with the reference's +-360 wrap: RPC00B's terms grouped by power
// of the normalised height.
__device__ void screen_poly(const double *rpc, double lon, double lat, int j0, double (*a)[4]) {
    double L = (lon - rpc[2]) / rpc[7];
    double P = (lat - rpc[3]) / rpc[8];
    if (L < -10.0 || L > 10.0) L = ((lon > 0 ? lon - 360 : lon + 360) - rpc[2]) / rpc[7];
    if (P < -10.0 || P > 10.0) P = ((lat > 0 ? lat - 360 : lat + 360) - rpc[3]) / rpc[8];
    const double LL = L * L, PP = P * P, LP = L * P;
#pragma unroll 1
    for (int j = j0; j < j0 + 2; ++j) {
        const double *c = rpc + 10 + 20 * j;
        double s = fma(c[1], L, c[0]);
        s = fma(c[2], P, s);
        s = fma(c[4], LP, s);
        s = fma(c[7], LL, s);
        s = fma(c[8], PP, s);
        s = fma(c[11], LL * L, s);
        s = fma(c[12], L * PP, s);
        s = fma(c[14], LL * P, s);
        a[j][0] = fma(c[15], PP * P, s);
        s = fma(c[5], L, c[3]);
        s = fma(c[6], P, s);
        s = fma(c[10], LP, s);
        s = fma(c[17], LL, s);
        a[j][1] = fma(c[18], PP, s);
        a[j][2] = fma(c[16], P, fma(c[13], L, c[9]));
        a[j][3] = c[19];
    }
}

// One pyramid coordinate from the scaled ratio v (clamped to [0, vmax] like
// the reference's) and whether it lies in an image of `size` texels (0 <= c,
// c + 1 < size).  `edge`: the coordinate lies within `near` (four errors) of a
// clamp or, unclamped, of a texel's position, the bounds among them, for the
// cubics to decide (a clamped one is exact).
__device__ __forceinline__ double screen_bound(double v, double vmax, double inv_s, double start,
                                               uint32_t size, float near, bool &in,
                                               bool &edge) {
    constexpr double kRint = 6755399441055744.0;   // 1.5 * 2^52
    const bool lo = v < 0, hi = v > vmax;
    const double c = fma(lo ? 0.0 : (hi ? vmax : v), inv_s, -start);
    const double last = (double)size - 1.0;
    if (!(fmin(fabs(v), fabs(v - vmax)) * inv_s > (double)near)) edge = true;
    if (!(lo || hi) && !(fabs(c - __dadd_rn(__dadd_rn(c, kRint), -kRint)) > (double)near)) edge = true;
    in = in && c >= 0 && c < last;
    return c;
}

// Pyramid coordinate of a screened cell at height z.
__device__ __forceinline__ double2 screen_coord(const double (*a)[4], const DevImage &im,
                                                const double *adj, double z, double hoff,
                                                double hinv, double inv_s, float near, bool &in,
                                                bool &edge) {
    const double H = (z - hoff) * hinv;
    double v[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) v[j] = fma(fma(fma(a[j][3], H, a[j][2]), H, a[j][1]), H, a[j][0]);
    const double y = adj[0] + fma(v[0] * screen_rcp(v[1], edge), im.rpc[5], im.rpc[0]);
    const double x = adj[1] + fma(v[2] * screen_rcp(v[3], edge), im.rpc[6], im.rpc[1]);
    const double ymax = __dadd_rn(im.rpc[0], __dmul_rn(im.rpc[5], 1.2));
    const double xmax = __dadd_rn(im.rpc[1], __dmul_rn(im.rpc[6], 1.2));
    return make_double2(screen_bound(x, xmax, inv_s, im.sx, im.w, near, in, edge),
                        screen_bound(y, ymax, inv_s, im.sy, im.h, near, in, edge));
}

// Bilinear samples of both planes of an image at (x, y), inside its bounds;
// step: raised to the largest step between the texels, of each plane.
__device__ __forceinline__ double2 screen_sample(const DevImage &im, double x, double y,
                                                 int (&step)[2]) {
    const int xi = __double2int_rd(x), yi = __double2int_rd(y);
    const double fx = x - (double)xi, fy = y - (double)yi;
    const int64_t p = (int64_t)yi * im.w + xi;
    double r[2];
#pragma unroll
    for (int k = 0; k < 2; ++k) {
        const uint16_t *I = (k ? im.mag : im.img) + p;
        const int a = __ldg(I), b = __ldg(I + 1), c = __ldg(I + im.w), d = __ldg(I + im.w + 1);
        const double t = fma(fx, (double)(b - a), (double)a);
        const double u = fma(fx, (double)(d - c), (double)c);
        r[k] = fma(fy, u - t, t);
        step[k] = max(step[k], max(max(a, b), max(c, d)) - min(min(a, b), min(c, d)));
    }
    return make_double2(r[0], r[1]);
}

struct ScreenAcc {
    double sl, sr, sll, srr, slr;
    __device__ void add(double l, double r) {
        sl += l;
        sr += r;
        sll = fma(l, l, sll);
        srr = fma(r, r, srr);
        slr = fma(l, r, slr);
    }
    // Correlate's value and in `off` what the coordinates' error can move it by:
    // samples off by 2 delta steps each (err: that times the root of their
    // number) turn the vectors by at most x in all, the correlation by x
    // times its sine and x^2.  A variance whose 1e-8 test the sums do not
    // decide, and an x that is not small, set `unsure`.
    __device__ double corr(double n, float err, int step, float &off,
                           bool &unsure) const {
        const double inv = 1.0 / n;
        const double vl = fma(-sl * inv, sl, sll), vr = fma(-sr * inv, sr, srr);
        const double cv = fma(-sl * inv, sr, slr);
        if ((vl > 1e-11 && vl < 1e-5) || (vr > 1e-11 && vr < 1e-5)) unsure = true;
        if (!(vl > 1e-8 && vr > 1e-8)) return -99.0;
        const double r = cv / sqrt(vl * vr);
        const float x = err * (float)step * (rsqrtf((float)vl) + rsqrtf((float)vr));
        const float c = (float)r;
        if (!(x < 0.1f)) unsure = true;
        off = x * (sqrtf(fmaxf(fmaf(-c, c, 1.f), 0.f)) + 2.f * x);
        return r;
    }
};

// What the reference's plane equation (exact_height) may differ from the
// triangle's linear form by, in metres of height: nine roundings of its terms,
// of the size `m` of the coordinates, over |C|, and of the normal, which a thin
// triangle magnifies, over the triangle.  v12, v13: its edges, len: the normal's
// length, den: its vertical component.  (A bound: FP32, whose own error the
// tenth of a rounding more covers.)
__device__ __forceinline__ float plane_error(float m, float3 v12, float3 v13, float den, float len) {
    const float a = sqrtf(v12.x * v12.x + v12.y * v12.y + v12.z * v12.z);
    const float b = sqrtf(v13.x * v13.x + v13.y * v13.y + v13.z * v13.z);
    return 1.01e-15f * (m + (a + b) * (a * b / len)) * len / fabsf(den);
}

// The correlation of the triangle at one height per thread: the mean over the
// target images, in *band the bound on its error and in *avg the mean number
// of samples; NaN where the screen does not decide it.  Every thread of the
// block takes part.
__device__ float screen_heights(const DevLevel &P, const double2 *__restrict__ lonlat,
                                const TriBox &T, double hgt, bool live, int *avg, float *band,
                                CellStage &st) {
    const int lane = threadIdx.x & 31;
    const double v12x = T.r2.x - T.r1.x, v12y = T.r2.y - T.r1.y, v12z = T.r2.z - T.r1.z;
    const double v13x = T.tg.x - T.r1.x, v13y = T.tg.y - T.r1.y, v13z = hgt - T.r1.z;
    const double den = v12x * v13y - v12y * v13x;
    bool unsure = !live;
    float delta;   // the coordinates' error in texels
    {
        const float3 v12 = make_float3((float)v12x, (float)v12y, (float)v12z);
        const float3 v13 = make_float3((float)v13x, (float)v13y, (float)v13z);
        const float nx = v12.y * v13.z - v12.z * v13.y, ny = v12.z * v13.x - v12.x * v13.z;
        const float nz = (float)den, len = sqrtf(nx * nx + ny * ny + nz * nz);
        // (a metre of height is at most a metre on the ground)
        const float m = (float)(fabs(T.r1.x) + fabs(T.r1.y) + fabs(T.r1.z));
        const float e = plane_error(m, v12, v13, nz, len) / (float)P.im_res;
        if (!(fabsf(nz) > kMinC * len) || !(e < kMaxError)) unsure = true;
        delta = kCubicError + e;
    }
    const double inv_s = 1.0 / (double)(1 << P.L);
    const DevImage &ri = P.im[P.ref];
    double sum_ncc = 0;
    float sum_off = 0.f;
    int n_img = 0, n_sum = 0;
    for (int ti = 1; ti < P.num_images; ++ti) {
        const DevImage &tI = P.im[ti];
        if (!tI.selected) continue;
        const double ho0 = ri.rpc[4], hi0 = 1.0 / ri.rpc[9], ho1 = tI.rpc[4], hi1 = 1.0 / tI.rpc[9];
        ScreenAcc acc[2];
        acc[0] = acc[1] = ScreenAcc{0, 0, 0, 0, 0};
        double2 s0 = make_double2(0, 0), s1 = make_double2(0, 0);
        int step[2] = {0, 0};   // of both images (a pair of registers less)
        int n = 0;
        const int64_t items = T.listed ? T.n_in : T.ncell;
        for (int64_t base = 0; base < items; base += 32) {
            // this chunk's cells: 32 of the list, or those of 32 box cells
            // that lie inside (every warp finds the same)
            unsigned m = base + 32 <= items ? 0xffffffffu : (1u << (int)(items - base)) - 1u;
            if (!T.listed) {
                const int64_t c = base + lane;
                m = __ballot_sync(0xffffffffu,
                                  c < items && cell_inside(P, T.r1, T.r2, T.tg, T.row0 + c / T.ncol,
                                                           T.col0 + c % T.ncol));
                if (!m) continue;
            }
            const int cnt = __popc(m);
            // a thread per cell, image and ratio (line, sample)
            const int k = threadIdx.x >> 2, im = (threadIdx.x >> 1) & 1, half = threadIdx.x & 1;
            if (k < cnt) {
                const int64_t cell = T.listed ? (int64_t)st.cell[base + k]
                                              : base + (int)__fns(m, 0, k + 1);
                const int64_t row = T.row0 + cell / T.ncol, col = T.col0 + cell % T.ncol;
                ScreenCell &S = st.sc[k];
                const double cx = __dadd_rn(__dmul_rn((double)col, P.grid_res), P.boundary[0]);
                const double cy = __dadd_rn(__dmul_rn((double)row, P.grid_res), P.boundary[1]);
                const double2 w = lonlat ? lonlat[row * P.grid_w + col] : ps2wgs_dev(P.param, cx, cy);
                screen_poly(im ? tI.rpc : ri.rpc, w.x, w.y, 2 * half, S.c[im]);
                if (im == 0 && half == 0) {
                    // barycentric weights of the second and the target vertex
                    const double dx = cx - T.r1.x, dy = cy - T.r1.y;
                    const double l2 = (dx * v13y - dy * v13x) / den;
                    const double l3 = (dy * v12x - dx * v12y) / den;
                    S.z1 = l3;
                    S.z0 = fma(l2, v12z, fma(-l3, T.r1.z, T.r1.z));
                }
            }
            __syncthreads();
#pragma unroll 2
            for (int c = 0; c < cnt; ++c) {
                const ScreenCell &S = st.sc[c];
                const double z = fma(hgt, S.z1, S.z0);
                bool in = true, edge = false;
                const double2 rp = screen_coord(S.c[0], ri, ri.adj, z, ho0, hi0, inv_s,
                                                4.f * delta, in, edge);
                const double2 tp = screen_coord(S.c[1], tI, ri.adj, z, ho1, hi1, inv_s,
                                                4.f * delta, in, edge);
                if (edge) unsure = true;
                in = in && !edge;
                // (a cell outside samples texel 0 and adds nothing)
                const double2 a = screen_sample(ri, in ? rp.x : 0.0, in ? rp.y : 0.0, step);
                const double2 b = screen_sample(tI, in ? tp.x : 0.0, in ? tp.y : 0.0, step);
                if (n == 0) {
                    s0 = a;
                    s1 = b;
                }
                acc[0].add(in ? a.x - s0.x : 0.0, in ? b.x - s1.x : 0.0);
                acc[1].add(in ? a.y - s0.y : 0.0, in ? b.y - s1.y : 0.0);
                n += in;
            }
            __syncthreads();   // the cells are rewritten by the next chunk
        }
        if (n >= 1) {
            double roh = 0, count = 0;
            const float err = 2.f * delta * sqrtf((float)n);
#pragma unroll
            for (int p = 0; p < 2; ++p) {
                float off = 0.f;
                const double c = acc[p].corr((double)n, err, step[p], off, unsure);
                // (the mean's error is at most the larger one's)
                sum_off += off;
                if (c != -99.0) {
                    roh += c;
                    count += 1.0;
                }
            }
            sum_ncc += count > 0 ? roh / count : -1.0;
            n_sum += n;
            ++n_img;
        }
    }
    *avg = n_img > 0 ? n_sum / n_img : -1;
    *band = (float)kScreenBand + 2e-7f + sum_off;
    if (unsure) return __int_as_float(0x7fc00000);
    return n_img > 0 ? (float)(sum_ncc / (double)n_img) : -2.f;
}

// The exact correlation of one height, in the reference's operation order
// (every thread of the block takes part and returns the same values): sum of
// the images' correlations, their number and the samples' number.  The cells
// are sampled a thread each; each of Correlate's sums is then formed by one
// thread in cell order.
template <int kThreads>
__device__ void exact_height(const DevLevel &P, const double2 *__restrict__ lonlat,
                             const TriBox &T, float iter_height, CellStage &st, double &sum_ncc,
                             int &count_ncc, int &sum_count_n) {
    const int t = threadIdx.x;
    const P3 T1 = T.r1, T2 = T.r2, T3 = {T.tg.x, T.tg.y, (double)iter_height};
    // the triangle's plane (the same for every cell of this height)
    const double v12x = __dadd_rn(T2.x, -T1.x), v12y = __dadd_rn(T2.y, -T1.y),
                 v12z = __dadd_rn(T2.z, -T1.z);
    const double v13x = __dadd_rn(T3.x, -T1.x), v13y = __dadd_rn(T3.y, -T1.y),
                 v13z = __dadd_rn(T3.z, -T1.z);
    double nx = __dadd_rn(__dmul_rn(v12y, v13z), -__dmul_rn(v12z, v13y));
    double ny = __dadd_rn(__dmul_rn(v12z, v13x), -__dmul_rn(v12x, v13z));
    double nz = __dadd_rn(__dmul_rn(v12x, v13y), -__dmul_rn(v12y, v13x));
    const double len =
        sqrt(__dadd_rn(__dadd_rn(__dmul_rn(nx, nx), __dmul_rn(ny, ny)), __dmul_rn(nz, nz)));
    bool plane_ok = len > 0;
    double A = 0, B = 0, C = 0, D = 0;
    if (plane_ok) {
        nx = __ddiv_rn(nx, len);
        ny = __ddiv_rn(ny, len);
        nz = __ddiv_rn(nz, len);
        A = nx;
        B = ny;
        C = nz;
        D = -__dadd_rn(__dadd_rn(__dmul_rn(A, T1.x), __dmul_rn(B, T1.y)), __dmul_rn(C, T1.z));
        plane_ok = C != 0;
    }
    sum_ncc = 0;
    count_ncc = 0;
    sum_count_n = 0;
    const int64_t n_items = T.listed ? T.n_in : T.ncell;
    for (int ti = 1; ti < P.num_images; ++ti) {
        if (!P.im[ti].selected) continue;
        // pass 0: sums for the means (threads 0..3); pass 1: centred products
        // (threads 0..5: intensity lr, ll, rr, magnitude lr, ll, rr)
        double ma = 0, mb = 0;
        int count_n = 0;
        for (int pass = 0; pass < 2; ++pass) {
            double acc = 0;
            int n = 0;
            for (int64_t base = 0; base < n_items; base += kCellCap) {
                const int chunk = (int)(n_items - base < kCellCap ? n_items - base : kCellCap);
                if (pass == 0 || !T.listed) {
                    for (int i = t; i < ((chunk + 31) & ~31); i += kThreads) {
                        double v[4] = {0, 0, 0, 0};
                        bool ok = false;
                        if (i < chunk) {
                            const int64_t c = T.listed ? (int64_t)st.cell[i] : base + i;
                            const int64_t row = T.row0 + c / T.ncol, col = T.col0 + c % T.ncol;
                            ok = (T.listed || cell_inside(P, T1, T2, T3, row, col)) &&
                                 cell_sample(P, lonlat, ti, plane_ok, A, B, C, D, row, col, v);
                        }
                        const unsigned m = __ballot_sync(0xffffffffu, ok);
#pragma unroll
                        for (int c = 0; c < 4; ++c) st.v[4 * i + c] = v[c];
                        if ((t & 31) == 0) st.valid[i >> 5] = m;
                    }
                    __syncthreads();
                }
                if (t < (pass == 0 ? 4 : 6)) {
                    const int p = t < 3 ? 0 : 2, kind = t < 3 ? t : t - 3;
                    for (int i = 0; i < chunk; ++i) {
                        if (!((st.valid[i >> 5] >> (i & 31)) & 1u)) continue;
                        if (pass == 0) {
                            acc = __dadd_rn(acc, st.v[4 * i + t]);
                            ++n;
                        } else {
                            const double l = __dadd_rn(st.v[4 * i + p], -ma);
                            const double r = __dadd_rn(st.v[4 * i + p + 1], -mb);
                            acc = __dadd_rn(acc, __dmul_rn(kind == 2 ? r : l, kind == 1 ? l : r));
                        }
                    }
                }
                if (!T.listed) __syncthreads();   // the samples are rewritten
            }
            if (t < 6) st.sum[t] = acc;
            if (t == 0 && pass == 0) st.count = n;
            __syncthreads();
            if (pass == 0) {
                count_n = st.count;
                if (count_n >= 1) {
                    const int p = t < 3 ? 0 : 2;
                    ma = __ddiv_rn(st.sum[p], (double)count_n);
                    mb = __ddiv_rn(st.sum[p + 1], (double)count_n);
                }
                __syncthreads();   // every thread has the sums
                if (count_n < 1) break;
            }
        }
        if (count_n >= 1) {
            double temp_roh = 0, count_roh = 0;
            const double ncc1 = corr_of(st.sum[0], st.sum[1], st.sum[2]);
            if (ncc1 != -99) {
                count_roh = __dadd_rn(count_roh, 1.0);
                temp_roh = __dadd_rn(temp_roh, ncc1);
            }
            const double ncc2 = corr_of(st.sum[3], st.sum[4], st.sum[5]);
            if (ncc2 != -99) {
                count_roh = __dadd_rn(count_roh, 1.0);
                temp_roh = __dadd_rn(temp_roh, ncc2);
            }
            const double ncc = count_roh > 0 ? __ddiv_rn(temp_roh, count_roh) : -1.0;
            sum_count_n += count_n;
            sum_ncc = __dadd_rn(sum_ncc, ncc);
            ++count_ncc;
        }
        __syncthreads();   // the sums and samples are rewritten
    }
}

// The triangle's box of grid cells (the reference recomputes it per height
// from the same x, y); false when every height skips it.
__device__ bool tri_box(const DevLevel &P, P3 r1, P3 r2, P3 tg, TriBox &T) {
    const double gs = P.grid_res;
    const int gw = (int)P.grid_w, gh = (int)P.grid_h;
    const double mn0 = dmin(dmin(r1.x, r2.x), tg.x), mn1 = dmin(dmin(r1.y, r2.y), tg.y);
    const double mx0 = dmax(dmax(r1.x, r2.x), tg.x), mx1 = dmax(dmax(r1.y, r2.y), tg.y);
    int pmin0 = (int)__dadd_rn(__ddiv_rn(__dadd_rn(mn0, -P.boundary[0]), gs), 0.5);
    int pmin1 = (int)__dadd_rn(__ddiv_rn(__dadd_rn(mn1, -P.boundary[1]), gs), 0.5);
    int pmax0 = (int)__dadd_rn(__ddiv_rn(__dadd_rn(mx0, -P.boundary[0]), gs), 0.5);
    int pmax1 = (int)__dadd_rn(__ddiv_rn(__dadd_rn(mx1, -P.boundary[1]), gs), 0.5);
    pmin0 -= 1;
    pmin1 -= 1;
    pmax0 += 1;
    pmax1 += 1;
    if (pmax0 >= gw) pmax0 = gw - 1;
    if (pmax1 >= gh) pmax1 = gh - 1;
    if (pmin0 < 0) pmin0 = 0;
    if (pmin1 < 0) pmin1 = 0;
    if (!(pmax1 - pmin1 > 0 && pmax0 - pmin0 > 0)) return false;
    T.r1 = r1;
    T.r2 = r2;
    T.tg = tg;
    T.row0 = pmin1;
    T.col0 = pmin0;
    T.ncol = pmax0 - pmin0 + 1;
    T.ncell = (int64_t)(pmax1 - pmin1 + 1) * T.ncol;
    T.n_in = 0;
    T.listed = true;
    return true;
}

// VerticalLineLocus_Ortho for one triangle, by one block (every thread
// returns the same result); st: the block's staging.
//
// The search keeps the first height of the largest correlation among those
// that pass their threshold, so only heights that can be it need the
// reference's exact value.  All heights are screened first, a thread each
// (FP64 cubics per cell, one pass of FP64 sums), and those whose screened
// correlation lies within the band of the best, or does not decide, are
// evaluated exactly, in order: about one in a hundred.  A few heights are all
// evaluated exactly (few_heights).  Ortho_blunder on a 700 x 690 grid with 9.7 k points (107 heights of 25 cells per search, 4
// rounds): 27.0 ms of search with every height evaluated exactly by a warp,
// 2.0 ms; bound by the latency of the FP64 chains (12 warps per SM, FP64 pipe
// 26 % busy).  Resident blocks 3, 4 or 5 per SM and one or two cells per
// iteration: 2.9 to 3.1 ms for the whole call.
// The step of the swept heights, and their number for a target node.
__device__ __forceinline__ double height_step(const DevLevel &P, double mpp) {
    if (mpp > 3) mpp = 3;
    if (mpp < 1) mpp = 1;
    return __dmul_rn(P.im_res, mpp);
}
__device__ __forceinline__ int height_count(const DevLevel &P, double hstep, int64_t target_index) {
    const int lo = P.gp3[target_index].minHeight, hi = P.gp3[target_index].maxHeight;
    return (int)__ddiv_rn((double)(hi - lo), hstep) + 1;
}

// Heights so few that the screen, which costs the same up to 128, costs more
// than their exact values: seven over a small box, four over a larger one
// (whole calls on a 700 x 690 grid, all evaluated exactly against all screened:
// 9.7 k points 3 heights 1.24 and 2.37 ms, 6 heights 1.85 and 2.38; 2.4 k points
// 2.24 and 2.90, 3.79 and 2.77; 483 points 13.3 and 19.7, 25.9 and 19.6).
__device__ __forceinline__ bool few_heights(int n_heights, int64_t ncell) {
    return n_heights <= (ncell < 160 ? 7 : 4);
}

template <int kThreads>
__device__ SearchOut ortho_search(const DevLevel &P, const double2 *__restrict__ lonlat,
                                  double mpp, P3 r1, P3 r2, P3 tg, int64_t target_index,
                                  CellStage &st) {
    constexpr int kWarps = kThreads / 32;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    SearchOut o{-9999.0, 0.0, 0};
    double f_ncc = -1.0;
    double selected_count = 0;
    const double hstep = height_step(P, mpp);
    const int start_h = P.gp3[target_index].minHeight;
    const int n_heights = height_count(P, hstep, target_index);
    const int th_count = 10;
    const int min_th_count = P.L < 4 ? 0 : 2;
    const double min_th_sncc = P.L < 4 ? 0.5 : 0.2;
    TriBox T;
    if (!tri_box(P, r1, r2, tg, T)) return o;
    // the inside cells, in cell order
    for (int64_t base = 0; base < T.ncell; base += kThreads) {
        const int64_t i = base + threadIdx.x;
        const bool in = i < T.ncell &&
                        cell_inside(P, r1, r2, tg, T.row0 + i / T.ncol, T.col0 + i % T.ncol);
        const unsigned m = __ballot_sync(0xffffffffu, in);
        if (lane == 0) st.warp_n[warp] = __popc(m);
        __syncthreads();
        int64_t at = T.n_in + __popc(m & ((1u << lane) - 1u));
        for (int w = 0; w < kWarps; ++w) {
            if (w < warp) at += st.warp_n[w];
            T.n_in += st.warp_n[w];
        }
        if (in && at < kCellCap) st.cell[at] = (int32_t)i;
        __syncthreads();
    }
    T.listed = T.n_in <= kCellCap;
    // no cell, or a plane without a vertical component (the reference's C is
    // 0): no height has samples
    if (T.n_in == 0 || __dmul_rn(r2.x - r1.x, tg.y - r1.y) == __dmul_rn(r2.y - r1.y, tg.x - r1.x))
        return o;
    // the height of index kh (the reference's float iter_height)
    auto height = [&](int kh) {
        return (float)__dadd_rn((double)start_h, __dmul_rn((double)kh, hstep));
    };
    // the exact value of one height, taken where it is the best so far
    auto take = [&](int kh) {
        const float iter_height = height(kh);
        double sum_ncc;
        int count_ncc, sum_count_n;
        exact_height<kThreads>(P, lonlat, T, iter_height, st, sum_ncc, count_ncc, sum_count_n);
        if (count_ncc <= 0) return;
        const double sncc = __ddiv_rn(sum_ncc, (double)count_ncc);
        const double cnt = __ddiv_rn((double)sum_count_n, (double)count_ncc);
        if (sum_count_n / count_ncc >= th_count) {
            if (sncc > min_th_sncc && f_ncc < sncc) {
                f_ncc = sncc;
                o.f_height = (double)iter_height;
                selected_count = cnt;
                o.f_sncc = f_ncc;
            }
        } else if (sum_count_n / count_ncc > min_th_count) {
            if (sncc > __dadd_rn(min_th_sncc, 0.2) && f_ncc < sncc) {
                f_ncc = sncc;
                o.f_height = __ddiv_rn(__dadd_rn(r1.z, r2.z), 2.0);
                selected_count = cnt;
                o.f_sncc = f_ncc;
            }
        }
    };
    for (int chunk = 0; chunk < n_heights; chunk += kThreads) {
        const int kh = chunk + threadIdx.x;
        const bool live = kh < n_heights;
        bool can = live;
        if constexpr (kThreads == kSearchThreads) {
            if (!few_heights(n_heights, T.ncell)) {
                // screen: a height that cannot pass its threshold is -2, one that
                // the screen does not decide NaN
                int avg;
                float band;
                float a = screen_heights(P, lonlat, T, (double)height(live ? kh : chunk), live, &avg,
                                         &band, st);
                float sure = -2.f;   // what the best that surely passes is at least
                if (!live) {
                    a = -2.f;
                } else if (!isnan(a)) {
                    const double th = avg >= th_count ? min_th_sncc : min_th_sncc + 0.2;
                    if (avg <= min_th_count && avg < th_count)
                        a = -2.f;
                    else if (!((double)a > th - (double)band))
                        a = -2.f;
                    else if ((double)a > th + (double)band)
                        sure = a - band;
                }
#pragma unroll
                for (int d = 16; d; d >>= 1)
                    sure = fmaxf(sure, __shfl_xor_sync(0xffffffffu, sure, d));
                if (lane == 0) st.warp_best[warp] = sure;
                __syncthreads();
                for (int w = 0; w < kWarps; ++w) sure = fmaxf(sure, st.warp_best[w]);
                // (a value that cannot beat the best so far is left out, NaN
                // compares false)
                can = isnan(a) ||
                      (a > -2.f && a + band >= sure && !(a + band < (float)f_ncc - 2e-7f));
            }
        }
        const unsigned m = __ballot_sync(0xffffffffu, can);
        if (lane == 0) st.todo[warp] = m;
        __syncthreads();
        // exact: the heights that can be the first of the largest correlation
        for (int w = 0; w < kWarps; ++w) {
            unsigned todo = st.todo[w];
            while (todo) {
                const int b = __ffs(todo) - 1;
                todo &= todo - 1;
                take(chunk + 32 * w + b);
            }
        }
        __syncthreads();   // the masks are rewritten by the next chunk
    }
    o.selected = (int)selected_count;
    return o;
}

// Grid node of a matched point (setsm_code.cpp:8073-8075).
__device__ __forceinline__ int64_t node_of(const DevLevel &P, const vll_point3 &p) {
    const int64_t r = (int64_t)__dadd_rn(__ddiv_rn(__dadd_rn(p.y, -P.boundary[1]), P.grid_res), 0.5);
    const int64_t c = (int64_t)__dadd_rn(__ddiv_rn(__dadd_rn(p.x, -P.boundary[0]), P.grid_res), 0.5);
    return r * P.grid_w + c;
}

__device__ __forceinline__ bool anchored(uint8_t f) { return f == 1 || f == 3; }

// Single search (the VerticalLineLocus_Ortho entry point): one block.
__global__ void __launch_bounds__(kSearchThreads) ortho_search_kernel(
    const DevLevel *__restrict__ Pp, double mpp, const vll_point3 *pts3, int64_t target_index,
    double *out) {
    const DevLevel &P = *Pp;
    __shared__ CellStage st;
    const SearchOut o = ortho_search<kSearchThreads>(P, nullptr, mpp, P3{pts3[0].x, pts3[0].y, pts3[0].z},
                                     P3{pts3[1].x, pts3[1].y, pts3[1].z},
                                     P3{pts3[2].x, pts3[2].y, pts3[2].z}, target_index, st);
    if (threadIdx.x == 0) {
        out[0] = o.f_height;
        out[1] = o.f_sncc;
        out[2] = (double)o.selected;
    }
}

// A triangle with two anchored vertices as Ortho_blunder orders it.
struct SearchTri {
    P3 r1, r2, tg;
    int64_t node;     // the target vertex's grid node
    uint32_t point;   // and point
};

// Ortho_blunder, first (parallel) loop over the triangles (setsm_code.cpp:
// 8060-8146): which triangle takes which vertex as target.
__device__ SearchTri search_tri(const DevLevel &P, const vll_point3 *pts, const vll_tri &tr,
                                const int64_t *nodes) {
    const vll_point3 &p0 = pts[tr.a], &p1 = pts[tr.b], &p2 = pts[tr.c];
    const P3 a = {p0.x, p0.y, p0.z}, b = {p1.x, p1.y, p1.z}, c = {p2.x, p2.y, p2.z};
    if (P.gp3[nodes[0]].anchor_flag == 2) return SearchTri{b, c, a, nodes[0], tr.a};
    if (P.gp3[nodes[1]].anchor_flag == 2) return SearchTri{a, c, b, nodes[1], tr.b};
    return SearchTri{a, b, c, nodes[2], tr.c};
}

// Boxes of this many cells are searched first: their searches are the
// longest, and one left for last would run alone.
constexpr int64_t kLargeBox = 512;

// The triangles to search this round, listed in any order: those with a
// large box from the front, the others from the back, and in `few` those of
// few heights and a box that is not large; n_list: their counts (others,
// large, [3] few).
__global__ void tri_select_kernel(const DevLevel *__restrict__ Pp, double mpp, const vll_point3 *pts,
                                  int64_t n_pts, const vll_tri *tris, int64_t n_tris,
                                  const int64_t *tri_nodes, uint8_t *tris_check,
                                  uint32_t *sort_key, int32_t *list, int32_t *few, int *n_list) {
    const DevLevel &P = *Pp;
    const int lane = threadIdx.x & 31;
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    const int64_t n_round = (n_tris + 31) & ~(int64_t)31;
    for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < n_round; t += stride) {
        int kind = 0;   // 1 search, 2 search early, 3 few heights
        if (t < n_tris) {
            sort_key[t] = (uint32_t)n_pts;
            const vll_tri tr = tris[t];
            if (tris_check[t] == 0 && tr.a < n_pts && tr.b < n_pts && tr.c < n_pts) {
                int nf = 0;
                for (int k = 0; k < 3; ++k)
                    nf += anchored(P.gp3[tri_nodes[3 * t + k]].anchor_flag);
                if (nf == 3) {
                    tris_check[t] = 1;
                } else if (nf == 2) {
                    const SearchTri q = search_tri(P, pts, tr, tri_nodes + 3 * t);
                    TriBox T;
                    if (tri_box(P, q.r1, q.r2, q.tg, T))
                        kind = T.ncell >= kLargeBox ? 2
                               : few_heights(height_count(P, height_step(P, mpp), q.node), T.ncell) ? 3
                                                                                                   : 1;
                }
            }
        }
#pragma unroll
        for (int k = 1; k <= 3; ++k) {
            const unsigned m = __ballot_sync(0xffffffffu, kind == k);
            if (!m) continue;
            int at = 0;
            if (lane == __ffs(m) - 1) at = atomicAdd(n_list + (k == 3 ? 3 : k - 1), __popc(m));
            at = __shfl_sync(0xffffffffu, at, __ffs(m) - 1) + __popc(m & ((1u << lane) - 1u));
            if (kind == k) {
                if (k == 3)
                    few[at] = (int32_t)t;
                else
                    list[k == 2 ? at : (int)n_tris - 1 - at] = (int32_t)t;
            }
        }
    }
}

// The listed triangles, a block each, from a queue.
__global__ void __launch_bounds__(kSearchThreads, 3) tri_search_kernel(
    const DevLevel *__restrict__ Pp, double mpp, const vll_point3 *pts, const vll_tri *tris,
    int64_t n_tris, const int64_t *tri_nodes, double *hgt, int32_t *cnt, uint32_t *sort_key,
    const int32_t *list, int *n_list, const double2 *__restrict__ lonlat) {
    const DevLevel &P = *Pp;
    __shared__ CellStage st;
    __shared__ int next;
    const int n_small = n_list[0], n_large = n_list[1];
    for (;;) {
        if (threadIdx.x == 0) next = atomicAdd(n_list + 2, 1);
        __syncthreads();
        const int i = next;
        __syncthreads();
        if (i >= n_small + n_large) return;
        const int64_t t = i < n_large ? list[i] : list[(int)n_tris - 1 - (i - n_large)];
        const SearchTri q = search_tri(P, pts, tris[t], tri_nodes + 3 * t);
        const SearchOut o = ortho_search<kSearchThreads>(P, lonlat, mpp, q.r1, q.r2, q.tg, q.node, st);
        if (threadIdx.x == 0 && o.f_height != -9999.0) {
            hgt[t] = o.f_height;
            cnt[t] = o.selected;
            sort_key[t] = q.point;
        }
        __syncthreads();   // the staging is rewritten by the next triangle
    }
}

// The listed triangles of few heights, a warp each, from a queue: a block's
// other warps would wait for most of an exact evaluation (700 x 690 grid, 145 k
// points, 3 heights each: 10.1 ms screened by blocks, 3.6 here).
__global__ void __launch_bounds__(32, 12) tri_few_kernel(
    const DevLevel *__restrict__ Pp, double mpp, const vll_point3 *pts, const vll_tri *tris,
    const int64_t *tri_nodes, double *hgt, int32_t *cnt, uint32_t *sort_key, const int32_t *few,
    int *n_list, const double2 *__restrict__ lonlat) {
    const DevLevel &P = *Pp;
    __shared__ CellStage st;
    const int n = n_list[3];
    for (;;) {
        int i = 0;
        if (threadIdx.x == 0) i = atomicAdd(n_list + 4, 1);
        i = __shfl_sync(0xffffffffu, i, 0);
        if (i >= n) return;
        const int64_t t = few[i];
        const SearchTri q = search_tri(P, pts, tris[t], tri_nodes + 3 * t);
        const SearchOut o = ortho_search<32>(P, lonlat, mpp, q.r1, q.r2, q.tg, q.node, st);
        if (threadIdx.x == 0 && o.f_height != -9999.0) {
            hgt[t] = o.f_height;
            cnt[t] = o.selected;
            sort_key[t] = q.point;
        }
        __syncwarp();   // the staging is rewritten by the next triangle
    }
}

// Record-breakers of the running maximum per target point: triangles sorted
// by point (stable, so in triangle order within a point).  The last record
// sets the point's height; each record anchors the point's grid node, and
// the node remembers the first triangle that anchored it.
__global__ void records_kernel(const uint32_t *skey, const int32_t *sval, int64_t n, uint32_t none,
                               const int32_t *cnt, const double *hgt, const int64_t *tnode_of_pt,
                               vll_point3 *pts, uint8_t *rec, unsigned long long *first_anchor,
                               int *any_record) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
         i += (int64_t)gridDim.x * blockDim.x) {
        const uint32_t k = skey[i];
        if (k == none || (i > 0 && skey[i - 1] == k)) continue;
        int32_t best = 0;
        int32_t last = -1, first = -1;
        for (int64_t j = i; j < n && skey[j] == k; ++j) {
            const int32_t t = sval[j];
            if (best < cnt[t]) {   // com_count[target] < selected_count[tcnt]
                best = cnt[t];
                rec[t] = 1;
                last = t;
                if (first < 0) first = t;
            }
        }
        if (last >= 0) {
            pts[k].z = hgt[last];
            pts[k].flag = 0;
            atomicMin(first_anchor + tnode_of_pt[k], (unsigned long long)first);
            *any_record = 1;
        }
    }
}

// Second half of the apply pass (setsm_code.cpp:8164-8212) for every
// triangle still unchecked: records are checked, and a triangle whose three
// nodes are anchored (before this pass, or by a record of a triangle at or
// before it) is checked; anchored vertices lose their flag.
__global__ void apply_kernel(const DevLevel *__restrict__ Pp, vll_point3 *pts, int64_t n_pts,
                             const vll_tri *tris, int64_t n_tris, const int64_t *tri_nodes,
                             uint8_t *tris_check, const uint8_t *rec,
                             const unsigned long long *first_anchor) {
    const DevLevel &P = *Pp;
    for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < n_tris;
         t += (int64_t)gridDim.x * blockDim.x) {
        if (tris_check[t] != 0) continue;
        const vll_tri tr = tris[t];
        if (!(tr.a < n_pts && tr.b < n_pts && tr.c < n_pts)) continue;
        bool done = rec[t] != 0;
        const uint32_t v[3] = {tr.a, tr.b, tr.c};
        int nf = 0;
        for (int k = 0; k < 3; ++k) {
            const int64_t nd = tri_nodes[3 * t + k];
            if (anchored(P.gp3[nd].anchor_flag) || first_anchor[nd] <= (unsigned long long)t) {
                ++nf;
                pts[v[k]].flag = 0;
            }
        }
        if (nf == 3) done = true;
        if (done) tris_check[t] = 1;
    }
}

// Anchors the record nodes (anchor_flag = 3) and clears the per-node and
// per-triangle marks for the next iteration.
__global__ void anchor_kernel(vll_ugrid *gp3, int64_t n_nodes, unsigned long long *first_anchor,
                              uint8_t *rec, int64_t n_tris) {
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n_nodes; i += stride) {
        if (first_anchor[i] != ~0ull) {
            gp3[i].anchor_flag = 3;
            first_anchor[i] = ~0ull;
        }
    }
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n_tris; i += stride)
        rec[i] = 0;
}

// Longitude / latitude of every grid cell position (col * gs + B0,
// row * gs + B1), the map projection VerticalLineLocus_Ortho applies to every
// cell it samples: computed once per call instead of per height and image.
__global__ void lonlat_kernel(const DevLevel *__restrict__ Pp, double2 *lonlat) {
    const DevLevel &P = *Pp;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < P.n_nodes;
         i += (int64_t)gridDim.x * blockDim.x) {
        const int64_t row = i / P.grid_w, col = i % P.grid_w;
        const double cx = __dadd_rn(__dmul_rn((double)col, P.grid_res), P.boundary[0]);
        const double cy = __dadd_rn(__dmul_rn((double)row, P.grid_res), P.boundary[1]);
        lonlat[i] = ps2wgs_dev(P.param, cx, cy);
    }
}

// Grid nodes of every triangle vertex and of every point, and the triangles'
// indices; flags vertices whose node lies outside the grid.
__global__ void nodes_kernel(const DevLevel *__restrict__ Pp, const vll_point3 *pts, int64_t n_pts,
                             const vll_tri *tris, int64_t n_tris, int64_t *tri_nodes,
                             int64_t *pt_nodes, int32_t *tri_index, int *bad) {
    const DevLevel &P = *Pp;
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n_pts; i += stride) {
        const int64_t nd = node_of(P, pts[i]);
        pt_nodes[i] = nd;
    }
    for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < n_tris; t += stride) {
        const vll_tri tr = tris[t];
        tri_index[t] = (int32_t)t;   // the sort's value
        const uint32_t v[3] = {tr.a, tr.b, tr.c};
        for (int k = 0; k < 3; ++k) {
            int64_t nd = 0;
            if (v[k] < n_pts) {
                nd = node_of(P, pts[v[k]]);
                if (nd < 0 || nd >= P.n_nodes) {
                    atomicExch(bad, 1);
                    nd = 0;
                }
            }
            tri_nodes[3 * t + k] = nd;
        }
    }
}

unsigned blocks_for(int64_t n, int threads) {
    int64_t b = (n + threads - 1) / threads;
    if (b < 1) b = 1;
    if (b > 148 * 32) b = 148 * 32;
    return (unsigned)b;
}

}  // namespace

cudaError_t launch_ortho_search(const DevLevel *dP, double mpp, const vll_point3 *d_pts3,
                                int64_t target_index, double *d_out, cudaStream_t s) {
    ortho_search_kernel<<<1, kSearchThreads, 0, s>>>(dP, mpp, d_pts3, target_index, d_out);
    return cudaGetLastError();
}

size_t ortho_blunder_scratch(int64_t n_pts, int64_t n_tris, int64_t n_nodes) {
    size_t tmp = 0;
    cub::DeviceRadixSort::SortPairs(nullptr, tmp, (const uint32_t *)nullptr, (uint32_t *)nullptr,
                                    (const int32_t *)nullptr, (int32_t *)nullptr, (int)n_tris);
    auto al = [](size_t b) { return (b + 255) & ~(size_t)255; };
    return al(tmp) + al(n_tris * 24) + al(n_pts * 8) + al(n_tris) * 2 + al(n_tris * 8) +
           al(n_tris * 4) * 6 + al(n_nodes * 8) + al(32) + al(n_nodes * 16);
}

// Ortho_blunder on device data (scratch of ortho_blunder_scratch bytes).
// Returns the number of iterations in *iterations, or an error.
cudaError_t run_ortho_blunder(const DevLevel *dP, const DevLevel &hP, double mpp, vll_point3 *pts,
                              int64_t n_pts, const vll_tri *tris, int64_t n_tris,
                              vll_ugrid *gp3, void *scratch, size_t scratch_bytes,
                              int *iterations, int *bad_input, cudaStream_t s) {
    *iterations = 0;
    *bad_input = 0;
    char *p = (char *)scratch;
    auto al = [](size_t b) { return (b + 255) & ~(size_t)255; };
    auto take = [&](size_t b) {
        void *r = p;
        p += al(b);
        return r;
    };
    size_t tmp_bytes = 0;
    cub::DeviceRadixSort::SortPairs(nullptr, tmp_bytes, (const uint32_t *)nullptr,
                                    (uint32_t *)nullptr, (const int32_t *)nullptr,
                                    (int32_t *)nullptr, (int)n_tris);
    void *tmp = take(tmp_bytes);
    int64_t *tri_nodes = (int64_t *)take(n_tris * 24);
    int64_t *pt_nodes = (int64_t *)take(n_pts * 8);
    uint8_t *tris_check = (uint8_t *)take(n_tris);
    uint8_t *rec = (uint8_t *)take(n_tris);
    double *hgt = (double *)take(n_tris * 8);
    int32_t *cnt = (int32_t *)take(n_tris * 4);
    uint32_t *key = (uint32_t *)take(n_tris * 4);
    uint32_t *skey = (uint32_t *)take(n_tris * 4);
    int32_t *val = (int32_t *)take(n_tris * 4);
    int32_t *sval = (int32_t *)take(n_tris * 4);
    int32_t *list = (int32_t *)take(n_tris * 4);
    unsigned long long *first_anchor = (unsigned long long *)take(hP.n_nodes * 8);
    // [0] any record, [1] bad input, [2..6] listed triangles: others, large
    // box, the search's queue, few heights, their queue
    int *flags = (int *)take(32);
    double2 *lonlat = (double2 *)take(hP.n_nodes * 16);
    if ((size_t)(p - (char *)scratch) > scratch_bytes) return cudaErrorInvalidValue;
    cudaError_t e;
    if ((e = cudaMemsetAsync(tris_check, 0, n_tris, s))) return e;
    if ((e = cudaMemsetAsync(rec, 0, n_tris, s))) return e;
    if ((e = cudaMemsetAsync(first_anchor, 0xff, hP.n_nodes * 8, s))) return e;
    if ((e = cudaMemsetAsync(flags, 0, 32, s))) return e;
    nodes_kernel<<<blocks_for(n_pts > n_tris ? n_pts : n_tris, 256), 256, 0, s>>>(
        dP, pts, n_pts, tris, n_tris, tri_nodes, pt_nodes, val, flags + 1);
    lonlat_kernel<<<blocks_for(hP.n_nodes, 128), 128, 0, s>>>(dP, lonlat);
    int hflags[2] = {0, 0};
    if ((e = cudaMemcpyAsync(hflags, flags, 8, cudaMemcpyDeviceToHost, s))) return e;
    if ((e = cudaStreamSynchronize(s))) return e;
    if (hflags[1]) {
        *bad_input = 1;
        return cudaSuccess;
    }
    int end_bit = 1;
    while (end_bit < 32 && ((uint64_t)1 << end_bit) <= (uint64_t)n_pts) ++end_bit;
    int dev = 0, sms = 148, per_sm = 1;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, tri_search_kernel, kSearchThreads, 0);
    const unsigned search_blocks =
        (unsigned)std::min<int64_t>(n_tris, (int64_t)sms * std::max(per_sm, 1));
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, tri_few_kernel, 32, 0);
    const unsigned few_blocks =
        (unsigned)std::min<int64_t>(n_tris, (int64_t)sms * std::max(per_sm, 1));
    // (the sort's output is free until the sort)
    int32_t *few = sval;
    for (int it = 0; it < 200; ++it) {
        *iterations = it + 1;
        if ((e = cudaMemsetAsync(flags, 0, 32, s))) return e;
        tri_select_kernel<<<blocks_for(n_tris, 256), 256, 0, s>>>(
            dP, mpp, pts, n_pts, tris, n_tris, tri_nodes, tris_check, key, list, few, flags + 2);
        tri_search_kernel<<<search_blocks, kSearchThreads, 0, s>>>(
            dP, mpp, pts, tris, n_tris, tri_nodes, hgt, cnt, key, list, flags + 2, lonlat);
        tri_few_kernel<<<few_blocks, 32, 0, s>>>(dP, mpp, pts, tris, tri_nodes, hgt, cnt, key, few,
                                                 flags + 2, lonlat);
        if ((e = cudaGetLastError())) return e;
        if ((e = cub::DeviceRadixSort::SortPairs(tmp, tmp_bytes, key, skey, val, sval, (int)n_tris,
                                                 0, end_bit, s)))
            return e;
        records_kernel<<<blocks_for(n_tris, 256), 256, 0, s>>>(
            skey, sval, n_tris, (uint32_t)n_pts, cnt, hgt, pt_nodes, pts, rec, first_anchor, flags);
        apply_kernel<<<blocks_for(n_tris, 256), 256, 0, s>>>(dP, pts, n_pts, tris, n_tris,
                                                             tri_nodes, tris_check, rec,
                                                             first_anchor);
        anchor_kernel<<<blocks_for(hP.n_nodes > n_tris ? hP.n_nodes : n_tris, 256), 256, 0, s>>>(
            gp3, hP.n_nodes, first_anchor, rec, n_tris);
        if ((e = cudaGetLastError())) return e;
        if ((e = cudaMemcpyAsync(hflags, flags, 4, cudaMemcpyDeviceToHost, s))) return e;
        if ((e = cudaStreamSynchronize(s))) return e;
        if (!hflags[0]) break;   // no record: check_ortho_cal false, the loop stops
    }
    return cudaSuccess;
}

}  // namespace vll
