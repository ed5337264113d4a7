// vll_ortho.cu -- the orthoimage-window variants of VerticalLineLocus:
// VerticalLineLocus_seeddem (setsm_code.cpp:7720-7880) and
// VerticalLineLocus_blunder (:7882-8026).  Both project every ortho pixel of
// the tile through the RPCs at its grid node's height (SetOrthoImageCoord,
// :6550-6670, at the matched level or at the blunder-selected level) and run
// the multi-window NCC of each grid node over the ortho pixels around it; the
// seed-DEM pass widens or voids the node's height range where that NCC is
// low, the blunder pass records it (ortho_ncc, Mean_ortho_ncc, one float per
// node).  FP64 in the reference's operation order (compiled -fmad=false).
#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstring>
#include <cuda_runtime.h>

#include "vll_exact.cuh"
#include "vll_geo.cuh"
#include "vll_internal.h"
#include "vll_split.h"

namespace vll {

namespace {

// SetOrthoImageCoord for a raster of ow x oh pixels at im_res; `use_b`
// selects the blunder level's pyramid (py_BStartpos, blunder_selected_level).
__global__ void __launch_bounds__(256) ortho_raster_kernel(const DevLevel *__restrict__ Pp,
                                                           double2 *const *__restrict__ cd,
                                                           int64_t ow, int64_t oh, double im_res,
                                                           int use_b) {
    const DevLevel &P = *Pp;
    const double *B = P.boundary;
    const int64_t total = ow * oh;
    for (int64_t it = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; it < total;
         it += (int64_t)gridDim.x * blockDim.x) {
        const int64_t row = it / ow;
        const int64_t col = it % ow;
        const double tX = __dadd_rn(B[0], __dmul_rn((double)col, im_res));
        const double tY = __dadd_rn(B[1], __dmul_rn((double)row, im_res));
        const int64_t t_col = (int64_t)__ddiv_rn(__dadd_rn(tX, -B[0]), P.grid_res);
        const int64_t t_row = (int64_t)__ddiv_rn(__dadd_rn(tY, -B[1]), P.grid_res);
        const int64_t pt = t_row * P.grid_w + t_col;
        if (!(pt < P.n_nodes && t_col < P.grid_w && t_row < P.grid_h)) continue;
        const float Hh = P.gp3[pt].Height;
        if (Hh == -1000) continue;
        const double2 w = ps2wgs_dev(P.param, tX, tY);
        for (int ti = 0; ti < P.num_images; ++ti) {
            const DevImage &im = P.im[ti];
            if (!im.selected) continue;
            const double2 ic = rpc_project(im.rpc, im.adj, w.x, w.y, (double)Hh);
            cd[ti][it] = use_b ? to_pyramid(ic, im.sxb, im.syb, P.blunder_level)
                               : to_pyramid(ic, im.sx, im.sy, P.L);
        }
    }
}

// UGRID.ortho_ncc[ti] = v with the reference's indexing: the array has two
// entries, so ti = 2..4 land on the record's following fields (Mean_ortho_ncc,
// the flags, padding).  ti >= 5 would reach the next node's record, a write
// that races with that node's own update in the reference; it is not made.
__device__ __forceinline__ void set_ortho_ncc(vll_ugrid &g, int ti, int16_t v) {
    const int byte = 10 + 2 * ti;
    if (byte + 2 <= (int)sizeof(vll_ugrid))
        *reinterpret_cast<int16_t *>(reinterpret_cast<unsigned char *>(&g) + byte) = v;
}

struct OrthoArgs {
    double2 *const *cd;     // [num_images] rasters
    int64_t ow, oh;
    double im_res;
    int H;
    int r2max;              // window offsets kept: row^2 + col^2 <= r2max
    int use_b;              // sample the blunder level's images
};

// Multi-window NCC of node pt against image ti over the ortho pixels of its
// window (the window loops of setsm_code.cpp:7772-7805 / :7958-7996).
__device__ void ortho_node_ncc(const DevLevel &P, const OrthoArgs &A, int64_t pt, int ti,
                               double &ncc, int &cnt0) {
    const DevImage &ri = P.im[P.ref], &tI = P.im[ti];
    PatchSrc S;
    if (A.use_b) {
        S = PatchSrc{ri.img_b, ri.mag_b, tI.img_b, tI.mag_b, ri.wb, ri.hb, tI.wb, tI.hb};
    } else {
        S = PatchSrc{ri.img, ri.mag, tI.img, tI.mag, ri.w, ri.h, tI.w, tI.h};
    }
    const double gx = P.grid_pts[2 * pt], gy = P.grid_pts[2 * pt + 1];
    const double *B = P.boundary;
    const double2 *cr = A.cd[P.ref], *ct = A.cd[ti];
    double count = 0, sum = 0;
    cnt0 = 0;
    multi_ncc(S, A.H,
              [&](int row, int col, double2 &pl, double2 &pr) -> bool {
                  if (row * row + col * col > A.r2max) return false;
                  const double tX = __dadd_rn(gx, __dmul_rn((double)col, A.im_res));
                  const double tY = __dadd_rn(gy, __dmul_rn((double)row, A.im_res));
                  const int64_t t_col = (int64_t)__ddiv_rn(__dadd_rn(tX, -B[0]), A.im_res);
                  const int64_t t_row = (int64_t)__ddiv_rn(__dadd_rn(tY, -B[1]), A.im_res);
                  const int64_t pit = t_row * A.ow + t_col;
                  const int64_t tt_col = (int64_t)__ddiv_rn(__dadd_rn(tX, -B[0]), P.grid_res);
                  const int64_t tt_row = (int64_t)__ddiv_rn(__dadd_rn(tY, -B[1]), P.grid_res);
                  const int64_t pdem = tt_row * P.grid_w + tt_col;
                  if (!(pit >= 0 && pit < A.ow * A.oh && t_col >= 0 && t_col < A.ow &&
                        t_row >= 0 && t_row < A.oh && pdem >= 0 && pdem < P.n_nodes &&
                        tt_col >= 0 && tt_col < P.grid_w && tt_row >= 0 && tt_row < P.grid_h &&
                        cr != nullptr && ct != nullptr))
                      return false;
                  if (P.gp3[pdem].Height == -1000) return false;
                  pl = cr[pit];
                  pr = ct[pit];
                  return true;
              },
              count, sum, &cnt0);
    ncc = sum;   // ComputeMultiNCC adds to a sum that starts at 0
}

// VerticalLineLocus_seeddem's per-node update (setsm_code.cpp:7806-7853).
__global__ void __launch_bounds__(128) seeddem_kernel(const DevLevel *__restrict__ Pp,
                                                      const OrthoArgs A,
                                                      vll_ugrid *__restrict__ gout) {
    const DevLevel &P = *Pp;
    for (int64_t pt = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; pt < P.n_nodes;
         pt += (int64_t)gridDim.x * blockDim.x) {
        vll_ugrid g = P.gp3[pt];
        for (int ti = 1; ti < P.num_images; ++ti) {
            if (!P.im[ti].selected) continue;
            double ncc;
            int cnt0;
            ortho_node_ncc(P, A, pt, ti, ncc, cnt0);
            if (cnt0 == 0) ncc = -10;
            if (ncc < 0.3 && !P.check_matchtag) {
                g.minHeight = (int16_t)(g.minHeight - 100);
                if (g.minHeight < P.minmax[0]) g.minHeight = (int16_t)floor(P.minmax[0]);
                g.maxHeight = (int16_t)(g.maxHeight + 100);
                if (g.maxHeight > P.minmax[1]) g.maxHeight = (int16_t)ceil(P.minmax[1]);
                if (ncc < 0.1) {
                    g.minHeight = -9999;
                    g.maxHeight = -9999;
                }
            }
            set_ortho_ncc(g, ti, q_result(ncc));
            if (P.check_matchtag) g.roh = q_result(ncc >= 0.2 ? ncc : -0.2);
        }
        gout[pt] = g;
    }
}

// VerticalLineLocus_blunder's per-node result (setsm_code.cpp:7940-8012).
__global__ void __launch_bounds__(128) blunder_kernel(const DevLevel *__restrict__ Pp,
                                                      const OrthoArgs A,
                                                      vll_ugrid *__restrict__ gout,
                                                      float *__restrict__ ncc_out) {
    const DevLevel &P = *Pp;
    for (int64_t pt = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; pt < P.n_nodes;
         pt += (int64_t)gridDim.x * blockDim.x) {
        vll_ugrid g = P.gp3[pt];
        double max_ncc = -100;
        for (int ti = 1; ti < P.num_images; ++ti) {
            if (!P.im[ti].selected) continue;
            double ncc;
            int cnt0;
            ortho_node_ncc(P, A, pt, ti, ncc, cnt0);
            if (max_ncc < ncc) max_ncc = ncc;
            set_ortho_ncc(g, ti, q_result(ncc));
        }
        g.Mean_ortho_ncc = q_result(max_ncc);
        gout[pt] = g;
        ncc_out[pt] = (float)max_ncc;
    }
}

// ---- sampled rasters ------------------------------------------------------------
// A node's window and its neighbours' overlap (a pixel lies in seven windows
// when the grid is four pixels apart), and a sample depends on its pixel
// alone, so a raster per image holds its samples: {intensity, magnitude} of
// each pixel, NaN first where SetVecKernelValue would drop the pixel for this
// image.  The node pass is then one pass of sums over rows of pixels of the
// reference's and a target's raster, shifted by the centre pixel's samples;
// FP64, so its NCC is within 1e-12 of the reference's two-pass one for the
// same samples.
//
// kExact samples at the reference's coordinates.  Otherwise the projection
// uses CUDA's sin, cos and arctangents (the reference's C library rounds
// correctly) and fused products: a coordinate off by up to `delta` pixel (see
// coord_error), a sample by 2 delta times the largest step between its texels,
// an NCC by what that is to the window's spread.  The fast raster therefore
// comes with the largest step of each of its tiles, and a node's band follows
// from those its window touches.  (One band for all, 2e-7, missed windows that
// rest on single texels at a corner's tiny weight.)  Either way a node whose
// rounding to 1/1000, thresholds or variance tests lie within the band is
// listed and evaluated again in the reference's order (exact_node_kernel).
//
// 1024^2 grid, 4097^2 pixels, 11x11 window: 9.85 ms with the samples formed
// per node and pass (raster 3.8, nodes 6.0), now 2.11 (2.04 with one band for
// all nodes; raster about 0.95, nodes 0.95, exact 0.2): the raster is bound by
// FP64 issue and latency (585 FP64 instructions per 32 pixels), the node pass by
// latency at 16 warps per SM (12 warps: 2.37 ms in all, 20: 2.54).
constexpr double kSumBand = 1e-9;   // one-pass against two-pass sums of the same samples
constexpr int kMaxSampledH = 15;   // larger windows take the per-node kernels
constexpr int kNodeLanes = 4;      // lanes per node: columns c = lane (mod 4)

// The rasters of a pair of images.
struct Raster {
    const double2 *ref, *tgt;
};

// A fast pyramid coordinate: clamped to [0, vmax] like the reference's, scaled
// and shifted.  `edge`: too close to the clamp, or (unclamped) to a texel's
// position, the image's bounds among them, for its error: the reference may
// sample the other side, whose texels are not among this one's.  near: four
// times the error.
constexpr double kPixelEdge = 1e-6;
__device__ __forceinline__ double fast_bound(double v, double vmax, double inv, double start,
                                             double near, bool &edge) {
    constexpr double kRint = 6755399441055744.0;   // 1.5 * 2^52
    const bool lo = v < 0, hi = v > vmax;
    const double c = fma(lo ? 0.0 : (hi ? vmax : v), inv, -start);
    if (!(fmin(fabs(v), fabs(v - vmax)) > kPixelEdge)) edge = true;
    if (!(lo || hi) && !(fabs(c - __dadd_rn(__dadd_rn(c, kRint), -kRint)) > near)) edge = true;
    return c;
}

// The RPCs of two images (or one) as a kernel parameter: their 160
// coefficients per pixel come from the constant bank, not through the load
// pipe, which they kept 75 % busy.
struct PairRpc {
    double rpc[2][90];
    double adj[2][2];
    double inv_scale[2][3];   // of longitude, latitude, height
};

// 1 / v from an FP32 seed and two Newton steps; `edge` is set where the seed
// is no finite non-zero float.
__device__ __forceinline__ double fast_recip(double v, bool &edge) {
    const float f = __frcp_rn((float)v);
    if (!(fabsf(f) > 0.f && fabsf(f) < 3.0e38f)) edge = true;
    double r = (double)f;
    r = fma(r, fma(-v, r, 1.0), r);
    return fma(r, fma(-v, r, 1.0), r);
}

// GetObjectToImageRPC_single and OriginalToPyramid_single with fused products
// (see rpc_project, to_pyramid).
__device__ __forceinline__ double2 fast_coord(const double *rpc, const double *adj,
                                              const double *inv_scale, double lon, double lat,
                                              double h, double inv, double sx, double sy,
                                              double near, bool &edge) {
    double L = (lon - rpc[2]) * inv_scale[0];
    double P = (lat - rpc[3]) * inv_scale[1];
    const double H = (h - rpc[4]) * inv_scale[2];
    if (!(fabs(fabs(L) - 10.0) > kPixelEdge) || !(fabs(fabs(P) - 10.0) > kPixelEdge)) edge = true;
    if (L < -10.0 || L > 10.0) L = ((lon > 0 ? lon - 360 : lon + 360) - rpc[2]) * inv_scale[0];
    if (P < -10.0 || P > 10.0) P = ((lat > 0 ? lat - 360 : lat + 360) - rpc[3]) * inv_scale[1];
    const double LL = L * L, PP = P * P, HH = H * H, LP = L * P, LH = L * H, PH = P * H;
    const double t[20] = {1.0,    L,      P,      H,      LP,     LH,     PH,
                          LL,     PP,     HH,     LP * H, LL * L, L * PP, L * HH,
                          LL * P, PP * P, P * HH, LL * H, PP * H, HH * H};
    double cf[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const double *c = rpc + 10 + 20 * j;
        double a = c[0];
#pragma unroll
        for (int i = 1; i < 20; ++i) a = fma(c[i], t[i], a);
        cf[j] = a;
    }
    const double y = adj[0] + fma(cf[0] * fast_recip(cf[1], edge), rpc[5], rpc[0]);
    const double x = adj[1] + fma(cf[2] * fast_recip(cf[3], edge), rpc[6], rpc[1]);
    return make_double2(
        fast_bound(x, __dadd_rn(rpc[1], __dmul_rn(rpc[6], 1.2)), inv, sx, near, edge),
        fast_bound(y, __dadd_rn(rpc[0], __dmul_rn(rpc[5], 1.2)), inv, sy, near, edge));
}

// ps2wgs_single with CUDA's functions (polar stereographic; UTM grids take
// the exact one).
__device__ __forceinline__ double2 ps2wgs_fast(const vll_transparam &p, double X, double Y) {
    if (p.projection != 1) return ps2wgs_dev(p, X, Y);
    const double e2 = p.e * p.e, e4 = e2 * e2, e6 = e2 * e4, e8 = e4 * e4;
    const double x = X * p.pm, y = Y * p.pm;
    const double t = sqrt(fma(x, x, y * y)) * (p.t_c / (p.a * p.m_c));
    const double chi = kPi / 2 - 2 * atan(t);
    double s2, c2;
    sincos(2 * chi, &s2, &c2);
    const double s4 = 2 * s2 * c2, c4 = fma(-2 * s2, s2, 1.0);
    const double s6 = fma(s4, c2, c4 * s2), s8 = 2 * s4 * c4;
    double phi = chi + (e2 / 2 + 5 * e4 / 24 + e6 / 12 + 13 * e8 / 360) * s2 +
                 (7 * e4 / 48 + 29 * e6 / 240 + 811 * e8 / 11520) * s4 +
                 (7 * e6 / 120 + 81 * e8 / 1120) * s6 + (4279 * e8 / 161280) * s8;
    double lambda = p.lambda_0 + atan2(x, -y);
    phi = p.pm * phi;
    lambda = p.pm * lambda;
    if (lambda > kPi)
        lambda = lambda - 2 * kPi;
    else if (lambda < -kPi)
        lambda = lambda + 2 * kPi;
    return make_double2(180 / kPi * lambda, 180 / kPi * phi);
}

// Grid column (row) of raster position t (SetOrthoImageCoord's truncation).
__device__ __forceinline__ int64_t grid_at(double t, double origin, double res) {
    return (int64_t)__ddiv_rn(__dadd_rn(t, -origin), res);
}

// The height of the raster pixel in grid cell (t_col, t_row); false when the
// pixel has none (its coordinates stay 0, setsm_code.cpp:6550-6670).
__device__ __forceinline__ bool cell_height(const DevLevel &P, int64_t t_col, int64_t t_row,
                                            float &h) {
    const int64_t pt = t_row * P.grid_w + t_col;
    if (!(pt < P.n_nodes && t_col < P.grid_w && t_row < P.grid_h)) return false;
    h = P.gp3[pt].Height;
    return h != -1000;
}
__device__ __forceinline__ bool pixel_height(const DevLevel &P, double tX, double tY, float &h) {
    return cell_height(P, grid_at(tX, P.boundary[0], P.grid_res),
                       grid_at(tY, P.boundary[1], P.grid_res), h);
}

__device__ __forceinline__ PatchSrc patch_of(const DevLevel &P, int ti, int use_b) {
    const DevImage &ri = P.im[P.ref], &tI = P.im[ti];
    return use_b ? PatchSrc{ri.img_b, ri.mag_b, tI.img_b, tI.mag_b, ri.wb, ri.hb, tI.wb, tI.hb}
                 : PatchSrc{ri.img, ri.mag, tI.img, tI.mag, ri.w, ri.h, tI.w, tI.h};
}

// An image's planes at the level the pass samples.
struct Planes {
    const uint16_t *img, *mag;
    uint32_t w, h;
};
__device__ __forceinline__ Planes planes_of(const DevImage &im, int use_b) {
    return use_b ? Planes{im.img_b, im.mag_b, im.wb, im.hb} : Planes{im.img, im.mag, im.w, im.h};
}

// One image's share of sample4: false where it drops the pixel.
__device__ __forceinline__ bool exact_sample(const Planes &S, double2 p, double v[2]) {
    if (!(p.y >= 0 && __dadd_rn(p.y, 1.0) < (double)S.h && p.x >= 0 &&
          __dadd_rn(p.x, 1.0) < (double)S.w))
        return false;
    const uint32_t xi = __double2uint_rz(p.x), yi = __double2uint_rz(p.y);
    const int64_t at = (int64_t)xi + (int64_t)yi * (int64_t)S.w;
    const double dx = __dadd_rn(p.x, -u32_to_double(xi)), dy = __dadd_rn(p.y, -u32_to_double(yi));
    v[0] = interp(S.img, at, S.w, dx, dy);
    v[1] = interp(S.mag, at, S.w, dx, dy);
    return v[0] > 0;
}

// The same at fast coordinates (fused products).  step: the largest step
// between the texels, of each plane; `edge`: an intensity so small that the
// coordinates' error (see fast_bound) could decide its sign.
__device__ __forceinline__ bool fast_sample(const Planes &S, double2 p, double v[2], double near,
                                            unsigned step[2], bool &edge) {
    if (!(p.y >= 0 && p.y + 1.0 < (double)S.h && p.x >= 0 && p.x + 1.0 < (double)S.w)) return false;
    const int xi = (int)p.x, yi = (int)p.y;
    const double fx = p.x - (double)xi, fy = p.y - (double)yi;
    const int64_t at = (int64_t)yi * S.w + xi;
#pragma unroll
    for (int c = 0; c < 2; ++c) {
        const uint16_t *I = (c ? S.mag : S.img) + at;
        const int a = I[0], b = I[1], d = I[S.w], e = I[S.w + 1];
        const double u = fma(fx, (double)(b - a), (double)a);
        const double q = fma(fx, (double)(e - d), (double)d);
        v[c] = fma(fy, q - u, u);
        step[c] = max(max(a, b), max(d, e)) - min(min(a, b), min(d, e));
        if (c == 0 && v[0] < near * (double)step[0]) edge = true;
    }
    return v[0] > 0;
}

// The samples of image im (k: its place in R) at a raster pixel's `lonlat` and
// height h (an uncovered pixel's coordinates are 0), exact or fast.
template <bool kExact>
__device__ __forceinline__ bool raster_sample(const DevLevel &P, const DevImage &im, const PairRpc &R,
                                              int k, int use_b, double v[2], double2 lonlat,
                                              bool covered, float h, double near,
                                              unsigned step[2], bool &edge) {
    const Planes S = planes_of(im, use_b);
    double2 p = make_double2(0, 0);
    if (covered) {
        const int lev = use_b ? P.blunder_level : P.L;
        const double sx = use_b ? im.sxb : im.sx, sy = use_b ? im.syb : im.sy;
        if constexpr (kExact)
            p = to_pyramid(rpc_project(R.rpc[k], R.adj[k], lonlat.x, lonlat.y, (double)h), sx, sy, lev);
        else
            p = fast_coord(R.rpc[k], R.adj[k], R.inv_scale[k], lonlat.x, lonlat.y, (double)h,
                           1.0 / (double)(1 << lev), sx, sy, near, edge);
    }
    if constexpr (kExact)
        return exact_sample(S, p, v);
    else
        return fast_sample(S, p, v, near, step, edge);
}

// A block's tile of one or two images' rasters.  Grid columns and rows (two divisions) are found
// once per tile column and row.  The fast projection is evaluated at 3 x 3
// points of the tile and interpolated quadratically: its third-order term
// over the tile is below kTileError pixels wherever the tile lies far enough
// from the pole (the projection's scale varies over the distance to it);
// nearer, or across the +-180 degree line, every pixel is projected.
constexpr int kTileW = 32, kTileH = 8;
constexpr double kTileError = 1e-8;

template <bool kExact, int kImages>
__global__ void __launch_bounds__(kTileW * kTileH, kExact ? 4 : 5) sample_raster_kernel(
    const DevLevel *__restrict__ Pp, const __grid_constant__ PairRpc R, int image0, int image1,
    double2 *__restrict__ out0, double2 *__restrict__ out1, ushort2 *__restrict__ steps0,
    ushort2 *__restrict__ steps1, int64_t ow, int64_t oh, double im_res, int use_b,
    int64_t tiles_x, double near) {
    __shared__ int at_col[kTileW], at_row[kTileH];
    __shared__ double2 stencil[9];
    __shared__ unsigned tile_step[kImages][2];
    const DevLevel &P = *Pp;
    const int64_t by = blockIdx.x / tiles_x, bx = blockIdx.x - by * tiles_x;
    const int64_t col = bx * kTileW + threadIdx.x, row = by * kTileH + threadIdx.y;
    const double tX = __dadd_rn(P.boundary[0], __dmul_rn((double)col, im_res));
    const double tY = __dadd_rn(P.boundary[1], __dmul_rn((double)row, im_res));
    if (threadIdx.y == 0) {
        const int64_t c = grid_at(tX, P.boundary[0], P.grid_res);
        at_col[threadIdx.x] = c < P.grid_w ? (int)c : -1;
    }
    if (threadIdx.x == 0) {
        const int64_t r = grid_at(tY, P.boundary[1], P.grid_res);
        at_row[threadIdx.y] = r < P.grid_h ? (int)r : -1;
    }
    const double x0 = P.boundary[0] + (double)(bx * kTileW) * im_res;
    const double y0 = P.boundary[1] + (double)(by * kTileH) * im_res;
    const double sx = 0.5 * (kTileW - 1) * im_res, sy = 0.5 * (kTileH - 1) * im_res;
    bool tiled = false;
    if constexpr (!kExact) {
        // half the tile's diagonal against the distance to the pole
        const double half2 = sx * sx + sy * sy;
        const double rho2 = (x0 + sx) * (x0 + sx) + (y0 + sy) * (y0 + sy);
        tiled = P.param.projection == 1 && half2 * sqrt(half2) < kTileError * im_res * rho2;
        const int t = threadIdx.x + kTileW * threadIdx.y - 32;   // the second warp
        if (t >= 32 && t < 32 + 2 * kImages) tile_step[(t - 32) >> 1][t & 1] = 0;
        if (tiled && t >= 0 && t < 9)
            stencil[t] = ps2wgs_fast(P.param, x0 + (double)(t % 3) * sx, y0 + (double)(t / 3) * sy);
    }
    __syncthreads();
    // (every thread of a fast tile takes part in its largest step)
    const bool live = col < ow && row < oh;
    if (kExact && !live) return;
    const int gc = at_col[threadIdx.x], gr = at_row[threadIdx.y];
    float h = 0.f;
    const bool covered = live && gc >= 0 && gr >= 0 && cell_height(P, gc, gr, h);
    double2 w = make_double2(0, 0);
    if (covered) {
        if constexpr (kExact) {
            w = ps2wgs_dev(P.param, tX, tY);
        } else {
            if (tiled)
                for (int k = 0; k < 8; ++k) tiled = tiled && fabs(stencil[k].x - stencil[8].x) < 90.0;
            if (tiled) {
                // Lagrange weights at 0, 1, 2 of the position in half tiles
                const double u = (double)threadIdx.x * (2.0 / (kTileW - 1));
                const double v = (double)threadIdx.y * (2.0 / (kTileH - 1));
                const double lu[3] = {0.5 * (u - 1) * (u - 2), u * (2 - u), 0.5 * u * (u - 1)};
                const double lv[3] = {0.5 * (v - 1) * (v - 2), v * (2 - v), 0.5 * v * (v - 1)};
#pragma unroll
                for (int k = 0; k < 9; ++k) {
                    // differences from the first point: the weights sum to 1
                    const double g = lu[k % 3] * lv[k / 3];
                    w.x = fma(g, stencil[k].x - stencil[0].x, w.x);
                    w.y = fma(g, stencil[k].y - stencil[0].y, w.y);
                }
                w.x += stencil[0].x;
                w.y += stencil[0].y;
            } else {
                w = ps2wgs_fast(P.param, tX, tY);
            }
        }
    }
    // a dropped pixel: NaN first; one the fast coordinates do not decide: NaN
    // twice
    const double nan = __longlong_as_double(0x7ff8000000000000ll);
    constexpr int kUnroll = kExact ? 1 : kImages;
#pragma unroll kUnroll
    for (int k = 0; k < kImages; ++k) {
        double o[2];
        unsigned step[2] = {0, 0};
        bool edge = false;
        if (!raster_sample<kExact>(P, P.im[k ? image1 : image0], R, k, use_b, o, w, covered, h, near,
                                   step, edge)) {
            o[0] = nan;
            o[1] = 0.0;
        }
        if (edge) o[0] = o[1] = nan;
        if (live) (k ? out1 : out0)[row * ow + col] = make_double2(o[0], o[1]);
        if constexpr (!kExact) {
#pragma unroll
            for (int c = 0; c < 2; ++c) {
                const unsigned m = __reduce_max_sync(0xffffffffu, step[c]);
                if (threadIdx.x == 0) atomicMax(&tile_step[k][c], m);
            }
        }
    }
    if constexpr (!kExact) {
        __syncthreads();
        if (threadIdx.y == 0 && threadIdx.x < kImages)
            (threadIdx.x ? steps1 : steps0)[blockIdx.x] =
                make_ushort2((unsigned short)tile_step[threadIdx.x][0],
                             (unsigned short)tile_step[threadIdx.x][1]);
    }
}

// Whether each node's height is set (the window's pixels of the others are
// dropped), and over fast rasters the largest steps of the tiles around each
// node's window, of every image sampled (node_steps: [num_images][n_nodes]).
// (Looked up by the node pass itself they cost it 6 %.)
__global__ void node_set_kernel(const DevLevel *__restrict__ Pp, uint8_t *__restrict__ set,
                                const ushort2 *__restrict__ steps, int64_t tiles_x, int64_t n_tiles,
                                int64_t ow, int64_t oh, double im_res, int H,
                                ushort2 *__restrict__ node_steps) {
    const DevLevel &P = *Pp;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < P.n_nodes;
         i += (int64_t)gridDim.x * blockDim.x) {
        set[i] = P.gp3[i].Height != -1000;
        if (!node_steps) continue;
        const int64_t a = (int64_t)((P.grid_pts[2 * i] - P.boundary[0]) / im_res);
        const int64_t b = (int64_t)((P.grid_pts[2 * i + 1] - P.boundary[1]) / im_res);
        const int64_t x0 = max(a - H - 1, (int64_t)0) / kTileW, x1 = min(a + H + 1, ow - 1) / kTileW;
        const int64_t y0 = max(b - H - 1, (int64_t)0) / kTileH, y1 = min(b + H + 1, oh - 1) / kTileH;
        for (int im = 0; im < P.num_images; ++im) {
            if (!P.im[im].selected || (im == 0 && P.ref != 0)) continue;
            ushort2 m = make_ushort2(0, 0);
            for (int64_t y = y0; y <= y1; ++y)
                for (int64_t x = x0; x <= x1; ++x) {
                    const ushort2 t = steps[im * n_tiles + y * tiles_x + x];
                    m = make_ushort2(max(m.x, t.x), max(m.y, t.y));
                }
            node_steps[im * P.n_nodes + i] = m;
        }
    }
}

// What a variant writes from a node's NCC values (VerticalLineLocus_seeddem,
// setsm_code.cpp:7806-7853; VerticalLineLocus_blunder, :7940-8012).
struct NodeState {
    vll_ugrid g;
    double max_ncc;
};

template <bool kBlunder>
__device__ __forceinline__ void node_begin(const DevLevel &P, int64_t pt, NodeState &n) {
    n.g = P.gp3[pt];
    n.max_ncc = -100;
}
template <bool kBlunder>
__device__ __forceinline__ void node_image(const DevLevel &P, int ti, double ncc, int cnt0,
                                           NodeState &n) {
    vll_ugrid &g = n.g;
    if (kBlunder) {
        if (n.max_ncc < ncc) n.max_ncc = ncc;
        set_ortho_ncc(g, ti, q_result(ncc));
        return;
    }
    if (cnt0 == 0) ncc = -10;
    if (ncc < 0.3 && !P.check_matchtag) {
        g.minHeight = (int16_t)(g.minHeight - 100);
        if (g.minHeight < P.minmax[0]) g.minHeight = (int16_t)floor(P.minmax[0]);
        g.maxHeight = (int16_t)(g.maxHeight + 100);
        if (g.maxHeight > P.minmax[1]) g.maxHeight = (int16_t)ceil(P.minmax[1]);
        if (ncc < 0.1) {
            g.minHeight = -9999;
            g.maxHeight = -9999;
        }
    }
    set_ortho_ncc(g, ti, q_result(ncc));
    if (P.check_matchtag) g.roh = q_result(ncc >= 0.2 ? ncc : -0.2);
}
template <bool kBlunder>
__device__ __forceinline__ void node_end(int64_t pt, NodeState &n, vll_ugrid *gout, float *ncc_out) {
    if (kBlunder) {
        n.g.Mean_ortho_ncc = q_result(n.max_ncc);
        ncc_out[pt] = (float)n.max_ncc;
    }
    gout[pt] = n.g;
}

// Whether a value within `band` of ncc could be rounded or compared otherwise
// (the blunder pass also returns it as a float, whose last bit a value near 0,
// a cancellation of the correlations it is the mean of, does not fix; the
// reference's two-pass sums leave 1e-17 where these cancel to 0).
template <bool kBlunder>
__device__ __forceinline__ bool near_decision(double ncc, bool counted, double band) {
    const double x = ncc * 1000.0;
    bool near = fabs(x - floor(x) - 0.5) <= band * 1000.0;
    if (kBlunder)
        near = near || (counted && fabs(ncc) < 1e-4);
    else
        near = near || fabs(ncc - 0.3) <= band || fabs(ncc - 0.1) <= band || fabs(ncc - 0.2) <= band;
    return near || !(fabs(ncc) <= 2.0);
}

struct RingSum {
    double n;
    double sl[2], sr[2], sll[2], srr[2], slr[2];
};
__device__ __forceinline__ void ring_add(RingSum &a, const double (&d)[4]) {
    a.n += 1.0;
#pragma unroll
    for (int p = 0; p < 2; ++p) {
        a.sl[p] += d[p];
        a.sr[p] += d[p + 2];
        a.sll[p] = fma(d[p], d[p], a.sll[p]);
        a.srr[p] = fma(d[p + 2], d[p + 2], a.srr[p]);
        a.slr[p] = fma(d[p], d[p + 2], a.slr[p]);
    }
}
__device__ __forceinline__ double lanes_sum(double v) {
#pragma unroll
    for (int o = 1; o < kNodeLanes; o <<= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}
__device__ __forceinline__ void ring_reduce(RingSum &a) {
    a.n = lanes_sum(a.n);
#pragma unroll
    for (int p = 0; p < 2; ++p) {
        a.sl[p] = lanes_sum(a.sl[p]);
        a.sr[p] = lanes_sum(a.sr[p]);
        a.sll[p] = lanes_sum(a.sll[p]);
        a.srr[p] = lanes_sum(a.srr[p]);
        a.slr[p] = lanes_sum(a.slr[p]);
    }
}
__device__ __forceinline__ void ring_join(RingSum &a, const RingSum &b) {
    a.n += b.n;
#pragma unroll
    for (int p = 0; p < 2; ++p) {
        a.sl[p] += b.sl[p];
        a.sr[p] += b.sr[p];
        a.sll[p] += b.sll[p];
        a.srr[p] += b.srr[p];
        a.slr[p] += b.slr[p];
    }
}

struct SampledArgs {
    const double2 *const *raster;   // [num_images]: the images' samples
    const uint8_t *set;           // node_set_kernel
    int64_t ow, oh;
    double im_res;
    int H, r2max, use_b;
    // fast rasters: see node_set_kernel; twice the coordinates' error in texels
    const ushort2 *node_steps;
    float delta;
};

// Four lanes per node, each the window columns congruent to it (NJ of them at
// most): a row of the window is then read in whole 128-byte pieces.
template <bool kBlunder, int NJ>
__global__ void __launch_bounds__(128, NJ <= 4 ? 4 : 2) node_ncc_kernel(const DevLevel *__restrict__ Pp,
                                                       const SampledArgs A,
                                                       vll_ugrid *__restrict__ gout,
                                                       float *__restrict__ ncc_out,
                                                       int64_t *__restrict__ todo,
                                                       unsigned long long *__restrict__ n_todo) {
    __shared__ int2 row_at[128 / kNodeLanes][2 * kMaxSampledH + 1];
    // A constant area's samples are equal in the fast raster and differ by
    // rounding (1e-11 at most) in the reference's order, which alone listed
    // every node over such an area (240 k nodes, two fifths of the images
    // constant: 1.37 -> 0.39 ms).
    constexpr double kNone = kBlunder ? 1e-10 : 0.0;
    const DevLevel &P = *Pp;
    const int sub = threadIdx.x & (kNodeLanes - 1);
    const unsigned group = ((1u << kNodeLanes) - 1u) << ((threadIdx.x & 31) - sub);
    int2 *rows = row_at[threadIdx.x / kNodeLanes];
    const int64_t stride = (int64_t)gridDim.x * (blockDim.x / kNodeLanes);
    const int H = A.H;
    const int s1 = H / 2, s2 = s1 + (int)((s1 / 2.0) + 0.5);
    const int e1 = H - s1, e2 = H - s2;
    // every lane of a warp takes part in the reductions: nodes past the end
    // repeat the last one
    const int64_t n_round = (P.n_nodes + 31) / 32 * 32;
    for (int64_t at = blockIdx.x * (int64_t)(blockDim.x / kNodeLanes) + threadIdx.x / kNodeLanes;
         at < n_round; at += stride) {
        const bool live = at < P.n_nodes;
        const int64_t pt = live ? at : P.n_nodes - 1;
        const double gx = P.grid_pts[2 * pt], gy = P.grid_pts[2 * pt + 1];
        const double *B = P.boundary;
        // raster and grid columns of this lane's window columns (-1: dropped)
        int tc[NJ], tt[NJ];
#pragma unroll
        for (int j = 0; j < NJ; ++j) {
            const int c = -H + sub + kNodeLanes * j;
            const double tX = __dadd_rn(gx, __dmul_rn((double)c, A.im_res));
            const int64_t a = (int64_t)__ddiv_rn(__dadd_rn(tX, -B[0]), A.im_res);
            const int64_t b = (int64_t)__ddiv_rn(__dadd_rn(tX, -B[0]), P.grid_res);
            const bool ok = c <= H && a >= 0 && a < A.ow && b >= 0 && b < P.grid_w;
            tc[j] = ok ? (int)a : -1;
            tt[j] = ok ? (int)b : 0;
        }
        // ... and of the window's rows, a share per lane
        for (int r = sub; r <= 2 * H; r += kNodeLanes) {
            const double tY = __dadd_rn(gy, __dmul_rn((double)(r - H), A.im_res));
            const int64_t a = (int64_t)__ddiv_rn(__dadd_rn(tY, -B[1]), A.im_res);
            const int64_t b = (int64_t)__ddiv_rn(__dadd_rn(tY, -B[1]), P.grid_res);
            const bool ok = a >= 0 && a < A.oh && b >= 0 && b < P.grid_h;
            rows[r] = make_int2(ok ? (int)a : -1, ok ? (int)b : 0);
        }
        __syncwarp();
        NodeState st;
        node_begin<kBlunder>(P, pt, st);
        bool unsure = false;
        for (int ti = 1; ti < P.num_images; ++ti) {
            if (!P.im[ti].selected) continue;
            const Raster R{A.raster[P.ref], A.raster[ti]};
            RingSum acc[3] = {};
            double sh[4];
            ushort2 step[2];
            if constexpr (!kBlunder) {
                step[0] = A.node_steps[P.ref * P.n_nodes + pt];
                step[1] = A.node_steps[ti * P.n_nodes + pt];
            }
            {
                // the shift: the pixel of the node itself, where it has samples
                const int64_t a = (int64_t)__ddiv_rn(__dadd_rn(gx, -B[0]), A.im_res);
                const int64_t b = (int64_t)__ddiv_rn(__dadd_rn(gy, -B[1]), A.im_res);
                const bool in = a >= 0 && a < A.ow && b >= 0 && b < A.oh;
                double2 l = in ? R.ref[b * A.ow + a] : make_double2(nan(""), 0);
                double2 r = in ? R.tgt[b * A.ow + a] : make_double2(0, 0);
                const bool none = isnan(l.x) || isnan(r.x);
                if (none) {
                    // ... else one of the innermost window's (whose sums would
                    // cancel about 0 and list every node beside an empty
                    // area); all of the node's lanes are here
                    bool mine = false;
                    for (int row = -e2; row <= e2 && !mine; ++row) {
                        const int2 at_row = rows[row + H];
                        if (at_row.x < 0) continue;
#pragma unroll
                        for (int j = 0; j < NJ; ++j) {
                            const int c = -H + sub + kNodeLanes * j;
                            if (mine || c < -e2 || c > e2 || tc[j] < 0) continue;
                            const int64_t q = (int64_t)at_row.x * A.ow + tc[j];
                            l = R.ref[q];
                            r = R.tgt[q];
                            mine = !isnan(l.x) && !isnan(r.x);
                        }
                    }
                    const unsigned have = __ballot_sync(group, mine);
                    const int src = have ? __ffs(have) - 1 : 0;
                    l.x = __shfl_sync(group, l.x, src);
                    l.y = __shfl_sync(group, l.y, src);
                    r.x = __shfl_sync(group, r.x, src);
                    r.y = __shfl_sync(group, r.y, src);
                    if (!have) l = r = make_double2(0, 0);
                }
                sh[0] = l.x;
                sh[1] = l.y;
                sh[2] = r.x;
                sh[3] = r.y;
            }
#pragma unroll 1
            for (int row = -H; row <= H; ++row) {
                const int2 at_row = rows[row + H];
                if (at_row.x < 0 || row * row > A.r2max) continue;
                const int64_t first = (int64_t)at_row.x * A.ow;
                const uint8_t *set = A.set + (int64_t)at_row.y * P.grid_w;
                const int ar = row < 0 ? -row : row;
                // the row's loads together, then their sums
                double2 lo[NJ], hi[NJ];
                bool use[NJ];
#pragma unroll
                for (int j = 0; j < NJ; ++j) {
                    const int c = -H + sub + kNodeLanes * j;
                    use[j] = row * row + c * c <= A.r2max && tc[j] >= 0;
                    lo[j] = hi[j] = make_double2(0, 0);
                    if (use[j]) {
                        lo[j] = R.ref[first + tc[j]];
                        hi[j] = R.tgt[first + tc[j]];
                        use[j] = set[tt[j]];
                    }
                }
#pragma unroll
                for (int j = 0; j < NJ; ++j) {
                    const int c = -H + sub + kNodeLanes * j;
                    const int ac = c < 0 ? -c : c;
                    const int r2 = row * row + c * c;
                    if (!use[j]) continue;
                    if (isnan(lo[j].x) || isnan(hi[j].x)) {
                        if (isnan(lo[j].y) || isnan(hi[j].y)) unsure = true;
                        continue;
                    }
                    const double d[4] = {lo[j].x - sh[0], lo[j].y - sh[1], hi[j].x - sh[2],
                                         hi[j].y - sh[3]};
                    const bool w2 = r2 <= (e2 + 1) * (e2 + 1) && ar <= e2 && ac <= e2;
                    const bool w1 = r2 <= (e1 + 1) * (e1 + 1) && ar <= e1 && ac <= e1;
                    if (w2)
                        ring_add(acc[2], d);
                    else if (w1)
                        ring_add(acc[1], d);
                    else
                        ring_add(acc[0], d);
                }
            }
            __syncwarp();
#pragma unroll
            for (int w = 0; w < 3; ++w) ring_reduce(acc[w]);
            // nested windows: 2 = ring 2; 1 = rings 1 + 2; 0 = all rings
            ring_join(acc[1], acc[2]);
            ring_join(acc[0], acc[1]);
            double ncc = 0, cnt = 0, band = kSumBand;
            if (acc[0].n > 0 && acc[1].n > 0 && acc[2].n > 0) {
                double tot = 0;
                float err = 0.f;
#pragma unroll
                for (int w = 0; w < 3; ++w) {
                    const double inv = 1.0 / acc[w].n;
                    const float root_n = sqrtf((float)acc[w].n);
#pragma unroll
                    for (int p = 0; p < 2; ++p) {
                        const double vl = fma(-acc[w].sl[p] * inv, acc[w].sl[p], acc[w].sll[p]);
                        const double vr = fma(-acc[w].sr[p] * inv, acc[w].sr[p], acc[w].srr[p]);
                        const double cv = fma(-acc[w].sl[p] * inv, acc[w].sr[p], acc[w].slr[p]);
                        // a variance that cancels, or that the sums do not
                        // decide against 1e-8 (squares that add up to kNone
                        // about the shift have none in any order)
                        const double ql = acc[w].sll[p], qr = acc[w].srr[p];
                        if ((ql > kNone && vl < fma(1e-3, ql, 1e-4)) ||
                            (qr > kNone && vr < fma(1e-3, qr, 1e-4)))
                            unsure = true;
                        if (vl > 1e-8 && vr > 1e-8) {
                            const double rho = cv / sqrt(vl * vr);
                            tot += rho;
                            cnt += 1.0;
                            if constexpr (!kBlunder) {
                                // samples off by `delta` steps turn the vectors
                                // by at most x in all, the correlation (a
                                // cosine) by x times its sine and x^2
                                const float x = A.delta * root_n *
                                                ((float)(p ? step[0].y : step[0].x) *
                                                     rsqrtf((float)vl) +
                                                 (float)(p ? step[1].y : step[1].x) *
                                                     rsqrtf((float)vr));
                                const float c = (float)rho;
                                err += x * (sqrtf(fmaxf(fmaf(-c, c, 1.f), 0.f)) + 2.f * x);
                            }
                        }
                    }
                }
                if (cnt > 0) {
                    ncc = tot / cnt;
                    if constexpr (!kBlunder) band += (double)err / cnt;
                }
            }
            if (near_decision<kBlunder>(ncc, cnt > 0, band)) unsure = true;
            node_image<kBlunder>(P, ti, ncc, (int)acc[0].n, st);
        }
        // (any of the node's lanes)
        unsure = (__ballot_sync(0xffffffffu, unsure) & group) != 0;
        __syncwarp();   // the row indices are rewritten by the next node
        if (live && sub == 0) {
            if (unsure)
                todo[atomicAdd(n_todo, 1ull)] = pt;
            else
                node_end<kBlunder>(pt, st, gout, ncc_out);
        }
    }
}

// Bytes of exact_node_kernel's staging for window half-size H.
__host__ __device__ constexpr size_t exact_node_bytes(int H) {
    return (size_t)(2 * H + 1) * (2 * H + 1) * 33 + 64;
}

// The listed nodes, a warp each: the window's pixels sampled at the
// reference's coordinates a lane each, then Correlate's six two-pass sums a
// lane each in its scan order (see multi_ncc).
template <bool kBlunder>
__global__ void __launch_bounds__(32, 16) exact_node_kernel(const DevLevel *__restrict__ Pp,
                                                        const SampledArgs A,
                                                        vll_ugrid *__restrict__ gout,
                                                        float *__restrict__ ncc_out,
                                                        const int64_t *__restrict__ todo,
                                                        const unsigned long long *__restrict__ n_todo) {
    extern __shared__ __align__(16) double smp[];
    __shared__ PairRpc R;
    const DevLevel &P = *Pp;
    const int lane = threadIdx.x;
    const int H = A.H, D = 2 * H + 1;
    unsigned char *flag = reinterpret_cast<unsigned char *>(smp + 4 * D * D);
    const int64_t n = (int64_t)*n_todo;
    for (int64_t i = blockIdx.x; i < n; i += gridDim.x) {
        const int64_t pt = todo[i];
        const double gx = P.grid_pts[2 * pt], gy = P.grid_pts[2 * pt + 1];
        const double *B = P.boundary;
        NodeState st;
        node_begin<kBlunder>(P, pt, st);
        for (int ti = 1; ti < P.num_images; ++ti) {
            if (!P.im[ti].selected) continue;
            const PatchSrc S = patch_of(P, ti, A.use_b);
            for (int k = lane; k < 180; k += 32)
                R.rpc[k / 90][k % 90] = P.im[k < 90 ? P.ref : ti].rpc[k % 90];
            if (lane < 4) R.adj[lane >> 1][lane & 1] = P.im[lane < 2 ? P.ref : ti].adj[lane & 1];
            __syncwarp();
            for (int k = lane; k < D * D; k += 32) {
                const int row = k / D - H, col = k % D - H;
                const int r2 = row * row + col * col;
                unsigned char f = 0;
                if (r2 <= A.r2max && r2 <= (H + 1) * (H + 1)) {
                    const double tX = __dadd_rn(gx, __dmul_rn((double)col, A.im_res));
                    const double tY = __dadd_rn(gy, __dmul_rn((double)row, A.im_res));
                    const int64_t tc = (int64_t)__ddiv_rn(__dadd_rn(tX, -B[0]), A.im_res);
                    const int64_t tr = (int64_t)__ddiv_rn(__dadd_rn(tY, -B[1]), A.im_res);
                    const int64_t ttc = (int64_t)__ddiv_rn(__dadd_rn(tX, -B[0]), P.grid_res);
                    const int64_t ttr = (int64_t)__ddiv_rn(__dadd_rn(tY, -B[1]), P.grid_res);
                    if (tc >= 0 && tc < A.ow && tr >= 0 && tr < A.oh && ttc >= 0 &&
                        ttc < P.grid_w && ttr >= 0 && ttr < P.grid_h &&
                        A.set[ttr * P.grid_w + ttc]) {
                        // the raster pixel's own position
                        const double rX = __dadd_rn(B[0], __dmul_rn((double)tc, A.im_res));
                        const double rY = __dadd_rn(B[1], __dmul_rn((double)tr, A.im_res));
                        float h = 0.f;
                        const bool covered = pixel_height(P, rX, rY, h);
                        double2 w = make_double2(0, 0);
                        if (covered) w = ps2wgs_dev(P.param, rX, rY);
                        double2 p[2] = {make_double2(0, 0), make_double2(0, 0)};
                        if (covered) {
                            const int lev = A.use_b ? P.blunder_level : P.L;
#pragma unroll 1
                            for (int im = 0; im < 2; ++im) {
                                const DevImage &I = P.im[im ? ti : P.ref];
                                p[im] = to_pyramid(
                                    rpc_project(R.rpc[im], R.adj[im], w.x, w.y, (double)h),
                                    A.use_b ? I.sxb : I.sx, A.use_b ? I.syb : I.sy, lev);
                            }
                        }
                        double v[4];
                        if (sample4(S, p[0], p[1], v)) {
                            f = (unsigned char)(1 + window_depth(H, row, col, r2));
#pragma unroll
                            for (int c = 0; c < 4; ++c) smp[4 * k + c] = v[c];
                        }
                    }
                }
                flag[k] = f;
            }
            __syncwarp();
            double r = -99.0;
            int cnt = 0;
            if (lane < 6) {
                const int w = lane >> 1, p = lane & 1;
                double Ls = 0, Rs = 0;
                for (int k = 0; k < D * D; ++k) {
                    if ((int)flag[k] - 1 < w) continue;
                    Ls = __dadd_rn(Ls, smp[4 * k + p]);
                    Rs = __dadd_rn(Rs, smp[4 * k + p + 2]);
                    ++cnt;
                }
                if (cnt > 0) {
                    const double Lm = __ddiv_rn(Ls, (double)cnt), Rm = __ddiv_rn(Rs, (double)cnt);
                    double lr = 0, ll = 0, rr = 0;
                    for (int k = 0; k < D * D; ++k) {
                        if ((int)flag[k] - 1 < w) continue;
                        const double dl = __dadd_rn(smp[4 * k + p], -Lm);
                        const double dr = __dadd_rn(smp[4 * k + p + 2], -Rm);
                        lr = __dadd_rn(lr, __dmul_rn(dl, dr));
                        ll = __dadd_rn(ll, __dmul_rn(dl, dl));
                        rr = __dadd_rn(rr, __dmul_rn(dr, dr));
                    }
                    if (ll > 1e-8 && rr > 1e-8) r = __ddiv_rn(lr, sqrt(__dmul_rn(ll, rr)));
                }
            }
            double ncc = 0, tot = 0, num = 0;
            bool all = true;
#pragma unroll
            for (int j = 0; j < 6; ++j) {
                const double rj = __shfl_sync(0xffffffffu, r, j);
                if (__shfl_sync(0xffffffffu, cnt, j) <= 0) all = false;
                if (rj != -99.0) {
                    num = __dadd_rn(num, 1.0);
                    tot = __dadd_rn(tot, rj);
                }
            }
            const int cnt0 = __shfl_sync(0xffffffffu, cnt, 0);
            if (all && num > 0) ncc = __ddiv_rn(tot, num);
            node_image<kBlunder>(P, ti, ncc, cnt0, st);
            __syncwarp();
        }
        if (lane == 0) node_end<kBlunder>(pt, st, gout, ncc_out);
        __syncwarp();
    }
}

unsigned blocks_for(int64_t n, int threads) {
    int64_t b = (n + threads - 1) / threads;
    if (b < 1) b = 1;
    if (b > 148 * 64) b = 148 * 64;
    return (unsigned)b;
}

}  // namespace

// Blunder windows of half-size 1 and 2 hold 1 and 5 pixels: forming a node's
// samples on the spot costs less than a raster of them (749 x 700 nodes, H = 2:
// 738 us per node, 772 over the raster; H = 3: 961 and 847).  The seed DEM's
// hold 9 and 29, and its raster is the cheaper fast one.
bool ortho_sampled(int H, bool blunder) { return H >= (blunder ? 3 : 1) && H <= kMaxSampledH; }

static int64_t raster_tiles(int64_t ow, int64_t oh) {
    return ((ow + kTileW - 1) / kTileW) * ((oh + kTileH - 1) / kTileH);
}
size_t ortho_sampled_scratch(int64_t n_nodes, int64_t ow, int64_t oh, int num_images) {
    return (((size_t)n_nodes + 255) & ~(size_t)255) + 256 + (size_t)n_nodes * 8 +
           (size_t)num_images * (raster_tiles(ow, oh) + n_nodes) * sizeof(ushort2);
}

// The fast coordinates' distance from the reference's in texels: the map
// projection's rounding (5e-9 m; 3.6e-9 m at most over 670 million points to
// 4000 km from either pole), and the third-order term of a tile's quadratic
// interpolation, which sample_raster_kernel keeps below kTileError pixels of
// the raster and which falls with the square of the distance to the pole.
static double coord_error(const DevLevel &P, double im_res, int use_b) {
    const double hx = 0.5 * (kTileW - 1) * im_res, hy = 0.5 * (kTileH - 1) * im_res;
    const double half2 = hx * hx + hy * hy;
    const double *B = P.boundary;
    const double dx = std::max(std::max(B[0], -B[2]), 0.0), dy = std::max(std::max(B[1], -B[3]), 0.0);
    const double rho2 = dx * dx + dy * dy;
    double tile = kTileError * im_res;
    if (rho2 > 0) tile = std::min(tile, half2 * sqrt(half2) / rho2);
    const double texel = P.im_res / (double)(1 << P.L) * (double)(1 << (use_b ? P.blunder_level : P.L));
    return (5e-9 + tile) / texel;
}

// The node pass of one variant over its sampled raster.
template <bool kBlunder>
static cudaError_t launch_nodes(const DevLevel *dP, int64_t n, const SampledArgs &A, vll_ugrid *gout,
                                float *ncc_out, int64_t *todo, unsigned long long *n_todo,
                                cudaStream_t s) {
    const unsigned blocks = blocks_for(n * kNodeLanes, 128);
    const int nj = (2 * A.H + 1 + kNodeLanes - 1) / kNodeLanes;
    // (300 x 280 nodes, H = 8 and 15: seed DEM 0.54 and 1.03 ms, blunder 0.48 and
    // 0.91; by the per-node kernels 1.95 and 5.36, 0.99 and 3.42)
    if (nj <= 3)
        node_ncc_kernel<kBlunder, 3><<<blocks, 128, 0, s>>>(dP, A, gout, ncc_out, todo, n_todo);
    else if (nj <= 4)
        node_ncc_kernel<kBlunder, 4><<<blocks, 128, 0, s>>>(dP, A, gout, ncc_out, todo, n_todo);
    else
        node_ncc_kernel<kBlunder, 8><<<blocks, 128, 0, s>>>(dP, A, gout, ncc_out, todo, n_todo);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    const size_t smem = exact_node_bytes(A.H);
    e = ensure_smem_limit((const void *)exact_node_kernel<kBlunder>, smem);
    if (e != cudaSuccess) return e;
    exact_node_kernel<kBlunder><<<148 * 16, 32, smem, s>>>(dP, A, gout, ncc_out, todo, n_todo);
    return cudaGetLastError();
}

cudaError_t launch_ortho_sampled(const DevLevel *dP, const DevLevel &hP, int64_t n_nodes,
                                 double2 *const *h_rasters, double2 *const *rasters, int64_t ow,
                                 int64_t oh, double im_res, int H, int use_b, vll_ugrid *gout,
                                 float *ncc_out, void *scratch, int64_t *launches,
                                 cudaStream_t s) {
    uint8_t *set = (uint8_t *)scratch;
    unsigned long long *n_todo =
        (unsigned long long *)((char *)scratch + (((size_t)n_nodes + 255) & ~(size_t)255));
    int64_t *todo = (int64_t *)((char *)n_todo + 256);
    cudaError_t e = cudaMemsetAsync(n_todo, 0, 8, s);
    if (e != cudaSuccess) return e;
    const int64_t tx = (ow + kTileW - 1) / kTileW, tiles = raster_tiles(ow, oh);
    ushort2 *steps = (ushort2 *)(todo + n_nodes), *node_steps = steps + hP.num_images * tiles;
    const double delta = coord_error(hP, im_res, use_b);
    if (tiles > 0x7fffffff) return cudaErrorInvalidValue;
    // the rasters of images a and b (b < 0: of a alone)
    auto sample = [&](int a, int b) {
        PairRpc R;
        for (int k = 0; k < 2; ++k) {
            const DevImage &im = hP.im[k && b >= 0 ? b : a];
            memcpy(R.rpc[k], im.rpc, sizeof(R.rpc[k]));
            memcpy(R.adj[k], im.adj, sizeof(R.adj[k]));
            for (int i = 0; i < 3; ++i) R.inv_scale[k][i] = 1.0 / im.rpc[7 + i];
        }
        // the blunder pass returns its NCC as a float: it keeps the reference's
        // coordinates, the seed-DEM pass's rounded NCC does not need them
        auto kernel = ncc_out ? (b >= 0 ? sample_raster_kernel<true, 2> : sample_raster_kernel<true, 1>)
                              : (b >= 0 ? sample_raster_kernel<false, 2> : sample_raster_kernel<false, 1>);
        kernel<<<(unsigned)tiles, dim3(kTileW, kTileH), 0, s>>>(
            dP, R, a, b, h_rasters[a], b >= 0 ? h_rasters[b] : nullptr, steps + a * tiles,
            steps + (b >= 0 ? b : a) * tiles, ow, oh, im_res, use_b, tx, 4.0 * delta);
        ++*launches;
    };
    // a pixel is projected to longitude and latitude once for the reference and
    // the first target image together
    int first = -1;
    for (int ti = 1; ti < hP.num_images && first < 0; ++ti)
        if (hP.im[ti].selected && ti != hP.ref) first = ti;
    sample(hP.ref, first);
    for (int ti = 1; ti < hP.num_images; ++ti)
        if (hP.im[ti].selected && ti != hP.ref && ti != first) sample(ti, -1);
    node_set_kernel<<<blocks_for(n_nodes, 256), 256, 0, s>>>(
        dP, set, steps, tx, tiles, ow, oh, im_res, H, ncc_out ? nullptr : node_steps);
    e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    const SampledArgs A{(const double2 *const *)rasters, set, ow, oh, im_res, H,
                        ncc_out ? (H - 1) * (H - 1) : (H + 1) * (H + 1), use_b, node_steps,
                        (float)(2.0 * delta)};
    *launches += 3;
    return ncc_out ? launch_nodes<true>(dP, n_nodes, A, gout, ncc_out, todo, n_todo, s)
                   : launch_nodes<false>(dP, n_nodes, A, gout, ncc_out, todo, n_todo, s);
}

cudaError_t launch_ortho_raster(const DevLevel *dP, double2 *const *cd, int64_t ow, int64_t oh,
                                double im_res, int use_b, cudaStream_t s) {
    ortho_raster_kernel<<<blocks_for(ow * oh, 256), 256, 0, s>>>(dP, cd, ow, oh, im_res, use_b);
    return cudaGetLastError();
}

cudaError_t launch_seeddem(const DevLevel *dP, int64_t n_nodes, double2 *const *cd, int64_t ow,
                           int64_t oh, double im_res, int H, int use_b, vll_ugrid *gout,
                           cudaStream_t s) {
    const OrthoArgs A{cd, ow, oh, im_res, H, (H + 1) * (H + 1), use_b};
    seeddem_kernel<<<blocks_for(n_nodes, 128), 128, 0, s>>>(dP, A, gout);
    return cudaGetLastError();
}

cudaError_t launch_blunder(const DevLevel *dP, int64_t n_nodes, double2 *const *cd, int64_t ow,
                           int64_t oh, double im_res, int H, vll_ugrid *gout, float *ncc_out,
                           cudaStream_t s) {
    const OrthoArgs A{cd, ow, oh, im_res, H, (H - 1) * (H - 1), 1};
    blunder_kernel<<<blocks_for(n_nodes, 128), 128, 0, s>>>(dP, A, gout, ncc_out);
    return cudaGetLastError();
}

}  // namespace vll
