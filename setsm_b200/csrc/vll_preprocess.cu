// vll_preprocess.cu -- image preprocessing on the device, bit-exact with
// SETSM's L2 functions (SubFunctions.cpp:2418-2560, Template.hpp:45-131):
// Sobel magnitude, 18-bin gradient orientation, 9x9 Gaussian 2x pyramid.
// The reference computes in FP64 in a fixed order; every output here is the
// same integer.  Where an output is a rounding or an argmax of FP64 values,
// it is decided from cheaper values whose distance from the reference's is
// bounded, and recomputed in the reference's own order when that bound does
// not decide it.  Compiled with -fmad=false.
#include <cmath>
#include <cstdint>
#include <cuda_runtime.h>

#include "vll_internal.h"
#include "vll_split.h"

namespace vll {

// ---- Sobel ------------------------------------------------------------------
// MakeSobelMagnitudeImage, SubFunctions.cpp:2418-2471: magnitude, and instead
// of the int16 degree image what Orientation consumes from it: the 20-degree
// bin of floor(atan2(gy, gx) * 180 / PI) after the [0, 360) wrap.
//
// The bin needs no arctangent: gx and gy are integers up to 2^18, no ratio of
// which comes closer than 1.8e-10 degrees to a boundary of 20, 40, 60 or 80
// degrees (continued fractions), 10^4 times the rounding of the reference's
// angle, so four FP64 comparisons |gy| > |gx| tan(20 k) give the reference's
// bin (and 0, 90, 180, 270 degrees, the bins 0, 4, 9, 13, are exact in it).
__device__ __forceinline__ uint8_t gradient_bin(int gx, int gy) {
    const double a = (double)abs(gx), b = (double)abs(gy);
    const int n = (int)(b > a * 0.36397023426620234) + (int)(b > a * 0.83909963117727993) +
                  (int)(b > a * 1.7320508075688772) + (int)(b > a * 5.6712818196177093);
    if (gx >= 0) return (uint8_t)(gy >= 0 ? n : 17 - n);
    return (uint8_t)(gy > 0 ? 8 - n : 9 + n);
}

// (uint16)(sqrt(gx^2 + gy^2) + 0.5): for gradients below 2^15 the sum of
// squares s is a 31-bit integer and k = floor(sqrt(s) + 0.5) is the integer
// with k^2 - k < s <= k^2 + k, found from an FP32 root and one correction
// (FP64's rounding of sqrt(s) cannot cross it: s is at least 1/4 away).
__device__ __forceinline__ uint16_t gradient_mag(int gx, int gy) {
    if (abs(gx) < 32768 && abs(gy) < 32768) {
        const uint32_t s = (uint32_t)(gx * gx) + (uint32_t)(gy * gy);
        uint32_t k = (uint32_t)(sqrtf((float)s) + 0.5f);
        if (k * k - k >= s && k > 0) --k;
        if (k * k + k < s) ++k;
        return (uint16_t)k;
    }
    const double x = (double)gx, y = (double)gy;
    const double m = sqrt(__dadd_rn(__dmul_rn(x, x), __dmul_rn(y, y)));
    return (uint16_t)__dadd_rn(m, 0.5);
}

// Rows per thread: three row registers slide down, so a pixel costs three
// loads instead of eight (0.19 ms for a 6001 x 5000 pyramid; 0.41 ms with a
// pixel per thread and the FP64 arctangent and root).
constexpr int kSobelRows = 4;

__global__ void __launch_bounds__(256) sobel_kernel(const uint16_t *__restrict__ s, uint32_t w,
                                                    uint32_t h, uint16_t *__restrict__ mag,
                                                    uint8_t *__restrict__ bin, int64_t tiles_x) {
    const int64_t ty = blockIdx.x / tiles_x, tx = blockIdx.x - ty * tiles_x;
    const int64_t x = tx * 32 + threadIdx.x;
    const int64_t y0 = (ty * 8 + threadIdx.y) * kSobelRows;
    if (x >= (int64_t)w || y0 >= (int64_t)h) return;
    const bool edge_x = x == 0 || x == (int64_t)w - 1;
    int a[3] = {0, 0, 0}, b[3] = {0, 0, 0}, c[3] = {0, 0, 0};
    auto load = [&](int64_t y, int v[3]) {
        if (edge_x || y < 0 || y >= (int64_t)h) return;
        const uint16_t *r = s + y * w + x;
        v[0] = r[-1];
        v[1] = r[0];
        v[2] = r[1];
    };
    load(y0 - 1, a);
    load(y0, b);
#pragma unroll
    for (int i = 0; i < kSobelRows; ++i) {
        const int64_t y = y0 + i;
        if (y >= (int64_t)h) return;
        load(y + 1, c);
        uint16_t m = 0;
        uint8_t q = 0;   // edge pixels: dir 0 -> bin 0
        if (!edge_x && y > 0 && y < (int64_t)h - 1) {
            const int gx = -a[0] + a[2] - 2 * b[0] + 2 * b[2] - c[0] + c[2];
            const int gy = a[0] + 2 * a[1] + a[2] - c[0] - 2 * c[1] - c[2];
            m = gradient_mag(gx, gy);
            q = gradient_bin(gx, gy);
        }
        mag[y * w + x] = m;
        bin[y * w + x] = q;
#pragma unroll
        for (int j = 0; j < 3; ++j) {
            a[j] = b[j];
            b[j] = c[j];
        }
    }
}

// ---- Orientation --------------------------------------------------------------
// Orientation, SubFunctions.cpp:2473-2560: Gaussian-weighted 18-bin histogram
// of gradient magnitude over a 13x13 disc-like window (113 samples), coarse
// 4-way sub-bin vote, then the best bin inside the winning sub-bin.
//
// What bounds it: the histogram update of each sample, a read and a write of
// the pixel's bin.  The bins are shared-memory columns, one per thread, so
// the dynamic index costs no bank conflict, and a thread keeps two adjacent
// pixels' bins side by side: one 64-bit read-modify-write (a packed FP32 FMA)
// adds a sample to both, 126 updates for the pair's 226 samples.  That is
// 8.9 bytes of shared memory per sample and pixel, the kernel's floor.  FP32
// sums are within kOriBand / 2 of the reference's FP64 ones, so a vote whose
// two best differ by more is decided; the rest (well under 1 % of textured
// pixels) and the pixels whose window leaves the image are recomputed in
// FP64 in the reference's order, by the block's threads together.  A five-level
// pyramid of a 6001 x 5000 image: 2.03 ms, the shared-memory pipe 89 % busy
// (39.4 ms with 18 FP64 bins per thread in local memory).
constexpr int kOriHalf = 7;                    // template 15: 2 * 7 - 1 = 13 rows
constexpr int kOriR = kOriHalf - 1;            // window radius
constexpr int kOriTW = 64, kOriTH = 16;        // pixels of a block
constexpr int kOriSW = kOriTW + 2 * kOriR;     // staged columns
constexpr int kOriSH = kOriTH + 2 * kOriR;
constexpr int kOriThreads = 256;
// Twice the relative error of an FP32 sum of at most 113 rounded products of
// rounded factors: 2 * (113 + 5 + 3) * 2^-24 = 1.45e-5.
constexpr float kOriBand = 2e-5f;

struct OriWeights {
    double w[(2 * kOriR + 1) * (2 * kOriR + 1)];   // exp(-(r^2 + c^2) / 4.5)
};

// Columns of the window at row distance ar (numcols, SubFunctions.cpp:8).
__host__ __device__ constexpr int ori_cols(int ar) {
    return ar == 0 ? 6 : (ar <= 3 ? 5 : (ar == 4 ? 4 : (ar == 5 ? 3 : 0)));
}
// exp(-d^2 / 4.5): the separable factors of the weights
__host__ __device__ constexpr float ori_g(int d) {
    return d == 0   ? 1.0f
           : d == 1 ? 0.80073740f
           : d == 2 ? 0.41111229f
           : d == 3 ? 0.13533528f
           : d == 4 ? 0.028565501f
           : d == 5 ? 0.0038659201f
                    : 0.00033546263f;
}
// sub-bin of a bin, (int)(bin / 4.6), and the bins [lo, hi) searched in it,
// (int)(sub * 4.6) and (int)(sub * 4.6 + 4.6)
__host__ __device__ constexpr int ori_sub(int b) { return b < 5 ? 0 : (b < 10 ? 1 : (b < 14 ? 2 : 3)); }
__host__ __device__ constexpr int ori_lo(int s) { return s == 0 ? 0 : (s == 1 ? 4 : (s == 2 ? 9 : 13)); }
__host__ __device__ constexpr int ori_hi(int s) { return s == 0 ? 4 : (s == 1 ? 9 : (s == 2 ? 13 : 18)); }

// The reference's own evaluation of pixel (mr, mc): FP64 sums in its order,
// its window bounds (the column lower bound is max(-mask_row, -numcols) and
// addresses may wrap into the previous row; those before the first pixel add
// 0).  col: the thread's 18 + 4 doubles, `stride` apart.
__device__ __noinline__ uint8_t orientation_exact(const uint16_t *__restrict__ mag,
                                                  const uint8_t *__restrict__ bin_img, int64_t W,
                                                  int64_t H, int64_t mr, int64_t mc,
                                                  const OriWeights &wt, double *col, int stride) {
    constexpr int sz = 2 * kOriR + 1;
    for (int i = 0; i < 22; ++i) col[i * stride] = 0.0;
    const int64_t r_lo = (-mr > -kOriR) ? -mr : -kOriR;
    const int64_t r_hi = (H - mr - 1 < kOriR) ? H - mr - 1 : kOriR;
    for (int64_t r = r_lo; r <= r_hi; ++r) {
        const int dcol = ori_cols((int)(r < 0 ? -r : r));
        const int64_t c_lo = (-mr > -dcol) ? -mr : -dcol;
        const int64_t c_hi = (dcol < W - mc - 1) ? dcol : W - mc - 1;
        for (int64_t c = c_lo; c <= c_hi; ++c) {
            const int64_t idx = (mr + r) * W + (mc + c);
            if (idx < 0) continue;
            const int bi = bin_img[idx];
            const double v = __dmul_rn((double)mag[idx], wt.w[(kOriR + r) * sz + (kOriR + c)]);
            col[bi * stride] = __dadd_rn(col[bi * stride], v);
            double *sb = col + (18 + ori_sub(bi)) * stride;
            *sb = __dadd_rn(*sb, v);
        }
    }
    double mx = -100;
    int sub = 0, th = 0;
    for (int i = 0; i < 4; ++i)
        if (col[(18 + i) * stride] > mx) {
            mx = col[(18 + i) * stride];
            sub = i;
        }
    mx = -100;
    for (int i = ori_lo(sub); i < ori_hi(sub); ++i)
        if (col[i * stride] > mx) {
            mx = col[i * stride];
            th = i;
        }
    return (uint8_t)th;
}

// The best bin from one pixel's FP32 bins, or -1 when the band does not
// decide it.  All-zero votes are zero in the reference too (its first bin).
__device__ __forceinline__ int orientation_of(const float (&b)[18]) {
    const float s[4] = {b[0] + b[1] + b[2] + b[3] + b[4], b[5] + b[6] + b[7] + b[8] + b[9],
                        b[10] + b[11] + b[12] + b[13], b[14] + b[15] + b[16] + b[17]};
    float m1 = s[0], m2 = -1.f;
    int sub = 0;
#pragma unroll
    for (int i = 1; i < 4; ++i) {
        if (s[i] > m1) {
            m2 = m1;
            m1 = s[i];
            sub = i;
        } else if (s[i] > m2) {
            m2 = s[i];
        }
    }
    if (m1 > 0.f && m2 >= m1 - m1 * kOriBand) return -1;
    const int lo = ori_lo(sub), hi = ori_hi(sub);
    float t1 = -1.f, t2 = -2.f;
    int th = 0;
#pragma unroll
    for (int i = 0; i < 18; ++i) {
        if (i < lo || i >= hi) continue;
        if (b[i] > t1) {
            t2 = t1;
            t1 = b[i];
            th = i;
        } else if (b[i] > t2) {
            t2 = b[i];
        }
    }
    if (t1 > 0.f && t2 >= t1 - t1 * kOriBand) return -1;
    return th;
}

// One window row of the pixel pair: texels at columns -D .. D + 1 from the
// left pixel (staged words in aligned pairs), each adding to both pixels'
// bins; a weight outside its pixel's window is 0.
template <int D>
__device__ __forceinline__ void ori_row(const uint32_t *__restrict__ t, float gr, char *hist) {
    constexpr int c_first = (D & 1) ? -(D + 1) : -D;   // even
#pragma unroll
    for (int c = c_first; c <= D + 1; c += 2) {
        const uint2 q = *reinterpret_cast<const uint2 *>(t + c);
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            const int cc = c + j;
            if (cc < -D || cc > D + 1) continue;
            const uint32_t word = j ? q.y : q.x;
            const float m =
                __fadd_rn(__int_as_float((word & 0xffffu) | 0x4B000000u), -8388608.0f) * gr;
            float2 *p = reinterpret_cast<float2 *>(hist + (word >> 16));
            const float w0 = cc <= D ? ori_g(cc < 0 ? -cc : cc) : 0.f;
            const int c1 = cc - 1;
            const float w1 = c1 >= -D ? ori_g(c1 < 0 ? -c1 : c1) : 0.f;
            *p = __ffma2_rn(make_float2(m, m), make_float2(w0, w1), *p);
        }
    }
}

// Blocks [0, edge_blocks): the pixels whose window leaves the image (a frame
// kOriR wide), one per thread; the others: a tile of interior pixels each.
__global__ void __launch_bounds__(kOriThreads) orientation_kernel(
    const uint16_t *__restrict__ mag, const uint8_t *__restrict__ bin_img, uint32_t w, uint32_t h,
    const __grid_constant__ OriWeights wt, uint8_t *__restrict__ ori, int64_t edge_blocks, int64_t n_edge,
    int64_t tiles_x) {
    // 22 columns of 8 bytes per thread: 18 float2 bins of a pixel pair, or 18
    // + 4 FP64 sums of one pixel; the staged tile and the list of undecided
    // pixels follow
    extern __shared__ __align__(16) unsigned char sm[];
    double *exact_col = reinterpret_cast<double *>(sm) + threadIdx.x;
    char *hist = reinterpret_cast<char *>(sm) + threadIdx.x * 8;
    uint32_t *tile = reinterpret_cast<uint32_t *>(sm + 22 * kOriThreads * 8);
    uint16_t *todo = reinterpret_cast<uint16_t *>(tile + kOriSW * kOriSH);
    int *n_todo = reinterpret_cast<int *>(todo + kOriTW * kOriTH);
    const int64_t W = w, H = h;
    if ((int64_t)blockIdx.x < edge_blocks) {
        int64_t i = (int64_t)blockIdx.x * kOriThreads + threadIdx.x;
        if (i >= n_edge) return;
        int64_t y, x;
        if (W <= 2 * kOriR || H <= 2 * kOriR) {   // every pixel
            y = i / W;
            x = i - y * W;
        } else if (i < 2 * kOriR * W) {           // the top and bottom rows
            y = i / W;
            x = i - y * W;
            if (y >= kOriR) y += H - 2 * kOriR;
        } else {                                  // the left and right columns between them
            i -= 2 * kOriR * W;
            y = i / (2 * kOriR);
            x = i - y * (2 * kOriR);
            y += kOriR;
            if (x >= kOriR) x += W - 2 * kOriR;
        }
        ori[y * W + x] = orientation_exact(mag, bin_img, W, H, y, x, wt, exact_col, kOriThreads);
        return;
    }
    const int64_t b = (int64_t)blockIdx.x - edge_blocks;
    const int64_t tyb = b / tiles_x;
    // tile origin: the first interior pixel of the block
    const int64_t y0 = kOriR + tyb * kOriTH, x0 = kOriR + (b - tyb * tiles_x) * kOriTW;
    if (threadIdx.x == 0) *n_todo = 0;
    for (int i = threadIdx.x; i < kOriSW * kOriSH; i += kOriThreads) {
        const int r = i / kOriSW, c = i - r * kOriSW;
        const int64_t y = y0 - kOriR + r, x = x0 - kOriR + c;
        uint32_t v = 0;
        if (y < H && x < W) {
            // magnitude, and the byte offset of the bin's row of columns
            v = (uint32_t)mag[y * W + x] | ((uint32_t)bin_img[y * W + x] * (kOriThreads * 8u)) << 16;
        }
        tile[i] = v;
    }
    __syncthreads();
    const int px = (threadIdx.x & 31) * 2;
    const float g[7] = {ori_g(0), ori_g(1), ori_g(2), ori_g(3), ori_g(4), ori_g(5), ori_g(6)};
#pragma unroll 1
    for (int ty = threadIdx.x >> 5; ty < kOriTH; ty += kOriThreads / 32) {
#pragma unroll
        for (int i = 0; i < 18; ++i)
            *reinterpret_cast<float2 *>(hist + i * kOriThreads * 8) = make_float2(0.f, 0.f);
        const uint32_t *t = tile + (ty + kOriR) * kOriSW + px + kOriR;
        ori_row<6>(t, g[0], hist);
#pragma unroll 1
        for (int sgn = -1; sgn <= 1; sgn += 2) {
            const int s = sgn * kOriSW;
            ori_row<5>(t + s, g[1], hist);
            ori_row<5>(t + 2 * s, g[2], hist);
            ori_row<5>(t + 3 * s, g[3], hist);
            ori_row<4>(t + 4 * s, g[4], hist);
            ori_row<3>(t + 5 * s, g[5], hist);
            ori_row<0>(t + 6 * s, g[6], hist);
        }
        float b0[18], b1[18];
#pragma unroll
        for (int i = 0; i < 18; ++i) {
            const float2 v = *reinterpret_cast<const float2 *>(hist + i * kOriThreads * 8);
            b0[i] = v.x;
            b1[i] = v.y;
        }
        const int64_t y = y0 + ty;
#pragma unroll
        for (int p = 0; p < 2; ++p) {
            const int64_t x = x0 + px + p;
            if (y >= H - kOriR || x >= W - kOriR) continue;
            const int th = p == 0 ? orientation_of(b0) : orientation_of(b1);
            if (th >= 0)
                ori[y * W + x] = (uint8_t)th;
            else
                todo[atomicAdd(n_todo, 1)] = (uint16_t)(ty * kOriTW + px + p);
        }
    }
    __syncthreads();
    for (int i = threadIdx.x; i < *n_todo; i += kOriThreads) {
        const int64_t y = y0 + todo[i] / kOriTW, x = x0 + todo[i] % kOriTW;
        ori[y * W + x] = orientation_exact(mag, bin_img, W, H, y, x, wt, exact_col, kOriThreads);
    }
}

// ---- pyramid ------------------------------------------------------------------
// CreateImagePyramid<uint16>(.., 9, 1.5), Template.hpp:82-131: the truncated
// 81-term FP64 sum.  The filter is separable up to rounding, so a block forms
// rows sums of nine columns (pairs at equal distance added as integers) and
// then column sums of nine of those: 33 FP64 operations per output instead
// of 162.  The two sums differ by less than 1e-8 (65535 * 81 roundings), so
// the truncation is the reference's unless an integer lies within 1e-6 of
// the sum; such a pixel is summed again in the reference's order.  6001 x 5000
// and its three halvings: 0.156 ms (0.426 ms as the 81-term sum).
struct PyrFilter {
    double f[81];   // the 9x9 filter
    double g[5];    // its separable factor, by distance
};
// A 32-bit unsigned integer as a double, by its bits in 2^52's mantissa (one
// FP64 addition; the conversion instruction runs at a quarter of that rate).
__device__ __forceinline__ double dbl_of(int v) {
    return __dadd_rn(__hiloint2double(0x43300000, v), -4503599627370496.0);
}

constexpr int kPyrW = 32, kPyrH = 16;              // outputs of a block
constexpr int kPyrSW = 2 * kPyrW + 8, kPyrSH = 2 * kPyrH + 7;

__global__ void __launch_bounds__(256) pyramid_kernel(const uint16_t *__restrict__ src, uint32_t w,
                                                      uint32_t h,
                                                      const __grid_constant__ PyrFilter flt,
                                                      uint16_t *__restrict__ out,
                                                      int64_t tiles_x) {
    __shared__ uint16_t tile[kPyrSH][kPyrSW];
    __shared__ double rows[kPyrSH][kPyrW];
    const int64_t ow = w / 2, oh = h / 2;
    const int64_t tyb = blockIdx.x / tiles_x, txb = blockIdx.x - tyb * tiles_x;
    const int64_t r0 = tyb * kPyrH, c0 = txb * kPyrW;
    for (int i = threadIdx.x; i < kPyrSH * kPyrSW; i += 256) {
        const int r = i / kPyrSW, c = i - r * kPyrSW;
        const int64_t y = 2 * r0 - 4 + r, x = 2 * c0 - 4 + c;
        tile[r][c] = (y >= 0 && x >= 0 && y < (int64_t)h && x < (int64_t)w) ? src[y * w + x] : 0;
    }
    __syncthreads();
    for (int i = threadIdx.x; i < kPyrSH * kPyrW; i += 256) {
        const int r = i / kPyrW, c = i - r * kPyrW;
        const uint16_t *t = &tile[r][2 * c];
        double v = flt.g[0] * dbl_of(t[4]);
#pragma unroll
        for (int k = 1; k <= 4; ++k) v = fma(flt.g[k], dbl_of((int)t[4 - k] + (int)t[4 + k]), v);
        rows[r][c] = v;
    }
    __syncthreads();
    for (int i = threadIdx.x; i < kPyrH * kPyrW; i += 256) {
        const int r = i / kPyrW, c = i - r * kPyrW;
        const int64_t orow = r0 + r, ocol = c0 + c;
        if (orow >= oh || ocol >= ow) continue;
        const int64_t y = 2 * orow, x = 2 * ocol;
        uint16_t o;
        if (y >= 4 && x >= 4 && y + 4 < (int64_t)h && x + 4 < (int64_t)w) {
            double v = flt.g[0] * rows[2 * r + 4][c];
#pragma unroll
            for (int k = 1; k <= 4; ++k)
                v = fma(flt.g[k], rows[2 * r + 4 - k][c] + rows[2 * r + 4 + k][c], v);
            if (v != 0.0 && fabs(v - rint(v)) < 1e-6) {
                v = 0;
#pragma unroll 1
                for (int l = -4; l <= 4; ++l)
#pragma unroll 1
                    for (int k = -4; k <= 4; ++k)
                        v = __dadd_rn(v, __dmul_rn(flt.f[(l + 4) * 9 + (k + 4)],
                                                   (double)tile[2 * r + 4 + l][2 * c + 4 + k]));
            }
            o = (uint16_t)v;
        } else {
            o = tile[2 * r + 4][2 * c + 4];   // the window leaves the image: the pixel itself
        }
        out[orow * ow + ocol] = o;
    }
}

cudaError_t launch_sobel(const uint16_t *src, uint32_t w, uint32_t h, uint16_t *mag, uint8_t *bin,
                         cudaStream_t s) {
    const int64_t tx = ((int64_t)w + 31) / 32;
    const int64_t ty = ((int64_t)h + 8 * kSobelRows - 1) / (8 * kSobelRows);
    if (tx * ty > 0x7fffffff) return cudaErrorInvalidValue;
    sobel_kernel<<<(unsigned)(tx * ty), dim3(32, 8), 0, s>>>(src, w, h, mag, bin, tx);
    return cudaGetLastError();
}

cudaError_t launch_orientation(const uint16_t *mag, const uint8_t *bin, uint32_t w, uint32_t h,
                               const double *wt, uint8_t *ori, cudaStream_t s) {
    OriWeights ow;
    for (int i = 0; i < (2 * kOriR + 1) * (2 * kOriR + 1); ++i) ow.w[i] = wt[i];
    const int64_t W = w, H = h;
    const bool small = W <= 2 * kOriR || H <= 2 * kOriR;
    const int64_t iw = small ? 0 : W - 2 * kOriR, ih = small ? 0 : H - 2 * kOriR;
    const int64_t n_edge = W * H - iw * ih;
    const int64_t edge_blocks = (n_edge + kOriThreads - 1) / kOriThreads;
    const int64_t tiles_x = (iw + kOriTW - 1) / kOriTW, tiles_y = (ih + kOriTH - 1) / kOriTH;
    const int64_t blocks = edge_blocks + tiles_x * tiles_y;
    if (blocks > 0x7fffffff) return cudaErrorInvalidValue;
    const size_t smem = 22 * kOriThreads * 8 + kOriSW * kOriSH * 4 + kOriTW * kOriTH * 2 + 16;
    cudaError_t e = ensure_smem_limit((const void *)orientation_kernel, smem);
    if (e != cudaSuccess) return e;
    orientation_kernel<<<(unsigned)blocks, kOriThreads, smem, s>>>(
        mag, bin, w, h, ow, ori, edge_blocks, n_edge, tiles_x > 0 ? tiles_x : 1);
    return cudaGetLastError();
}

cudaError_t launch_pyramid(const uint16_t *src, uint32_t w, uint32_t h, const double *f,
                           uint16_t *out, cudaStream_t s) {
    PyrFilter flt;
    for (int i = 0; i < 81; ++i) flt.f[i] = f[i];
    // f[i][j] = g[|i|] g[|j|] up to rounding; sum(f) = 1 gives g[0]^2 = f[0][0]
    flt.g[0] = sqrt(f[4 * 9 + 4]);
    for (int k = 1; k <= 4; ++k) flt.g[k] = f[4 * 9 + 4 + k] / flt.g[0];
    const int64_t tx = ((int64_t)(w / 2) + kPyrW - 1) / kPyrW;
    const int64_t ty = ((int64_t)(h / 2) + kPyrH - 1) / kPyrH;
    if (tx * ty > 0x7fffffff) return cudaErrorInvalidValue;
    pyramid_kernel<<<(unsigned)(tx * ty), 256, 0, s>>>(src, w, h, flt, out, tx);
    return cudaGetLastError();
}

}  // namespace vll
