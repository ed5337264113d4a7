// vll_stream.cuh -- what the streaming kernels of the split pipeline share: the
// window kernel (vll_split.cu) and the combined levels' kernel
// (vll_combined.cu).  Level sets, the FP32 error band, the RPC cubics and the
// per-node state in shared memory.
#pragma once

#include "vll_exact.cuh"
#include "vll_window.cuh"

namespace vll {

// Half-width of the FP32 error band of rho: decisions whose FP32 inputs lie
// closer than this to their boundary are settled in FP64, which holds while
// the FP32 error of rho stays below half of it.  Over textured scenes it stays
// below 4.4e-7 (4.4 M slots of 7x7 and 11x11 windows, tests/test_gpu_accuracy.py;
// combined levels 2.8e-7 over 0.9 M).  Combined levels of images with
// saturated, constant or quantised areas: 2.5e-6 at one of 8 M slots, 2e-6 at
// no other (see kCentreFloor).
constexpr float kBand = 4e-6f;
constexpr double kEdge = 1e-7;          // coordinate distance to an integer / clamp
constexpr int kSlotCap = 512;           // slots per node the peak kernel holds in shared memory
constexpr int kWarpPerSlotMax = 8;      // re-checks per round done a warp per slot (more: a lane each)
constexpr int kMaxRounds = 3;           // scan / re-check rounds before a full FP64 pass

// Per-slot markers in the rho buffer (.x):
constexpr float kNotEvaluated = INFINITY;    // slot skipped (range / image bounds)
constexpr float kRejected = -INFINITY;       // orientation check failed

// ---------------------------------------------------------------------------
// Level set: the levels matched by one pass of the pipeline (one level for a
// VerticalLineLocus call; many tiles and pyramid levels for a batch).  Their
// nodes are numbered consecutively: global node g belongs to the level l with
// base[l] <= g < base[l + 1] and is that level's node g - base[l].  Per-node
// and per-slot work arrays are indexed by g.
// ---------------------------------------------------------------------------
struct LevelSet {
    const DevLevel *lv;       // [n] level blocks (device)
    const int64_t *base;      // [n + 1] first global node of each level (device)
    int n;
    int64_t total;            // base[n]
};

__device__ __forceinline__ int level_of(const LevelSet &S, int64_t g) {
    int lo = 0, hi = S.n - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (__ldg(S.base + mid) <= g)
            lo = mid;
        else
            hi = mid - 1;
    }
    return lo;
}

// ---------------------------------------------------------------------------
// geometry helpers of the window kernel
// ---------------------------------------------------------------------------
// Per-node RPC: normalised L, P (with the reference's +-360 wrap) and the
// four cubics in the normalised height.  RPC00B terms grouped by power of H:
//   a0: 1 L P LP LL PP LLL LPP LLP PPP   a1: H LH PH PLH LLH PPH
//   a2: HH LHH PHH                        a3: HHH
// Coefficients a0..a3 of one of the four RPC cubics (j: LINE_NUM, LINE_DEN,
// SAMP_NUM, SAMP_DEN) as a polynomial in the normalised height, for fixed
// normalised L, P (with the reference's +-360 wrap).
__device__ __forceinline__ void node_horner_poly(const double *rpc, double lon, double lat, int j,
                                                 double *a) {
    double L = (lon - rpc[2]) / rpc[7];
    double P = (lat - rpc[3]) / rpc[8];
    if (L < -10.0 || L > 10.0) {
        const double X = lon > 0 ? lon - 360 : lon + 360;
        L = (X - rpc[2]) / rpc[7];
    }
    if (P < -10.0 || P > 10.0) {
        const double Y = lat > 0 ? lat - 360 : lat + 360;
        P = (Y - rpc[3]) / rpc[8];
    }
    const double *c = rpc + 10 + 20 * j;
    a[0] = c[0] + c[1] * L + c[2] * P + c[4] * L * P + c[7] * L * L + c[8] * P * P +
           c[11] * L * L * L + c[12] * L * P * P + c[14] * L * L * P + c[15] * P * P * P;
    a[1] = c[3] + c[5] * L + c[6] * P + c[10] * P * L + c[17] * L * L + c[18] * P * P;
    a[2] = c[9] + c[13] * L + c[16] * P;
    a[3] = c[19];
}

// Reciprocal for the fast geometry path: FP32 seed refined by two Newton
// steps (relative error ~1e-16).  A seed that is not a finite non-zero float
// sends the slot to the exact projection.
__device__ __forceinline__ double fast_rcp(double v, bool &edge) {
    const float f = __frcp_rn((float)v);
    if (!(fabsf(f) > 0.f && fabsf(f) < 3.0e38f)) edge = true;
    double r = (double)f;
    r = fma(r, fma(-v, r, 1.0), r);
    r = fma(r, fma(-v, r, 1.0), r);
    return r;
}

__device__ __forceinline__ bool near_round(double v) {
    const double x = v * 1000.0;
    return fabs(x - floor(x) - 0.5) < (double)kBand * 1000.0;
}
__device__ __forceinline__ bool near_trunc(double v) {
    const double x = v * 1000.0;
    return fabs(x - rint(x)) < (double)kBand * 1000.0;
}

__device__ __forceinline__ bool bit(const uint32_t *m, int k) { return (m[k >> 5] >> (k & 31)) & 1u; }
__device__ __forceinline__ void set_bit(uint32_t *m, int k) { atomicOr(&m[k >> 5], 1u << (k & 31)); }

// Index of the last evaluated slot before k (or -1); `carry` is the last
// evaluated slot of earlier 32-slot groups.
__device__ __forceinline__ int prev_eval(uint32_t mask, int lane, int carry) {
    const uint32_t below = mask & ((1u << lane) - 1u);
    return below ? (31 - __clz(below)) : carry;
}

// ---------------------------------------------------------------------------
// per-node state of the streaming kernels
// ---------------------------------------------------------------------------
// Warps per window block and the minimum resident blocks per SM (the latter
// sets the register budget: 65536 / (warps * 32 * blocks)).
#ifndef VLL_WIN_WARPS
#define VLL_WIN_WARPS 4
#endif
#ifndef VLL_WIN_MINB
#define VLL_WIN_MINB 3
#endif
constexpr int kWinWarps = VLL_WIN_WARPS;
constexpr int kWinMaxBlocksPerSm = 2048 / (kWinWarps * 32);
constexpr int kZeroCap = 32;          // zero intensity texels listed per staged group

// Node flags of the window kernel
constexpr uint32_t kNfCmr = 1u;       // memory-tight route (FindPeakNcc on the values)
constexpr uint32_t kNfOri = 2u;       // orientation-difference test (level >= 3)
constexpr uint32_t kNfVox = 4u;       // voxel rows written
constexpr uint32_t kNfChc = 8u;       // check_height_change (max_WNCC written)
constexpr uint32_t kNfGncc = 16u;     // rho blends the INCC with the node's GNCC
constexpr uint32_t kNfVec = 32u;      // image rows 16-byte aligned (vector staging)
constexpr uint32_t kNfTma = 64u;      // the level has tensor maps for its footprints
constexpr uint32_t kNfDbg = 128u;     // per-slot debug values written

// Per-node state of the window kernel in shared memory: the RPC cubics, the
// level constants the slot loop reads (here rather than from the level block
// in global memory), the record folded by lane 0 and the streamed scan's
// carry.  A warp holds two: the node of the group being evaluated and the
// node of the group being fetched.
struct NodeCtx {
    double horner[2][4][4];           // [image][num/den poly][a0..a3]
    double hnorm[2][2];               // [image] {h_off, 1 / h_scale}
    double geo[2][8];                 // [image] adj0, adj1, rpc0, rpc1, rpc5, rpc6, sx, sy
    double inv_s, hbase, hstep, bin_angle, alpha, gterm;
    const uint16_t *img[2], *mag[2];
    const uint8_t *ori[2];
    const DevLevel *P;
    vll_voxel *vrow;
    int64_t gn, pt;
    uint32_t w[2], h[2];
    int tma_w[2], tma_h[2];
    int K, H, start_H, end_H;
    uint32_t flags;
    vll_nccresult R;
    float pre_v;                      // streamed scan: the last evaluated slot's value,
    int pre_dir, pre_k, have;         // direction and index, and whether there is one
};

// The constants of the launch's first level, loaded once per block: node
// set-ups on that level (every node of a single-level call) read them from
// shared memory and fetch only the node's own records from global memory.
struct LevelConst {
    double rpc[2][90];                // [image] RPC00B block (offsets, scales, 4 x 20 terms)
    double geo[2][8];                 // as NodeCtx::geo
    double inv_s, hstep, bin_angle, alpha, beta;
    const uint16_t *img[2], *mag[2];
    const uint8_t *ori[2];
    uint32_t w[2], h[2];
    int tma_w[2], tma_h[2];
    int H, is_ra, cmr, check_ortho, voxels;
    uint32_t flags;                   // kNfOri | kNfVec | kNfTma | kNfDbg
};

// Per-warp shared state of the window kernel.
struct WinShared {
    NodeCtx node[2];
    uint32_t zl[kZeroCap];            // zero intensity texels of the staged boxes
    int zn;                           // their count (more than kZeroCap: not listed)
    uint64_t mbar;                    // completion of the group's tile copies
    const DevLevel *tmap_level;       // level whose tensor maps lane 0 has acquired
};

__host__ __device__ constexpr size_t win_level_offset() {
    return (sizeof(WinShared) * kWinWarps + 15) & ~(size_t)15;
}

__host__ __device__ constexpr size_t win_boxes_offset() {
    return (win_level_offset() + sizeof(LevelConst) + 15) & ~(size_t)15;
}

// Fills the block's LevelConst from level P (every thread of the block takes
// part; the caller synchronises the block afterwards).
static __device__ void level_const_load(LevelConst &C, const DevLevel &P) {
    const int t = threadIdx.x, nt = blockDim.x;
    for (int i = t; i < 180; i += nt) {
        const int im = i / 90;
        C.rpc[im][i - im * 90] = P.im[im == 0 ? P.ref : 1].rpc[i - im * 90];
    }
    if (t < 2) {
        const DevImage &I = P.im[t == 0 ? P.ref : 1];
        double *g = C.geo[t];
        g[0] = I.adj[0];
        g[1] = I.adj[1];
        g[2] = I.rpc[0];
        g[3] = I.rpc[1];
        g[4] = I.rpc[5];
        g[5] = I.rpc[6];
        g[6] = I.sx;
        g[7] = I.sy;
        C.img[t] = I.img;
        C.mag[t] = I.mag;
        C.ori[t] = I.ori;
        C.w[t] = I.w;
        C.h[t] = I.h;
        C.tma_w[t] = P.tma_w[t];
        C.tma_h[t] = P.tma_h[t];
    } else if (t == 2) {
        const DevImage &ri = P.im[P.ref], &tI = P.im[1];
        C.inv_s = 1.0 / (double)(1 << P.L);
        C.hstep = P.height_step;
        C.bin_angle = P.bin_angle;
        C.alpha = P.alpha;
        C.beta = P.beta;
        C.H = P.H;
        C.is_ra = P.is_ra;
        C.cmr = P.cmr;
        C.check_ortho = P.check_ortho;
        C.voxels = P.vox && !P.cmr && !P.is_ra;
        const bool vec_ok = (ri.w % 8 == 0) && (tI.w % 8 == 0) &&
                            ((reinterpret_cast<uintptr_t>(ri.img) | reinterpret_cast<uintptr_t>(ri.mag) |
                              reinterpret_cast<uintptr_t>(tI.img) |
                              reinterpret_cast<uintptr_t>(tI.mag)) & 15) == 0;
        C.flags = ((!P.is_ra && P.L >= 3) ? kNfOri : 0u) | (vec_ok ? kNfVec : 0u) |
                  (P.tma_w[0] > 0 ? kNfTma : 0u) | (P.dbg_rho ? kNfDbg : 0u);
    }
}

// the TMA tiles follow the boxes, 128-byte aligned (warp_raw is a multiple of 128)
__host__ __device__ constexpr size_t win_raw_offset(int warp_quads) {
    return (win_boxes_offset() + (size_t)kWinWarps * warp_quads * 16 + 127) & ~(size_t)127;
}

// FP32 window statistics of one slot for the level's window half-size
// (the window code is unrolled per half-size; a batch may mix them).
// kStrict: see kCentreFloor.
template <bool kStrict = false>
__device__ __forceinline__ void window_any(int H, const float4 *qr, int rbw, float rfx, float rfy,
                                           const TgtBox &tb, float tfx, float tfy, float c,
                                           float s, float &incc, bool &unsure) {
    switch (H) {
        case 2: window_fp32<2, kStrict>(qr, rbw, rfx, rfy, tb, tfx, tfy, c, s, incc, unsure); break;
        case 3: window_fp32<3, kStrict>(qr, rbw, rfx, rfy, tb, tfx, tfy, c, s, incc, unsure); break;
        case 4: window_fp32<4, kStrict>(qr, rbw, rfx, rfy, tb, tfx, tfy, c, s, incc, unsure); break;
        case 5: window_fp32<5, kStrict>(qr, rbw, rfx, rfy, tb, tfx, tfy, c, s, incc, unsure); break;
        case 6: window_fp32<6, kStrict>(qr, rbw, rfx, rfy, tb, tfx, tfy, c, s, incc, unsure); break;
        default: window_fp32<7, kStrict>(qr, rbw, rfx, rfy, tb, tfx, tfy, c, s, incc, unsure); break;
    }
}

// Fills the warp's node context for global node gn (level lvl, K slots);
// every lane takes part, the context is complete after the final __syncwarp.
static __device__ __noinline__ void node_setup(NodeCtx &N, const LevelSet &LS, int lvl, int64_t gn, int K,
                                        const double *__restrict__ gsum,
                                        const double *__restrict__ gcnt,
                                        const LevelConst *lc, int lane) {
    const DevLevel &P = LS.lv[lvl];
    const int64_t pt = gn - __ldg(LS.base + lvl);
    if (lc) {
        // the level's constants from the block's copy; the node's own
        // records from global memory, one load per lane
        if (lane < 8) {
            const int im = lane >> 2, j = lane & 3;
            const double *rpc = lc->rpc[im];
            node_horner_poly(rpc, P.grid_wgs[2 * pt], P.grid_wgs[2 * pt + 1], j, N.horner[im][j]);
            if (j == 0) {
                N.hnorm[im][0] = rpc[4];
                N.hnorm[im][1] = 1.0 / rpc[9];
            }
        } else if (lane < 26) {
            const int i = lane - 8;   // 16 geo values, then 2 lanes of pointers
            if (i < 16) {
                N.geo[i >> 3][i & 7] = lc->geo[i >> 3][i & 7];
            } else {
                const int im = i - 16;
                N.img[im] = lc->img[im];
                N.mag[im] = lc->mag[im];
                N.ori[im] = lc->ori[im];
                N.w[im] = lc->w[im];
                N.h[im] = lc->h[im];
                N.tma_w[im] = lc->tma_w[im];
                N.tma_h[im] = lc->tma_h[im];
            }
        } else if (lane == 26) {
            const vll_ugrid g = P.gp3[pt];
            const vll_nccresult R = P.ncc[pt];
            const double cnt_g = gcnt ? gcnt[gn] : 0.0;
            const double sum_g = gcnt ? gsum[gn] : 0.0;
            N.P = &P;
            N.gn = gn;
            N.pt = pt;
            N.K = K;
            N.H = lc->H;
            N.start_H = g.minHeight;
            N.end_H = g.maxHeight;
            N.R = R;
            N.hbase = (double)((lc->is_ra || lc->cmr) ? g.minHeight : R.minHeight);
            N.hstep = lc->hstep;
            N.inv_s = lc->inv_s;
            N.bin_angle = lc->bin_angle;
            N.alpha = lc->alpha;
            const bool gncc = lc->check_ortho && cnt_g > 0;
            N.gterm = gncc ? (sum_g / cnt_g) * lc->beta : 0.0;
            N.vrow = lc->voxels ? P.vox + P.vox_off[pt] : nullptr;
            N.flags = lc->flags | (lc->cmr ? kNfCmr : 0u) | (lc->voxels ? kNfVox : 0u) |
                      (R.check_height_change ? kNfChc : 0u) | (gncc ? kNfGncc : 0u);
            N.pre_v = -1.0f;
            N.pre_dir = 0;
            N.pre_k = -1;
            N.have = 0;
        }
        __syncwarp();
        return;
    }
    if (lane < 8) {
        // per-node RPC cubics: lanes 0..7 = (image, polynomial)
        const int im = lane >> 2, j = lane & 3;
        const double *rpc = P.im[im == 0 ? P.ref : 1].rpc;
        node_horner_poly(rpc, P.grid_wgs[2 * pt], P.grid_wgs[2 * pt + 1], j, N.horner[im][j]);
        if (j == 0) {
            N.hnorm[im][0] = rpc[4];
            N.hnorm[im][1] = 1.0 / rpc[9];
        }
    } else if (lane < 10) {
        const int im = lane - 8;
        const DevImage &I = P.im[im == 0 ? P.ref : 1];
        double *g = N.geo[im];
        g[0] = I.adj[0];
        g[1] = I.adj[1];
        g[2] = I.rpc[0];
        g[3] = I.rpc[1];
        g[4] = I.rpc[5];
        g[5] = I.rpc[6];
        g[6] = I.sx;
        g[7] = I.sy;
        N.img[im] = I.img;
        N.mag[im] = I.mag;
        N.ori[im] = I.ori;
        N.w[im] = I.w;
        N.h[im] = I.h;
        N.tma_w[im] = P.tma_w[im];
        N.tma_h[im] = P.tma_h[im];
    } else if (lane == 10) {
        const vll_ugrid g = P.gp3[pt];
        const vll_nccresult R = P.ncc[pt];
        const DevImage &ri = P.im[P.ref], &tI = P.im[1];
        N.P = &P;
        N.gn = gn;
        N.pt = pt;
        N.K = K;
        N.H = P.H;
        N.start_H = g.minHeight;
        N.end_H = g.maxHeight;
        N.R = R;
        N.hbase = (double)((P.is_ra || P.cmr) ? g.minHeight : R.minHeight);
        N.hstep = P.height_step;
        N.inv_s = 1.0 / (double)(1 << P.L);
        N.bin_angle = P.bin_angle;
        N.alpha = P.alpha;
        const double cnt_g = gcnt ? gcnt[gn] : 0.0;
        const bool gncc = P.check_ortho && cnt_g > 0;
        N.gterm = gncc ? (gsum[gn] / cnt_g) * P.beta : 0.0;
        const bool voxels = P.vox && !P.cmr && !P.is_ra;
        N.vrow = voxels ? P.vox + P.vox_off[pt] : nullptr;
        const bool vec_ok = (ri.w % 8 == 0) && (tI.w % 8 == 0) &&
                            ((reinterpret_cast<uintptr_t>(ri.img) | reinterpret_cast<uintptr_t>(ri.mag) |
                              reinterpret_cast<uintptr_t>(tI.img) |
                              reinterpret_cast<uintptr_t>(tI.mag)) & 15) == 0;
        N.flags = (P.cmr ? kNfCmr : 0u) | ((!P.is_ra && P.L >= 3) ? kNfOri : 0u) |
                  (voxels ? kNfVox : 0u) | (R.check_height_change ? kNfChc : 0u) |
                  (gncc ? kNfGncc : 0u) | (vec_ok ? kNfVec : 0u) | (P.tma_w[0] > 0 ? kNfTma : 0u) |
                  (P.dbg_rho ? kNfDbg : 0u);
        N.pre_v = -1.0f;
        N.pre_dir = 0;
        N.pre_k = -1;
        N.have = 0;
    }
    __syncwarp();
}

}  // namespace vll
