// vll_combined.cu -- combined levels of the split pipeline (setsm_code.cpp:
// 6378-6464): the INCC is the mean of the windows at the matched and at the
// next finer pyramid level.  In a file of its own because the window kernel's
// time depends on what it is compiled with: in one file with this kernel it
// took 1 % longer, with its scan shared as functions 3 % (it is bound by
// instruction fetch), so window_kernel keeps the scan below in its own body.
#include <algorithm>
#include <climits>
#include <cmath>

#include "vll_split.h"
#include "vll_stream.cuh"

namespace vll {

// The slot counts of a mixed set's other levels (0 at the combined ones).
__global__ void plain_counts_kernel(const LevelSet S, const int32_t *__restrict__ node_k,
                                    int32_t *__restrict__ plain_k) {
    for (int64_t g = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; g < S.total;
         g += (int64_t)gridDim.x * blockDim.x)
        plain_k[g] = S.lv[level_of(S, g)].combined_incc ? 0 : node_k[g];
}

// Per-lane running values of the streamed scan over a node.
struct PeakScan {
    float vmax = -100.0f, amb = -INFINITY, amb_peak = -INFINITY;
    float b1 = -INFINITY, b2 = -INFINITY;
    bool need = false;
};

// FindPeakNcc streamed over one group of 32 slots (setsm_code.cpp:6672-6752 on
// the FP32 values; every decision within the error band, and every value the
// FP32 pass could not take -- deferred windows, unsure variances, voxel
// truncations near an integer, NaN --, sends the node to the exact pass).
// Lane `lane` holds slot k = ck0 + lane: its status (2 evaluated, 1 rejected),
// rho and INCC (NaN: not decided in FP32).
__device__ __forceinline__ void scan_group(NodeCtx &C, PeakScan &S, int K, uint32_t flags,
                                           int k, int ck0, int status, float rho_v, float incc_v,
                                           bool all_pos, bool deferred, float *wv,
                                           int64_t *fix_list, int64_t fix_cap,
                                           unsigned long long *ctl, int lane) {
    const bool voxels = (flags & kNfVox) != 0;
    const bool ev = k < K && status == 2;
    // a voxel INCC whose truncation FP32 cannot decide needs only its
    // own exact value: the slot is listed for slot_fix_kernel (or,
    // the list full, taken as unusable)
    bool unusable = ev && (isnan(incc_v) || isnan(rho_v));
    if (ev && !unusable && voxels && near_trunc((double)incc_v)) {
        const unsigned long long q = atomicAdd(&ctl[5], 1ull);
        if ((int64_t)q < fix_cap)
            fix_list[q] = C.gn * kSlotCap + k;
        else
            unusable = true;
    }
    if (k < K) wv[k] = unusable ? __int_as_float(0x7fc00000) : rho_v;
    bool band = unusable;
    const uint32_t em = __ballot_sync(0xffffffffu, ev);
    if (em) {
        const int p_in = prev_eval(em, lane, -1);
        const float pv_in = __shfl_sync(0xffffffffu, rho_v, p_in < 0 ? 0 : p_in);
        const bool has_p = p_in >= 0 || C.have;
        const float pv = p_in >= 0 ? pv_in : C.pre_v;
        // direction of this slot: the sign of the change (the
        // reference's sign rule reduces to it); -1 on the first one
        const int td = has_p ? (rho_v > pv) - (rho_v < pv) : -1;
        const int td_in = __shfl_sync(0xffffffffu, td, p_in < 0 ? 0 : p_in);
        const int dp = p_in >= 0 ? td_in : C.pre_dir;
        bool is_peak = false;
        if (ev && !unusable) {
            const float fv = rho_v;
            if (fv > S.vmax) S.vmax = fv;
            if (near_round((double)fv) && fv > S.amb) S.amb = fv;
            if ((flags & kNfCmr) && has_p) {
                if (fabsf(fv - pv) < kBand || fabsf(fv) < kBand || fabsf(pv) < kBand)
                    band = true;
                is_peak = pv != -1.0f && dp > 0 && td < 0;
            }
        }
        // each peak's rounded value and height (its lane), then the
        // ordered top-two fold of this group's peaks (lane 0)
        int q_l = 0;
        float ph_l = 0.f;
        if (is_peak) {
            if (near_round((double)pv) && pv > S.amb_peak) S.amb_peak = pv;
            if (pv > S.b1) {
                S.b2 = S.b1;
                S.b1 = pv;
            } else if (pv > S.b2) {
                S.b2 = pv;
            }
            const int p_slot = p_in >= 0 ? ck0 + p_in : C.pre_k;
            q_l = q_result((double)pv);
            ph_l = (float)__dadd_rn(C.hbase, __dmul_rn((double)p_slot, C.hstep));
        }
        uint32_t pm = __ballot_sync(0xffffffffu, is_peak);
        if (pm) {
            // the fold in registers on every lane (the same values);
            // the replaced maximum re-quantised, q_result(dq_result(x)),
            // is x for every int16 x (|x / 1000 * 1000 - x| < 1e-11)
            vll_nccresult &R = C.R;
            int16_t r0 = R.result0, r1 = R.result1;
            float r2 = R.result2, r3 = R.result3;
            int r4 = R.result4;
            do {
                const int b = __ffs(pm) - 1;
                pm &= pm - 1;
                const int16_t qpre = (int16_t)__shfl_sync(0xffffffffu, q_l, b);
                const float ph = __shfl_sync(0xffffffffu, ph_l, b);
                if (r4 < 10) ++r4;
                if (r0 < qpre) {
                    if (r1 < r0) {
                        r1 = r0;
                        r3 = r2;
                    }
                    r0 = qpre;
                    r2 = ph;
                } else if (r1 < qpre) {
                    r1 = qpre;
                    r3 = ph;
                }
            } while (pm);
            __syncwarp();
            if (lane == 0) {
                R.result0 = r0;
                R.result1 = r1;
                R.result2 = r2;
                R.result3 = r3;
                R.result4 = (decltype(R.result4))r4;
            }
        }
        // carry the last evaluated slot into the next group
        const int last = 31 - __clz(em);
        const float lv = __shfl_sync(0xffffffffu, rho_v, last);
        const int ld = __shfl_sync(0xffffffffu, td, last);
        __syncwarp();
        if (lane == 0) {
            C.pre_v = lv;
            C.pre_dir = ld;
            C.pre_k = ck0 + last;
            C.have = 1;
        }
    }
    if (__any_sync(0xffffffffu, band)) S.need = true;
    if (status == 2 && (flags & kNfDbg))
        C.P->dbg_rho[C.P->dbg_off[C.pt] + k] =
            deferred ? __longlong_as_double(0x7ff8000000000000ll) : (double)rho_v;
    if (k < K && voxels) {
        vll_voxel *v = C.vrow + k;
        if (status == 1) v->flag_cal = 0;
        if (status == 2) {
            if (all_pos) v->flag_cal = 1;
            v->INCC = q_voxel(isnan(incc_v) ? 0.0 : (double)incc_v);
        }
    }
    __syncwarp();
}

// The node's last group has been scanned: writes the node, or queues it with
// its FP32 values for the exact pass.
__device__ __forceinline__ void finish_node(NodeCtx &C, PeakScan &S, int K, uint32_t flags,
                                            const float *wv, float *pend_vals, int64_t pend_cap,
                                            int64_t *pend_node, int64_t *pend_off,
                                            unsigned long long *ctl, int lane) {
    // the maximum, and roundings that could change the maximum or
    // the top two (a peak more than 0.002 + 2 bands below the
    // second best rounds strictly below it)
#pragma unroll
    for (int o = 16; o; o >>= 1) {
        S.vmax = fmaxf(S.vmax, __shfl_xor_sync(0xffffffffu, S.vmax, o));
        S.amb = fmaxf(S.amb, __shfl_xor_sync(0xffffffffu, S.amb, o));
        S.amb_peak = fmaxf(S.amb_peak, __shfl_xor_sync(0xffffffffu, S.amb_peak, o));
        const float o1 = __shfl_xor_sync(0xffffffffu, S.b1, o);
        const float o2 = __shfl_xor_sync(0xffffffffu, S.b2, o);
        const float n1 = fmaxf(S.b1, o1);
        const float n2 = fmaxf(fminf(S.b1, o1), fmaxf(S.b2, o2));
        S.b1 = n1;
        S.b2 = n2;
    }
    if ((flags & kNfChc) && (double)S.amb >= (double)S.vmax - (double)kBand) S.need = true;
    if ((flags & kNfCmr) && S.amb_peak > -1e29f) {
        const double thr =
            (double)(S.b2 > -1e29f ? S.b2 : S.b1) - 0.002 - 2.0 * (double)kBand;
        if ((double)S.amb_peak >= thr) S.need = true;
    }
    if (!S.need) {
        if (lane == 0) {
            vll_nccresult R = C.R;
            if (R.check_height_change) R.max_WNCC = q_result((double)S.vmax);
            C.P->ncc[C.pt] = R;
        }
    } else {
        long long off = -1;
        if (lane == 0) {
            off = (long long)atomicAdd(&ctl[4], (unsigned long long)K);
            if (off + K > pend_cap) off = -1;
            const unsigned long long idx = atomicAdd(&ctl[2], 1ull);
            pend_node[idx] = C.gn;
            pend_off[idx] = off;
        }
        off = __shfl_sync(0xffffffffu, off, 0);
        if (off >= 0)
            for (int kk = lane; kk < K; kk += 32) pend_vals[off + kk] = wv[kk];
    }
    S = PeakScan();
    __syncwarp();
}

// The next finer level of a combined level's two images, per warp.
struct NextLevel {
    const uint16_t *img[2], *mag[2];
    const uint8_t *ori[2];
    double start[2][2];               // py_Startpos_next
    uint32_t w[2], h[2];
    double inv_s;                     // 2^-(L-1)
};

struct CombinedShared {
    NodeCtx node;
    NextLevel next;
};

// Both images' coordinates of a slot at the matched (p) and the next finer
// level (q) from the node's cubics; see node_coord.
__device__ __forceinline__ void node_coord_both(const NodeCtx &N, const NextLevel &X, int im,
                                                double hgt, bool &edge, double2 &p, double2 &q) {
    const double H = (hgt - N.hnorm[im][0]) * N.hnorm[im][1];
    double v[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const double *a = N.horner[im][j];
        v[j] = fma(fma(fma(a[3], H, a[2]), H, a[1]), H, a[0]);
    }
    const double *g = N.geo[im];
    double y = g[0] + ((v[0] * fast_rcp(v[1], edge)) * g[4] + g[2]);
    double x = g[1] + ((v[2] * fast_rcp(v[3], edge)) * g[5] + g[3]);
    const double ymax = g[2] + g[4] * 1.2, xmax = g[3] + g[5] * 1.2;
    if (fabs(y) < kEdge || fabs(y - ymax) < kEdge || fabs(x) < kEdge || fabs(x - xmax) < kEdge)
        edge = true;
    y = y < 0 ? 0 : (y > ymax ? ymax : y);
    x = x < 0 ? 0 : (x > xmax ? xmax : x);
    p = make_double2(x * N.inv_s - g[6], y * N.inv_s - g[7]);
    q = make_double2(x * X.inv_s - X.start[im][0], y * X.inv_s - X.start[im][1]);
    const double fx = p.x - floor(p.x), fy = p.y - floor(p.y);
    const double gx = q.x - floor(q.x), gy = q.y - floor(q.y);
    if (fx < kEdge || fx > 1.0 - kEdge || fy < kEdge || fy > 1.0 - kEdge || gx < kEdge ||
        gx > 1.0 - kEdge || gy < kEdge || gy > 1.0 - kEdge)
        edge = true;
}

// The same by the reference's RPC order.
__device__ __noinline__ void slot_coords_both_exact(const NodeCtx &N, int im, double hgt, double2 &p,
                                                    double2 &q) {
    const DevLevel &P = *N.P;
    const DevImage &I = P.im[im == 0 ? P.ref : 1];
    const double2 c =
        rpc_project(I.rpc, I.adj, P.grid_wgs[2 * N.pt], P.grid_wgs[2 * N.pt + 1], hgt);
    p = to_pyramid(c, I.sx, I.sy, P.L);
    q = to_pyramid(c, I.sxn, I.syn, P.L - 1);
}

// FP32 multi-window NCC of the group's slots at one level: the boxes covering
// the 32 footprints are staged by the warp and every slot whose footprints
// lie inside both images and hold no zero texel is evaluated.  `ok`: the slot
// takes part; returns whether its INCC was formed (else it needs FP64).
__device__ __forceinline__ bool combined_level(const uint16_t *const img[2],
                                               const uint16_t *const mag[2], const uint32_t w[2],
                                               const uint32_t h[2], bool vec, int H,
                                               unsigned char *smem, uint32_t box_off, int quads,
                                               bool ok, double2 rp, double2 tp, float cf, float sf,
                                               float &incc, bool &unsure, int lane) {
    const int R = H + 2;
    const int rix = (int)floor(rp.x), riy = (int)floor(rp.y);
    const int tix = (int)floor(tp.x), tiy = (int)floor(tp.y);
    const bool inside = ok && rix - H >= 0 && riy - H >= 0 && rix + H + 2 < (int)w[0] &&
                        riy + H + 2 < (int)h[0] && tix - R >= 0 && tiy - R >= 0 &&
                        tix + R + 2 < (int)w[1] && tiy + R + 2 < (int)h[1];
    const int rx0 = __reduce_min_sync(0xffffffffu, inside ? rix - H : INT_MAX);
    const int ry0 = __reduce_min_sync(0xffffffffu, inside ? riy - H : INT_MAX);
    const int rx1 = __reduce_max_sync(0xffffffffu, inside ? rix + H + 1 : INT_MIN);
    const int ry1 = __reduce_max_sync(0xffffffffu, inside ? riy + H + 1 : INT_MIN);
    const int tx0 = __reduce_min_sync(0xffffffffu, inside ? tix - R : INT_MAX);
    const int ty0 = __reduce_min_sync(0xffffffffu, inside ? tiy - R : INT_MAX);
    const int tx1 = __reduce_max_sync(0xffffffffu, inside ? tix + R + 1 : INT_MIN);
    const int ty1 = __reduce_max_sync(0xffffffffu, inside ? tiy + R + 1 : INT_MIN);
    if (rx0 == INT_MAX) return false;
    const int rw = rx1 - rx0 + 1, rh = ry1 - ry0 + 1, tw = tx1 - tx0 + 1, th = ty1 - ty0 + 1;
    const int rs = rw | 1, ts = tw | 1;
    if (rs * rh + ts * th > quads) return false;
    float4 *boxes = reinterpret_cast<float4 *>(smem + box_off);
    float4 *tbox = boxes + rs * rh;
    // box shifts: the centre texels
    const int64_t rc = (int64_t)(ry0 + rh / 2) * w[0] + (rx0 + rw / 2);
    const int64_t tc = (int64_t)(ty0 + th / 2) * w[1] + (tx0 + tw / 2);
    const float sI = (float)__ldg(img[0] + rc), sM = (float)__ldg(mag[0] + rc);
    const float tI = (float)__ldg(img[1] + tc), tM = (float)__ldg(mag[1] + tc);
    __syncwarp();   // the boxes' previous readers
    bool z;
    if (vec) {
        z = stage_box_vec<false>(boxes, rs, img[0], mag[0], w[0], rx0, ry0, rw, rh, sI, sM, lane);
        z |= stage_box_vec<true>(tbox, ts, img[1], mag[1], w[1], tx0, ty0, tw, th, tI, tM, lane);
    } else {
        z = stage_box_strided<false>(boxes, rs, img[0], mag[0], w[0], rx0, ry0, rw, rh, sI, sM,
                                     lane);
        z |= stage_box_strided<true>(tbox, ts, img[1], mag[1], w[1], tx0, ty0, tw, th, tI, tM,
                                     lane);
    }
    __syncwarp();
    if (z || !inside) return false;
    const float4 *qr = boxes + (riy - H - ry0) * rs + (rix - H - rx0);
    const uint32_t tcen =
        box_off + (uint32_t)(rs * rh + (tiy - ty0) * ts + (tix - tx0)) * 16u;
    window_any<true>(H, qr, rs, (float)(rp.x - (double)rix), (float)(rp.y - (double)riy),
               tgt_box(smem, tcen, (uint32_t)ts * 16u), (float)(tp.x - (double)tix),
               (float)(tp.y - (double)tiy), cf, sf, incc, unsure);
    return true;
}

__host__ __device__ constexpr size_t combined_boxes_offset() {
    return (sizeof(CombinedShared) * kWinWarps + 15) & ~(size_t)15;
}

// The nodes of combined levels (setsm_code.cpp:6378-6464: the windows at the
// matched and at the next finer level, the rotation of their averaged
// orientation difference, both levels' bounds), a warp per node and 32 slots
// at a time like window_kernel, but staged by loads without a pipeline: the
// two levels' windows follow each other through the same boxes, which leaves
// room for three blocks per SM.  Decisions inside the error band go to the
// exact pass.  205 x 199 grid at level 2 (46 slots a node, 7x7 windows):
// 1.0 ms, and the whole call 7.5 to 2.1 ms (all FP64 before: 6.7 ms of it).
__global__ void __launch_bounds__(kWinWarps * 32, VLL_WIN_MINB) combined_kernel(
    const LevelSet LS, const int32_t *__restrict__ node_k, const double *__restrict__ gsum,
    const double *__restrict__ gcnt, float *__restrict__ pend_vals, int64_t pend_cap,
    int64_t *__restrict__ pend_node, int64_t *__restrict__ pend_off,
    float *__restrict__ warp_vals, int64_t *__restrict__ fix_list, int64_t fix_cap,
    unsigned long long *__restrict__ counters, unsigned long long *__restrict__ ctl, int quads) {
    extern __shared__ __align__(128) unsigned char smem_raw[];
    const int lane = threadIdx.x & 31;
    const int warp = threadIdx.x >> 5;
    CombinedShared &W = reinterpret_cast<CombinedShared *>(smem_raw)[warp];
    const uint32_t box_off = (uint32_t)(combined_boxes_offset() + (size_t)warp * quads * 16);
    float *wv = warp_vals + ((size_t)blockIdx.x * kWinWarps + warp) * kSlotCap;
    NodeCtx &N = W.node;
    NextLevel &X = W.next;
    int x_level = -1;
    unsigned long long evals = 0;
    PeakScan scan;
    for (;;) {
        unsigned long long b = 0;
        if (lane == 0) b = atomicAdd(&ctl[6], 1ull);
        const int64_t gn = (int64_t)__shfl_sync(0xffffffffu, b, 0);
        if (gn >= LS.total) break;
        const int K = node_k[gn];
        if (K == 0) continue;
        const int lvl = level_of(LS, gn);
        const DevLevel &P = LS.lv[lvl];
        if (!P.combined_incc) continue;
        if (K > kSlotCap) {
            if (lane == 0) {
                const unsigned long long idx = atomicAdd(&ctl[2], 1ull);
                pend_node[idx] = gn;
                pend_off[idx] = -2;
            }
            continue;
        }
        __syncwarp();
        if (lvl != x_level) {
            if (lane < 2) {
                const DevImage &I = P.im[lane == 0 ? P.ref : 1];
                X.img[lane] = I.img_n;
                X.mag[lane] = I.mag_n;
                X.ori[lane] = I.ori_n;
                X.start[lane][0] = I.sxn;
                X.start[lane][1] = I.syn;
                X.w[lane] = I.wn;
                X.h[lane] = I.hn;
                if (lane == 0) X.inv_s = 1.0 / (double)(1 << (P.L - 1));
            }
            x_level = lvl;
        }
        node_setup(N, LS, lvl, gn, K, gsum, gcnt, nullptr, lane);
        const bool vec_n = X.w[0] % 8 == 0 && X.w[1] % 8 == 0 &&
                           ((reinterpret_cast<uintptr_t>(X.img[0]) |
                             reinterpret_cast<uintptr_t>(X.mag[0]) |
                             reinterpret_cast<uintptr_t>(X.img[1]) |
                             reinterpret_cast<uintptr_t>(X.mag[1])) & 15) == 0;
        for (int k0 = 0; k0 < K; k0 += 32) {
            const int k = k0 + lane;
            int status = 0;
            double2 rp = make_double2(0, 0), tp = rp, rq = rp, tq = rp;
            float cf = 1.f, sf = 0.f;
            if (k < K) {
                const float hgt = (float)__dadd_rn(N.hbase, __dmul_rn((double)k, N.hstep));
                if (hgt >= (float)N.start_H && hgt <= (float)N.end_H) {
                    bool edge = false;
                    node_coord_both(N, X, 0, (double)hgt, edge, rp, rq);
                    node_coord_both(N, X, 1, (double)hgt, edge, tp, tq);
                    if (edge) {
                        slot_coords_both_exact(N, 0, (double)hgt, rp, rq);
                        slot_coords_both_exact(N, 1, (double)hgt, tp, tq);
                    }
                    if (in_image(rp, N.w[0], N.h[0]) && in_image(tp, N.w[1], N.h[1]) &&
                        in_image(rq, X.w[0], X.h[0]) && in_image(tq, X.w[1], X.h[1])) {
                        // twice the averaged orientation difference
                        const int od = (int)N.ori[0][(int64_t)(int)rp.y * N.w[0] + (int)rp.x] -
                                       (int)N.ori[1][(int64_t)(int)tp.y * N.w[1] + (int)tp.x] +
                                       (int)X.ori[0][(int64_t)(int)rq.y * X.w[0] + (int)rq.x] -
                                       (int)X.ori[1][(int64_t)(int)tq.y * X.w[1] + (int)tq.x];
                        status = 2;
                        if (N.flags & kNfOri) {
                            const double a = __dmul_rn((double)od / 2.0, N.bin_angle);
                            if (!(a < 90 && a > -90)) status = 1;
                        }
                        cf = (float)P.rot_cos[od + kRotOffset];
                        sf = (float)P.rot_sin[od + kRotOffset];
                    }
                }
            }
            // the two levels' windows, coarse first
            float incc[2] = {-2.f, -2.f};
            bool unsure = false, formed = true;
#pragma unroll 1
            for (int lev = 0; lev < 2; ++lev) {
                float v = -2.f;
                const bool f = combined_level(lev ? X.img : N.img, lev ? X.mag : N.mag,
                                              lev ? X.w : N.w, lev ? X.h : N.h,
                                              lev ? vec_n : (N.flags & kNfVec) != 0, N.H, smem_raw,
                                              box_off, quads, status == 2, lev ? rq : rp,
                                              lev ? tq : tp, cf, sf, v, unsure, lane);
                formed = formed && f;
                if (lev)
                    incc[1] = v;
                else
                    incc[0] = v;
            }
            float rho_v = kNotEvaluated, incc_v = 0.f;
            bool all_pos = false, deferred = false;
            if (status == 1) {
                rho_v = kRejected;
            } else if (status == 2) {
                if (formed) {
                    // the mean of the levels that have one
                    const int n = (incc[0] != -2.f) + (incc[1] != -2.f);
                    const double sum = (incc[0] != -2.f ? (double)incc[0] : 0.0) +
                                       (incc[1] != -2.f ? (double)incc[1] : 0.0);
                    const double incc_d = n > 0 ? sum / (double)n : -1.0;
                    double rho_d = incc_d;
                    if (N.flags & kNfGncc)
                        rho_d = n > 0 ? incc_d * N.alpha + N.gterm : __ddiv_rn(0.0, 0.0);
                    rho_v = (float)rho_d;
                    incc_v = unsure ? __int_as_float(0x7fc00000) : (float)incc_d;
                    all_pos = true;
                } else {
                    rho_v = 0.f;
                    incc_v = __int_as_float(0x7fc00000);
                    deferred = true;
                }
                evals++;
            }
            // (the debug values of undecided slots are the exact pass's)
            scan_group(N, scan, K, N.flags, k, k0, status, rho_v, incc_v, all_pos,
                       deferred || unsure, wv, fix_list, fix_cap, ctl, lane);
        }
        finish_node(N, scan, K, N.flags, wv, pend_vals, pend_cap, pend_node, pend_off, ctl, lane);
    }
    for (int o = 16; o; o >>= 1) evals += __shfl_down_sync(0xffffffffu, evals, o);
    if (lane == 0 && evals) atomicAdd(&counters[1], evals);
}

cudaError_t launch_plain_counts(const LevelSet &LS, const int32_t *node_k, int32_t *plain_k,
                                cudaStream_t s) {
    const int64_t blocks = std::min<int64_t>(std::max<int64_t>((LS.total + 255) / 256, 1), 148 * 16);
    plain_counts_kernel<<<(unsigned)blocks, 256, 0, s>>>(LS, node_k, plain_k);
    return cudaGetLastError();
}

cudaError_t launch_combined(const LevelSet &LS, const int32_t *node_k, const double *gsum,
                            const double *gcnt, float *pend_vals, int64_t pend_cap,
                            int64_t *pend_node, int64_t *pend_off, int64_t *fix_list,
                            int64_t fix_cap, unsigned long long *counters,
                            unsigned long long *ctl, int quads, int max_blocks_per_sm,
                            cudaStream_t s) {
    // at most ~200 KB for the block: larger boxes go to the exact pass
    const size_t most = (200 * 1024 - combined_boxes_offset()) / kWinWarps / sizeof(float4);
    quads = (int)std::min<size_t>((size_t)quads, most);
    const size_t smem = combined_boxes_offset() + (size_t)kWinWarps * quads * sizeof(float4);
    cudaError_t e = ensure_smem_limit((const void *)combined_kernel, smem);
    if (e != cudaSuccess) return e;
    int dev = 0, sms = 148, per_sm = 1;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, combined_kernel, kWinWarps * 32, smem);
    // (the warps' slot scratch is sized for the window kernel's grid)
    per_sm = std::max(1, std::min(per_sm, max_blocks_per_sm));
    combined_kernel<<<sms * per_sm, kWinWarps * 32, smem, s>>>(
        LS, node_k, gsum, gcnt, pend_vals, pend_cap, pend_node, pend_off, pend_vals + pend_cap,
        fix_list, fix_cap, counters, ctl, quads);
    return cudaGetLastError();
}

}  // namespace vll
