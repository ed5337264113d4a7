// vll_tin.cu -- TINCreate_list (SubFunctions.cpp:2768-2846) on the GPU: the
// Delaunay triangulation of the matched points snapped to the level's grid,
// returned as the reference's ordered list of vertex-index triples.
//
// The reference triangulates with an alternating-cut divide and conquer
// (grid_triangulation.cpp, after Guibas-Stolfi and Wu et al.): a node sorts
// its points by (col, row) -- or by (row, -col) one level down --, splits them
// at the median, triangulates both halves and zips them together from the
// lower (or right) common tangent, preferring the left candidate on
// co-circular ties.  On an integer grid co-circular points are common, so
// the triangles depend on that exact order of decisions, and the list's
// order on where each half-edge lives in memory (the edge allocator's stack,
// split and merged with the recursion; a point's triangles are listed from
// the edge of it stored last).  This file replays the same recursion: both
// sorted orders are made once and split down the tree by stable partitions
// (no node is sorted again), every subtree of fewer than 100 points is
// triangulated by one thread, and then, deepest first, every node of a depth
// merges its halves in one thread, each on its own slice of the shared
// half-edge pool and allocator stack.  Then one thread per point walks its
// triangles in the reference's order.  The tree's shape follows from the
// number of points alone, so the host only counts depths.  Integer predicates
// are 64-bit with the reference's wrap-around arithmetic.
//
// What bounds it: the merges near the root, one thread each, a chain of some
// hundred steps per cut (vll_tin_core.cuh).  Threads that walk alone have a
// warp to themselves, so the warps' chains neither diverge nor share an L1
// slice with 31 others.  224 k points of a 700 x 640 grid: 5.0 ms, of which
// the merges are 4.1, the root's alone 1.4 (42.4 ms with a record per field,
// 32 nodes to a warp, a segmented sort per depth and the tree on the host).
#include <algorithm>
#include <cstdio>
#include <string>
#include <vector>
#include <cub/block/block_scan.cuh>
#include <cub/device/device_radix_sort.cuh>
#include <cub/device/device_scan.cuh>

#include "vll_internal.h"
#include "vll_tin_core.cuh"

namespace vll {
namespace {

using namespace tin;

// THREADED_CUTOFF (basic_topology_types.hpp:15): nodes below it recurse
// serially on one edge list.
constexpr int kThreadedCutoff = 100;
// Nodes of at most this many points are partitioned down to the leaves by one
// block in shared memory; larger ones a depth at a time over all points.
constexpr int kBlockPoints = 1024;
// Up to this many points the three orders are made by counting: three library
// sorts of so few keys are some forty dependent passes.  Calls of 48, 1000, 4000
// and 8192 points: 306, 635, 1186 and 1443 us sorted, 265, 593, 939 and 1275
// counted; the counting grows with the square (12000: 1681 and 1598, 16000: 1719
// and 1810), so the line lies well below the crossing.
constexpr int kRankPoints = 8192;
constexpr int kRankLanes = 8, kRankTile = 1024;

// ---------------------------------------------------------------------------
// points and their two orders
// ---------------------------------------------------------------------------
// Grid coordinates of the points (SubFunctions.cpp:2793-2798: 0.5 plus the
// offset in grid cells, truncated to int), their grid index and the keys of
// the orders (col, row) and (row, -col), non-negative in biased 32-bit halves.
__global__ void tin_coords_kernel(const vll_point3 *__restrict__ pts, int n, double minx,
                                  double miny, double res, int width, int2 *__restrict__ xy,
                                  unsigned long long *__restrict__ gkey,
                                  unsigned long long *__restrict__ kx,
                                  unsigned long long *__restrict__ ky, int *__restrict__ ids) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const int c = (int)(0.5 + __ddiv_rn(__dadd_rn(pts[i].x, -minx), res));
        const int r = (int)(0.5 + __ddiv_rn(__dadd_rn(pts[i].y, -miny), res));
        xy[i] = make_int2(c, r);
        // grid index row * width + col, biased so that any int pair sorts
        gkey[i] = (unsigned long long)((long long)r * width + c + (1ll << 62));
        const unsigned int br = (unsigned int)r ^ 0x80000000u, bc = (unsigned int)c ^ 0x80000000u;
        kx[i] = ((unsigned long long)bc << 32) | br;
        ky[i] = ((unsigned long long)br << 32) | (0xFFFFFFFFu - bc);
        ids[i] = i;
    }
}

// The three orders of a short list at once (blockIdx.y: the grid order with its
// sorted keys, then (col, row) and (row, -col)): eight lanes count the keys
// before a point's own, equal keys by index as a stable sort takes them.
__global__ void __launch_bounds__(256) tin_rank_kernel(const unsigned long long *__restrict__ gkey,
                                                       const unsigned long long *__restrict__ kx,
                                                       const unsigned long long *__restrict__ ky,
                                                       int n,
                                                       unsigned long long *__restrict__ gkey_sorted,
                                                       int *__restrict__ ids_sorted,
                                                       int *__restrict__ px, int *__restrict__ py) {
    __shared__ unsigned long long tile[kRankTile];
    const unsigned long long *key = blockIdx.y == 0 ? gkey : blockIdx.y == 1 ? kx : ky;
    int *out = blockIdx.y == 0 ? ids_sorted : blockIdx.y == 1 ? px : py;
    const int sub = threadIdx.x & (kRankLanes - 1);
    const int i = blockIdx.x * (256 / kRankLanes) + threadIdx.x / kRankLanes;
    const unsigned long long mine = i < n ? key[i] : 0;
    int rank = 0;
    for (int j0 = 0; j0 < n; j0 += kRankTile) {
        const int m = min(kRankTile, n - j0);
        __syncthreads();
        for (int j = threadIdx.x; j < m; j += 256) tile[j] = key[j0 + j];
        __syncthreads();
#pragma unroll 4
        for (int j = sub; j < m; j += kRankLanes) {
            const unsigned long long k = tile[j];
            rank += k < mine || (k == mine && j0 + j < i);
        }
    }
#pragma unroll
    for (int o = 1; o < kRankLanes; o <<= 1) rank += __shfl_xor_sync(0xffffffffu, rank, o);
    if (i < n && sub == 0) {
        out[rank] = i;
        if (blockIdx.y == 0) gkey_sorted[rank] = mine;
    }
}

// Flags a grid cell holding two points (the triangulation needs distinct points).
__global__ void tin_dup_kernel(const unsigned long long *__restrict__ sorted, int n,
                               unsigned int *__restrict__ err) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x + 1; i < n; i += gridDim.x * blockDim.x)
        if (sorted[i] == sorted[i - 1]) atomicExch(err + 1, 1u);
}

// The depth-d node holding position i.
__device__ __forceinline__ void node_at(int n, int d, int i, int &lo, int &cnt) {
    lo = 0;
    cnt = n;
    for (int b = 0; b < d; ++b) {
        const int mid = cnt / 2;
        if (i < lo + mid) {
            cnt = mid;
        } else {
            lo += mid;
            cnt -= mid;
        }
    }
}

// One depth: `a` is the order the depth's nodes are cut in.  Which half each
// point falls in ...
__global__ void tin_side_kernel(const int *__restrict__ a, int n, int d,
                                unsigned char *__restrict__ left) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        int lo, cnt;
        node_at(n, d, i, lo, cnt);
        left[a[i]] = i < lo + cnt / 2;
    }
}
__global__ void tin_flag_kernel(const int *__restrict__ b, int n,
                                const unsigned char *__restrict__ left, int *__restrict__ flag) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
        flag[i] = left[b[i]];
}
// ... and the other order `b` stably split by it (sum: exclusive sums of the
// left flags along b).
__global__ void tin_split_kernel(const int *__restrict__ b, int n, int d,
                                 const int *__restrict__ flag, const int *__restrict__ sum,
                                 int *__restrict__ out) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        int lo, cnt;
        node_at(n, d, i, lo, cnt);
        const int s = sum[i] - sum[lo];
        out[flag[i] ? lo + s : lo + cnt / 2 + (i - lo - s)] = b[i];
    }
}

// The same for all remaining depths of one node per block (at most
// kBlockPoints points): px, py its points in both orders.  Writes the points'
// coordinates in the order their leaves take them: the order their parent cut.
__global__ void __launch_bounds__(256) tin_leaves_kernel(const int *__restrict__ px,
                                                         const int *__restrict__ py, int n, int d0,
                                                         int *__restrict__ inv,
                                                         const int2 *__restrict__ xy,
                                                         int2 *__restrict__ out) {
    constexpr int kItems = kBlockPoints / 256;
    typedef cub::BlockScan<int, 256> Scan;
    __shared__ typename Scan::TempStorage scan_tmp;
    __shared__ int gid[kBlockPoints];
    __shared__ unsigned short order[2][kBlockPoints], next[kBlockPoints], leaf[kBlockPoints];
    __shared__ unsigned short sum[kBlockPoints];
    __shared__ unsigned char left[kBlockPoints];
    int lo0, cnt0;
    node_range(n, d0, blockIdx.x, lo0, cnt0);
    // local ids: the position in the (col, row) order
    for (int i = threadIdx.x; i < cnt0; i += 256) {
        gid[i] = px[lo0 + i];
        inv[gid[i]] = i;
        order[0][i] = leaf[i] = (unsigned short)i;
    }
    __syncthreads();
    for (int i = threadIdx.x; i < cnt0; i += 256) order[1][i] = (unsigned short)inv[py[lo0 + i]];
    __syncthreads();
    int widest = cnt0;
    for (int d = d0; widest >= 4; ++d, widest = (widest + 1) / 2) {
        unsigned short *a = order[d & 1], *b = order[(d & 1) ^ 1];
        for (int i = threadIdx.x; i < cnt0; i += 256) {
            int lo = 0, cnt = cnt0;
            for (int k = d0; k < d && cnt >= 4; ++k) {
                const int mid = cnt / 2;
                if (i < lo + mid) {
                    cnt = mid;
                } else {
                    lo += mid;
                    cnt -= mid;
                }
            }
            if (cnt < 4) continue;   // a leaf of an earlier depth
            leaf[i] = a[i];
            left[a[i]] = i < lo + cnt / 2;
        }
        __syncthreads();
        int f[kItems], s[kItems];
#pragma unroll
        for (int k = 0; k < kItems; ++k) {
            const int i = threadIdx.x * kItems + k;
            f[k] = i < cnt0 ? left[b[i]] : 0;
        }
        Scan(scan_tmp).ExclusiveSum(f, s);
#pragma unroll
        for (int k = 0; k < kItems; ++k) sum[threadIdx.x * kItems + k] = (unsigned short)s[k];
        __syncthreads();
        for (int i = threadIdx.x; i < cnt0; i += 256) {
            int lo = 0, cnt = cnt0;
            for (int k = d0; k < d && cnt >= 4; ++k) {
                const int mid = cnt / 2;
                if (i < lo + mid) {
                    cnt = mid;
                } else {
                    lo += mid;
                    cnt -= mid;
                }
            }
            int to = i;
            if (cnt >= 4) {
                const int before = sum[i] - sum[lo];
                to = left[b[i]] ? lo + before : lo + cnt / 2 + (i - lo - before);
            }
            next[to] = b[i];
        }
        __syncthreads();
        for (int i = threadIdx.x; i < cnt0; i += 256) b[i] = next[i];
        __syncthreads();
    }
    for (int i = threadIdx.x; i < cnt0; i += 256) out[lo0 + i] = xy[gid[leaf[i]]];
}

__global__ void tin_iota_kernel(int *__restrict__ a, long long n) {
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
         i += (long long)gridDim.x * blockDim.x)
        a[i] = (int)i;
}

// ---------------------------------------------------------------------------
// triangulation
// ---------------------------------------------------------------------------
__device__ __forceinline__ TinNode *node_of(TinNode *nodes, int d, unsigned j) {
    return nodes + ((1ll << d) - 1 + j);
}

// A warp per node of depth d that is the root of a subtree of fewer than 100
// points (and not inside one): lane 0 triangulates it.
__global__ void __launch_bounds__(32) tin_serial_kernel(TinGraph G, TinNode *nodes,
                                                        const int2 *__restrict__ pts, int n, int d,
                                                        long long bound) {
    if (threadIdx.x != 0 || G.err[1]) return;
    int lo, cnt;
    if (d > 0) {
        node_range(n, d - 1, blockIdx.x >> 1, lo, cnt);
        if (cnt < kThreadedCutoff) return;
    }
    node_range(n, d, blockIdx.x, lo, cnt);
    if (cnt >= kThreadedCutoff) return;
    Alloc a = alloc_at(G, 6 * lo, 6 * cnt);
    TinNode *N = node_of(nodes, d, blockIdx.x);
    N->ex = serial_subtree(G, pts, lo, cnt, (d & 1) == 0, a, bound);
    N->idx = a.idx;
}

// A warp per node of depth d of 100 points or more
// (TriangulateHorizontalThreaded / TriangulateVerticalThreaded): its halves
// drew from split slices of its stack, which are concatenated
// (EdgeList::MergeEdgeLists, edge_list.cpp:96-106: the right (top) child's
// free stack moves down onto the left (bottom) child's; the destination
// precedes the source, so copying 32 entries at a time in increasing order,
// each group read before written, is safe); then lane 0 merges the halves.
__global__ void __launch_bounds__(32) tin_merge_kernel(TinGraph G, TinNode *nodes, int n, int d,
                                                       long long bound) {
    if (G.err[1]) return;
    int lo, cnt;
    node_range(n, d, blockIdx.x, lo, cnt);
    if (cnt < kThreadedCutoff) return;
    const TinNode L = *node_of(nodes, d + 1, 2 * blockIdx.x);
    const TinNode R = *node_of(nodes, d + 1, 2 * blockIdx.x + 1);
    const int lane = threadIdx.x;
    const int src = 6 * (lo + cnt / 2), dst = 6 * lo + L.idx;
    for (int k0 = 0; k0 < R.idx; k0 += 32) {
        const int k = k0 + lane;
        int v = 0;
        if (k < R.idx) v = G.unused[src + k];
        __syncwarp();
        if (k < R.idx) G.unused[dst + k] = v;
        __syncwarp();
    }
    if (lane != 0) return;
    Alloc a = alloc_at(G, 6 * lo, L.idx + R.idx);
    TinNode *N = node_of(nodes, d, blockIdx.x);
    N->ex = merge_halves(G, (d & 1) == 0, L.ex, R.ex, a, bound);
    N->idx = a.idx;
}

// ---------------------------------------------------------------------------
// the triangle list
// ---------------------------------------------------------------------------
// Free edges take dnext -1.
__global__ void tin_free_kernel(TinGraph G, const TinNode *__restrict__ root) {
    const int n = root->idx;
    if (G.err[1]) return;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
        G.edge[G.unused[i]].x = -1;
}

// EdgeList::SetGrid (basic_topology_types.hpp:157-202): a point keeps the
// in-use edge out of it that is last in the pool.  The edges' points, as
// positions in grid order, are found by their grid index.
__global__ void tin_store_kernel(TinGraph G, const unsigned long long *__restrict__ gkey, int n,
                                 int width, long long n_edges, int *__restrict__ pos,
                                 int *__restrict__ stored) {
    if (G.err[1]) return;
    for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < n_edges;
         t += (long long)gridDim.x * blockDim.x) {
        const int4 E = G.edge[t];
        if (E.x < 0) continue;
        const unsigned long long key =
            (unsigned long long)((long long)E.w * width + E.z + (1ll << 62));
        int lo = 0, hi = n - 1;
        while (lo < hi) {
            const int mid = (lo + hi) >> 1;
            if (__ldg(gkey + mid) < key)
                lo = mid + 1;
            else
                hi = mid;
        }
        pos[t] = lo;
        atomicMax(stored + lo, (int)t);
    }
}

// Grid::GetAllTris (grid.cpp:16-51): the points in grid order, each listing
// the triangles around it (AdjTriIter, counter-clockwise from its stored
// edge) of which it is the (col, row)-smallest vertex.  Pass 0 counts, pass 1
// writes the vertices' input indices at the exclusive prefix `off` (off[n]:
// the total; nothing is written when it exceeds cap or the input was refused).
template <bool WRITE>
__global__ void tin_tris_kernel(TinGraph G, const int *__restrict__ order, int n,
                                const int *__restrict__ pos, const int *__restrict__ stored,
                                long long *__restrict__ cnt, const long long *__restrict__ off,
                                vll_tri *__restrict__ out, long long cap, long long bound) {
    if (G.err[1] || (WRITE && (G.err[0] || off[n] > cap))) return;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        long long c = 0;
        long long o = WRITE ? off[i] : 0;
        point_tris(G, stored[i], bound, [&](int e0, int e1, int e2) {
            if (WRITE && o < cap)
                out[o] = vll_tri{(uint32_t)order[pos[e0]], (uint32_t)order[pos[e1]],
                                 (uint32_t)order[pos[e2]]};
            ++o;
            ++c;
        });
        if (!WRITE) cnt[i] = c;
    }
}

inline int grid1(long long n, int threads, int cap = 148 * 32) {
    const long long b = (n + threads - 1) / threads;
    return (int)std::max<long long>(1, std::min<long long>(b, cap));
}

}  // namespace

// ---------------------------------------------------------------------------
// host driver
// ---------------------------------------------------------------------------
void tin_release(TinWork &w) {
    for (auto &b : w.bufs)
        if (b.first) cudaFree(b.first);
    w.bufs.clear();
}

namespace {

// A device array of the work area, grown on demand (kept between calls).
template <class T>
cudaError_t tin_buf(TinWork &w, size_t slot, size_t count, T **out) {
    if (w.bufs.size() <= slot) w.bufs.resize(slot + 1, {nullptr, 0});
    auto &b = w.bufs[slot];
    const size_t bytes = std::max<size_t>(count, 1) * sizeof(T);
    if (b.second < bytes) {
        if (b.first) cudaFree(b.first);
        b.first = nullptr;
        b.second = 0;
        const cudaError_t e = cudaMalloc(&b.first, bytes);
        if (e != cudaSuccess) return e;
        b.second = bytes;
    }
    *out = (T *)b.first;
    return cudaSuccess;
}

}  // namespace

int run_tin_create(TinWork &w, const vll_point3 *d_pts, int64_t n64, const double min_max[4],
                   double resolution, vll_tri *d_tris, int64_t capacity, int64_t *count,
                   cudaStream_t s, std::string *err) {
#define TIN_CUDA(call)                                              \
    do {                                                            \
        const cudaError_t e__ = (call);                             \
        if (e__ != cudaSuccess) {                                   \
            *err = std::string(#call) + ": " + cudaGetErrorString(e__); \
            return VLL_ERR_CUDA;                                    \
        }                                                           \
    } while (0)
    *count = 0;
    if (n64 <= 2) return VLL_OK;   // TINCreate_list: no triangulation below 3 points
    if (n64 > (1 << 26)) {
        *err = "more points than the triangulation's 32-bit edge indices allow";
        return VLL_ERR_CAPACITY;
    }
    const int n = (int)n64;
    const int width = (int)(1 + (min_max[2] - min_max[0]) / resolution);
    const int height = (int)(1 + (min_max[3] - min_max[1]) / resolution);
    if (width > 32767 || height > 32767) {
        char m[160];
        snprintf(m, sizeof m, "grid of %d x %d cells exceeds the triangulation's 16-bit limit",
                 width, height);
        *err = m;
        return VLL_ERR_INVALID;
    }
    // ---- the recursion tree's depths (its nodes of a depth differ by one point) ----
    auto smallest = [n](int d) { return n >> d; };
    auto largest = [n](int d) { return (int)(((long long)n + (1ll << d) - 1) >> d); };
    int d_block = 0;    // first depth whose nodes a block can partition
    while (largest(d_block) > kBlockPoints) ++d_block;
    int d_serial = 0;   // first depth with a node of fewer than 100 points
    while (smallest(d_serial) >= kThreadedCutoff) ++d_serial;
    // at that depth the larger nodes may still be of 100 points: their halves
    // are then the subtrees
    const bool mixed = largest(d_serial) >= kThreadedCutoff;
    // ---- device buffers ----
    const long long n_edges = 6ll * n;
    int *ids, *ids_sorted, *px, *py, *p2, *flag, *sum, *inv, *unused, *stored, *pos;
    unsigned long long *gkey, *gkey_sorted, *kx, *ky, *ktmp;
    unsigned int *flags;
    unsigned char *left;
    long long *tcnt, *toff;
    int2 *xy, *leaf_xy;
    int4 *edge;
    TinNode *nodes;
    size_t slot = 0;
    TIN_CUDA(tin_buf(w, slot++, n, &ids));
    TIN_CUDA(tin_buf(w, slot++, n, &ids_sorted));
    TIN_CUDA(tin_buf(w, slot++, n, &px));
    TIN_CUDA(tin_buf(w, slot++, n, &py));
    TIN_CUDA(tin_buf(w, slot++, n, &p2));
    TIN_CUDA(tin_buf(w, slot++, n, &flag));
    TIN_CUDA(tin_buf(w, slot++, n, &sum));
    TIN_CUDA(tin_buf(w, slot++, n, &inv));
    TIN_CUDA(tin_buf(w, slot++, (size_t)n_edges, &unused));
    TIN_CUDA(tin_buf(w, slot++, n, &stored));
    TIN_CUDA(tin_buf(w, slot++, (size_t)n_edges, &pos));
    TIN_CUDA(tin_buf(w, slot++, (size_t)n_edges, &edge));
    TIN_CUDA(tin_buf(w, slot++, n, &gkey));
    TIN_CUDA(tin_buf(w, slot++, n, &gkey_sorted));
    TIN_CUDA(tin_buf(w, slot++, n, &kx));
    TIN_CUDA(tin_buf(w, slot++, n, &ky));
    TIN_CUDA(tin_buf(w, slot++, n, &ktmp));
    TIN_CUDA(tin_buf(w, slot++, 4, &flags));
    TIN_CUDA(tin_buf(w, slot++, n, &left));
    TIN_CUDA(tin_buf(w, slot++, (size_t)n + 1, &tcnt));
    TIN_CUDA(tin_buf(w, slot++, (size_t)n + 1, &toff));
    TIN_CUDA(tin_buf(w, slot++, n, &xy));
    TIN_CUDA(tin_buf(w, slot++, n, &leaf_xy));
    TIN_CUDA(tin_buf(w, slot++, (size_t)2 << (d_serial + 1), &nodes));
    // temporary storage of the library sorts and scans
    size_t tmp_bytes = 0, t1 = 0;
    TIN_CUDA(cub::DeviceRadixSort::SortPairs(nullptr, t1, gkey, gkey_sorted, ids, ids_sorted, n, 0,
                                             64, s));
    tmp_bytes = std::max(tmp_bytes, t1);
    TIN_CUDA(cub::DeviceScan::ExclusiveSum(nullptr, t1, tcnt, toff, n + 1, s));
    tmp_bytes = std::max(tmp_bytes, t1);
    TIN_CUDA(cub::DeviceScan::ExclusiveSum(nullptr, t1, flag, sum, n, s));
    tmp_bytes = std::max(tmp_bytes, t1);
    void *tmp;
    TIN_CUDA(tin_buf(w, slot++, tmp_bytes, (unsigned char **)&tmp));

    TIN_CUDA(cudaMemsetAsync(flags, 0, 4 * sizeof(unsigned int), s));
    tin_coords_kernel<<<grid1(n, 256), 256, 0, s>>>(d_pts, n, min_max[0], min_max[1], resolution,
                                                    width, xy, gkey, kx, ky, ids);
    TIN_CUDA(cudaGetLastError());
    // grid order of the points (GetAllTris walks it) and both cutting orders
    if (n <= kRankPoints) {
        const int per_block = 256 / kRankLanes;
        tin_rank_kernel<<<dim3((unsigned)((n + per_block - 1) / per_block), 3), 256, 0, s>>>(
            gkey, kx, ky, n, gkey_sorted, ids_sorted, px, py);
        TIN_CUDA(cudaGetLastError());
    } else {
        t1 = tmp_bytes;
        TIN_CUDA(cub::DeviceRadixSort::SortPairs(tmp, t1, gkey, gkey_sorted, ids, ids_sorted, n, 0,
                                                 64, s));
        t1 = tmp_bytes;
        TIN_CUDA(cub::DeviceRadixSort::SortPairs(tmp, t1, kx, ktmp, ids, px, n, 0, 64, s));
        t1 = tmp_bytes;
        TIN_CUDA(cub::DeviceRadixSort::SortPairs(tmp, t1, ky, ktmp, ids, py, n, 0, 64, s));
    }
    // the distinctness check
    tin_dup_kernel<<<grid1(n, 256), 256, 0, s>>>(gkey_sorted, n, flags);
    TIN_CUDA(cudaGetLastError());
    // ---- the cutting orders, split down the tree ----
    for (int d = 0; d < d_block; ++d) {
        const bool horiz = (d & 1) == 0;
        const int *a = horiz ? px : py;
        int *&b = horiz ? py : px;
        tin_side_kernel<<<grid1(n, 256), 256, 0, s>>>(a, n, d, left);
        tin_flag_kernel<<<grid1(n, 256), 256, 0, s>>>(b, n, left, flag);
        t1 = tmp_bytes;
        TIN_CUDA(cub::DeviceScan::ExclusiveSum(tmp, t1, flag, sum, n, s));
        tin_split_kernel<<<grid1(n, 256), 256, 0, s>>>(b, n, d, flag, sum, p2);
        TIN_CUDA(cudaGetLastError());
        std::swap(b, p2);
    }
    tin_leaves_kernel<<<1u << d_block, 256, 0, s>>>(px, py, n, d_block, inv, xy, leaf_xy);
    TIN_CUDA(cudaGetLastError());
    // ---- triangulation bottom-up ----
    TinGraph G{edge, unused, flags};
    tin_iota_kernel<<<grid1(n_edges, 256), 256, 0, s>>>(unused, n_edges);
    TIN_CUDA(cudaGetLastError());
    const long long bound = 64ll * n + 1024;
    for (int d = d_serial; d <= d_serial + (mixed ? 1 : 0); ++d) {
        tin_serial_kernel<<<1u << d, 32, 0, s>>>(G, nodes, leaf_xy, n, d, bound);
        TIN_CUDA(cudaGetLastError());
    }
    for (int d = d_serial - (mixed ? 0 : 1); d >= 0; --d) {
        tin_merge_kernel<<<1u << d, 32, 0, s>>>(G, nodes, n, d, bound);
        TIN_CUDA(cudaGetLastError());
    }
    // ---- stored edge per point, then the triangle list ----
    TIN_CUDA(cudaMemsetAsync(stored, 0xff, (size_t)n * sizeof(int), s));
    tin_free_kernel<<<grid1(n, 256), 256, 0, s>>>(G, nodes);
    TIN_CUDA(cudaGetLastError());
    tin_store_kernel<<<grid1(n_edges, 256), 256, 0, s>>>(G, gkey_sorted, n, width, n_edges, pos,
                                                         stored);
    TIN_CUDA(cudaGetLastError());
    TIN_CUDA(cudaMemsetAsync(tcnt, 0, ((size_t)n + 1) * sizeof(long long), s));
    tin_tris_kernel<false><<<grid1(n, 128), 128, 0, s>>>(G, ids_sorted, n, pos, stored, tcnt,
                                                         nullptr, nullptr, 0, bound);
    TIN_CUDA(cudaGetLastError());
    t1 = tmp_bytes;
    TIN_CUDA(cub::DeviceScan::ExclusiveSum(tmp, t1, tcnt, toff, n + 1, s));
    tin_tris_kernel<true><<<grid1(n, 128), 128, 0, s>>>(G, ids_sorted, n, pos, stored, nullptr,
                                                        toff, d_tris, capacity, bound);
    TIN_CUDA(cudaGetLastError());
    long long total = 0;
    unsigned int hflags[4];
    TIN_CUDA(cudaMemcpyAsync(&total, toff + n, sizeof(total), cudaMemcpyDeviceToHost, s));
    TIN_CUDA(cudaMemcpyAsync(hflags, flags, sizeof(hflags), cudaMemcpyDeviceToHost, s));
    TIN_CUDA(cudaStreamSynchronize(s));
    if (hflags[1]) {
        *err = "two points fall into one grid cell (the triangulation needs distinct points)";
        return VLL_ERR_INVALID;
    }
    if (hflags[0]) {
        *err = "triangulation walk exceeded its bound (malformed input)";
        return VLL_ERR_INVALID;
    }
    *count = total;
    if (total > capacity) {
        *err = "triangle list longer than the output capacity";
        return VLL_ERR_CAPACITY;
    }
#undef TIN_CUDA
    return VLL_OK;
}

}  // namespace vll
