// vll_tin_core.cuh -- the triangulation steps of TINCreate_list
// (grid_triangulation.cpp): half-edge pool, the reference's edge allocator,
// integer predicates, base cases and the merge of two halves.
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

namespace vll {
namespace tin {

// Half-edges (struct Edge, basic_topology_types.hpp:73-79).  An edge is one
// 16-byte record {dnext, oprev, origin column, origin row}: dnext is the next
// edge out of the destination and oprev the previous edge into the origin,
// both counter-clockwise.  The points are distinct, so coordinates stand for
// the point, and a predicate needs no further access.  Edges are allocated
// and freed in pairs from a stack that starts as 0, 1, 2, ..., so an edge's
// twin is always e ^ 1 and the pair is one 32-byte sector: a merge, which is a
// chain of dependent accesses by one thread, waits once per pair.
struct TinGraph {
    int4 *edge;
    int *unused;            // the allocator's stack of free edges
    unsigned int *err;      // [0] set when a walk exceeds its bound, [1] equal points
};

struct Pt {
    int c, r;
};
__device__ __forceinline__ Pt pt_of(const int4 &e) { return Pt{e.z, e.w}; }
__device__ __forceinline__ bool same(Pt a, Pt b) { return a.c == b.c && a.r == b.r; }

__device__ __forceinline__ int4 rec(const TinGraph &G, int e) { return G.edge[e]; }
__device__ __forceinline__ int dnext(const TinGraph &G, int e) { return G.edge[e].x; }
__device__ __forceinline__ int oprev(const TinGraph &G, int e) { return G.edge[e].y; }
__device__ __forceinline__ Pt orig(const TinGraph &G, int e) { return pt_of(G.edge[e]); }
__device__ __forceinline__ Pt dest(const TinGraph &G, int e) { return pt_of(G.edge[e ^ 1]); }

// A node's hull extremes: left ccw, right cw, bottom ccw, top cw.
struct Ext {
    int l, r, b, t;
};
// A node of 100 points or more, or the root of a smaller subtree.
struct TinNode {
    int idx;   // height of the node's free-edge stack (base 6 lo)
    Ext ex;
};

// Points [lo, lo + cnt) of node j at depth d (its path's bits, the topmost
// first): every node is cut at half its points.
__device__ __forceinline__ void node_range(int n, int d, unsigned j, int &lo, int &cnt) {
    lo = 0;
    cnt = n;
    for (int b = d - 1; b >= 0; --b) {
        const int mid = cnt / 2;
        if ((j >> b) & 1u) {
            lo += mid;
            cnt -= mid;
        } else {
            cnt = mid;
        }
    }
}

__device__ __forceinline__ bool less_xy(Pt a, Pt b) { return a.c < b.c || (a.c == b.c && a.r < b.r); }
__device__ __forceinline__ bool less_yx(Pt a, Pt b) { return a.r < b.r || (a.r == b.r && a.c > b.c); }

// Orientation / InCircle (grid_triangulation.cpp:29-61) in 64-bit integers;
// the products wrap like the reference's (its 128-bit type is an alias of
// int64_t), computed unsigned to keep the wrap-around defined.  Differences
// within +-2^14 -- any grid up to 16384 cells a side -- need no wide
// products: the same values from 32-bit terms and 32 x 32 -> 64 products.
constexpr int kNear = 1 << 14;
__device__ __forceinline__ bool near14(int d) { return (unsigned)(d + kNear) <= 2u * kNear; }

__device__ __forceinline__ long long orient(Pt a, Pt b, Pt c) {
    const int d11 = a.c - c.c, d21 = b.c - c.c, d12 = a.r - c.r, d22 = b.r - c.r;
    if (near14(d11) && near14(d21) && near14(d12) && near14(d22))
        return (long long)(d11 * d22 - d12 * d21);
    typedef unsigned long long U;
    return (long long)((U)(long long)d11 * (U)(long long)d22 -
                       (U)(long long)d12 * (U)(long long)d21);
}

__device__ __forceinline__ long long incircle(Pt a, Pt b, Pt c, Pt d) {
    const int d11 = a.c - d.c, d12 = a.r - d.r, d21 = b.c - d.c, d22 = b.r - d.r;
    const int d31 = c.c - d.c, d32 = c.r - d.r;
    if (near14(d11) && near14(d12) && near14(d21) && near14(d22) && near14(d31) && near14(d32)) {
        const int s1 = d11 * d11 + d12 * d12, s2 = d21 * d21 + d22 * d22, s3 = d31 * d31 + d32 * d32;
        const int bc = d21 * d32 - d31 * d22, ac = d11 * d32 - d31 * d12, ab = d11 * d22 - d21 * d12;
        return (long long)s1 * bc - (long long)s2 * ac + (long long)s3 * ab;
    }
    typedef unsigned long long U;
    const U e11 = (U)(long long)d11, e12 = (U)(long long)d12, e21 = (U)(long long)d21,
            e22 = (U)(long long)d22, e31 = (U)(long long)d31, e32 = (U)(long long)d32;
    const U s1 = e11 * e11 + e12 * e12, s2 = e21 * e21 + e22 * e22, s3 = e31 * e31 + e32 * e32;
    const U bc = e21 * e32 - e31 * e22, ac = e11 * e32 - e31 * e12, ab = e11 * e22 - e21 * e12;
    return (long long)(s1 * bc - s2 * ac + s3 * ab);
}

// The node's slice of the allocator (EdgeList::GetNewEdge / RemoveEdge,
// edge_list.cpp:62-83): a stack of free edge indices at unused[base ...).
// `top` is the stack's top entry, held ahead of its use.
struct Alloc {
    int base, idx, top;
};
__device__ __forceinline__ Alloc alloc_at(const TinGraph &G, int base, int idx) {
    return Alloc{base, idx, idx > 0 ? G.unused[base + idx - 1] : -1};
}
// The next pair of edges: the first popped is the new edge, its twin follows.
// (A stack never runs out on distinct points; should it, the slice's first
// pair is reused and the error flag raised.)
__device__ __forceinline__ int new_pair(const TinGraph &G, Alloc &a) {
    int e = a.top;
    if (a.idx < 2) {
        atomicExch(G.err, 1u);
        a.idx = 2;
        e = a.base;
    }
    a.idx -= 2;
    a.top = a.idx > 0 ? G.unused[a.base + a.idx - 1] : -1;
    return e;
}
__device__ __forceinline__ void free_pair(const TinGraph &G, Alloc &a, int e) {
    G.unused[a.base + a.idx] = e;
    G.unused[a.base + a.idx + 1] = e ^ 1;
    a.idx += 2;
    a.top = e ^ 1;
}

// AddEdgeAndTwin, RemoveEdgeAndTwin, Bridge (grid_triangulation.cpp:95-177).
__device__ __forceinline__ int add_edge_twin(const TinGraph &G, Alloc &a, Pt o, Pt d) {
    const int e = new_pair(G, a), et = e ^ 1;
    G.edge[e] = make_int4(et, et, o.c, o.r);
    G.edge[et] = make_int4(e, e, d.c, d.r);
    return e;
}

__device__ __forceinline__ void remove_edge_twin(const TinGraph &G, Alloc &a, int e) {
    const int4 E = rec(G, e), T = rec(G, e ^ 1);
    G.edge[E.y].x = T.x;
    G.edge[E.x].y = T.y;
    G.edge[T.y].x = E.x;
    G.edge[T.x].y = E.y;
    free_pair(G, a, e);
}

// Weld (grid_triangulation.cpp:127-140) of edge `in` before edge `out`.
__device__ __forceinline__ void weld(const TinGraph &G, int in, int out) {
    const int prev = oprev(G, out);
    G.edge[out].y = in;
    G.edge[in].x = out;
    G.edge[in ^ 1].y = prev;
    G.edge[prev].x = in ^ 1;
}

__device__ __forceinline__ int bridge(const TinGraph &G, Alloc &a, int start, int end) {
    const int e = add_edge_twin(G, a, dest(G, start), orig(G, end));
    weld(G, e ^ 1, dnext(G, start));
    weld(G, e, end);
    return e;
}

// Walks in this file stop after this many steps (a well-formed structure
// never needs that many) and raise the error flag.
__device__ __forceinline__ bool step_ok(const TinGraph &G, long long &steps, long long bound) {
    if (++steps <= bound) return true;
    atomicExch(G.err, 1u);
    return false;
}

// One side's candidate of the merge zipper and what follows it: the edge and
// its twin, the destination of the next edge around the candidate's origin
// (the one whose circle test decides whether the candidate stays), and the
// pair that becomes the candidate when the zipper advances on this side.
struct Cand {
    int e;
    int4 a, b;      // records of e and e ^ 1
    Pt next;        // destination of the next edge around the origin
    int adv;        // the candidate after an advance on this side
    int4 va, vb;    // its records
};

// kLeft: the next edge around the origin is dnext(twin), and the advance goes
// to dnext; else they are twin(oprev) and twin(oprev(twin)).
template <bool kLeft>
__device__ __forceinline__ void cand_follow(const TinGraph &G, Cand &c) {
    c.adv = kLeft ? c.a.x : (c.b.y ^ 1);
    const int4 nx = rec(G, kLeft ? (c.b.x ^ 1) : c.a.y);
    c.va = rec(G, c.adv);
    c.vb = rec(G, c.adv ^ 1);
    c.next = pt_of(nx);
}
template <bool kLeft>
__device__ __forceinline__ void cand_load(const TinGraph &G, int e, Cand &c) {
    c.e = e;
    c.a = rec(G, e);
    c.b = rec(G, e ^ 1);
    cand_follow<kLeft>(G, c);
}

// The merge zipper (NextCrossEdge, grid_triangulation.cpp:1287-1335, from the
// lower common tangent up): bridges from `base` until neither side has a
// candidate above; returns the last bridge.  The reference's steps in its
// order.  It is a chain of dependent accesses, so the base edge and both
// candidates with what follows them stay in registers: an advance on one
// side finds its candidate already loaded and waits only for the records
// after it, and a bridge's stores are applied to the held records; where
// they touch others than the usual ones, or an edge was removed, the records
// are loaded again.
__device__ int zipper(const TinGraph &G, Alloc &al, int base, long long &steps, long long bound) {
    int4 Ba = rec(G, base), Bb = rec(G, base ^ 1);
    Cand L, R;
    cand_load<true>(G, Ba.x, L);
    cand_load<false>(G, Ba.y ^ 1, R);
    for (;;) {
        if (!step_ok(G, steps, bound)) return base;
        const Pt bo = pt_of(Ba), bd = pt_of(Bb);
        const bool valid_l = orient(bo, pt_of(L.a), pt_of(L.b)) < 0;
        bool removed = false;
        if (valid_l && incircle(pt_of(L.a), bo, pt_of(L.b), L.next) > 0) {
            removed = true;
            int l = L.e, next = dnext(G, l ^ 1);
            do {
                if (!step_ok(G, steps, bound)) return base;
                remove_edge_twin(G, al, l);
                l = next;
                next = dnext(G, l ^ 1);
            } while (incircle(orig(G, l), bo, dest(G, l), dest(G, next)) > 0);
            cand_load<false>(G, R.e, R);
            L.e = l;
        }
        const bool valid_r = orient(bd, bo, pt_of(R.b)) > 0;
        if (valid_r && incircle(bd, bo, pt_of(R.b), R.next) > 0) {
            removed = true;
            int r = R.e, next = oprev(G, r) ^ 1;
            do {
                if (!step_ok(G, steps, bound)) return base;
                remove_edge_twin(G, al, r);
                r = next;
                next = oprev(G, r) ^ 1;
            } while (incircle(bd, bo, dest(G, r), dest(G, next)) > 0);
            R.e = r;
        }
        if (removed) {
            Ba = rec(G, base);
            Bb = rec(G, base ^ 1);
            cand_load<true>(G, L.e, L);
            cand_load<false>(G, R.e, R);
        }
        if (!valid_l && !valid_r) return base;
        const int e = new_pair(G, al), et = e ^ 1;
        if (!valid_l || (valid_r && incircle(pt_of(L.b), pt_of(L.a), pt_of(R.a), pt_of(R.b)) > 0)) {
            // bridge(base, twin(r)): advance on the right
            const int end = R.e ^ 1, X = L.e, prev = L.a.y;
            const int prev2 = end == X ? et : R.b.y;
            const Pt d = pt_of(R.b);
            G.edge[e] = make_int4(end, prev, bd.c, bd.r);
            G.edge[et] = make_int4(X, prev2, d.c, d.r);
            G.edge[X].y = et;
            G.edge[prev].x = e;
            G.edge[end].y = e;
            G.edge[prev2].x = et;
            // (pairs of the stores against the pairs held: unusual)
            const int pl = L.e >> 1, pa = L.adv >> 1, pr = R.adv >> 1;
            const int s1 = prev >> 1, s2 = end >> 1, s3 = prev2 >> 1;
            const bool odd = s1 == pl || s1 == pa || s1 == pr || s2 == pl || s2 == pa || s2 == pr ||
                             s3 == pl || s3 == pa || pa == pl || prev2 == et;
            base = et;
            if (odd) {
                Ba = rec(G, base);
                Bb = rec(G, base ^ 1);
                cand_load<true>(G, Ba.x, L);
                cand_load<false>(G, Ba.y ^ 1, R);
            } else {
                Ba = make_int4(X, prev2, d.c, d.r);
                Bb = make_int4(end, prev, bd.c, bd.r);
                L.a.y = et;
                R.e = R.adv;          // prev2 ^ 1
                R.a = R.va;
                R.b = R.vb;
                R.b.x = et;
                cand_follow<false>(G, R);
            }
        } else {
            // bridge(l, base): advance on the left
            const int end = base, X = L.a.x, prev = L.va.y;
            const int prev2 = end == X ? et : Ba.y;
            const Pt o = pt_of(L.b);
            G.edge[e] = make_int4(end, prev, o.c, o.r);
            G.edge[et] = make_int4(X, prev2, bo.c, bo.r);
            G.edge[X].y = et;
            G.edge[prev].x = e;
            G.edge[end].y = e;
            G.edge[prev2].x = et;
            const int pa = L.adv >> 1, pr = R.e >> 1, pv = R.adv >> 1;
            const int s1 = prev >> 1, s2 = end >> 1, s3 = prev2 >> 1;
            const bool odd = s1 == pa || s1 == pr || s1 == pv || s2 == pa || s2 == pr || s2 == pv ||
                             s3 == pa || s3 == pv || pa == pr || pa == pv || prev2 == et;
            base = et;
            if (odd) {
                Ba = rec(G, base);
                Bb = rec(G, base ^ 1);
                cand_load<true>(G, Ba.x, L);
                cand_load<false>(G, Ba.y ^ 1, R);
            } else {
                Ba = make_int4(X, prev2, bo.c, bo.r);
                Bb = make_int4(end, prev, o.c, o.r);
                R.b.x = et;           // prev2 is twin(r)
                L.e = X;
                L.a = L.va;
                L.b = L.vb;
                L.a.y = et;
                cand_follow<true>(G, L);
            }
        }
    }
}

// Triangulate2 / Triangulate3 (grid_triangulation.cpp:580-699) on the node's
// points in the order its parent sorted them.
__device__ inline Ext base_case(const TinGraph &G, const int2 *pts, int cnt, Alloc &a) {
    Ext x;
    if (cnt == 2) {
        const Pt pa{pts[0].x, pts[0].y}, pb{pts[1].x, pts[1].y};
        const int e = add_edge_twin(G, a, pa, pb);
        const bool xy = less_xy(pa, pb), yx = less_yx(pa, pb);
        x.l = xy ? e : e ^ 1;
        x.r = xy ? e ^ 1 : e;
        x.b = yx ? e : e ^ 1;
        x.t = yx ? e ^ 1 : e;
        return x;
    }
    Pt A{pts[0].x, pts[0].y}, B{pts[1].x, pts[1].y}, C{pts[2].x, pts[2].y};
    auto order = [](Pt &p, Pt &q, bool swap) {
        if (swap) {
            const Pt t = p;
            p = q;
            q = t;
        }
    };
    // sort the three by (col, row)
    order(A, B, less_xy(B, A));
    order(B, C, less_xy(C, B));
    order(A, B, less_xy(B, A));
    int e1 = add_edge_twin(G, a, A, B);
    int e2 = add_edge_twin(G, a, B, C);
    weld(G, e1, e2);
    int e3;
    long long s = orient(A, B, C);
    if (s > 0) {
        e3 = bridge(G, a, e2, e1);
        x.l = e1;
        x.r = e2 ^ 1;
    } else if (s < 0) {
        e3 = bridge(G, a, e2, e1);
        x.l = e3 ^ 1;
        x.r = e3;
    } else {
        x.l = e1;
        x.r = e2 ^ 1;
    }
    // the same three by (row, -col)
    order(A, B, less_yx(B, A));
    order(B, C, less_yx(C, B));
    order(A, B, less_yx(B, A));
    const int e = same(orig(G, e1), A) ? e1 : (same(orig(G, e2), A) ? e2 : e2 ^ 1);
    e1 = same(dest(G, e), B) ? e : dnext(G, e ^ 1);
    e2 = dnext(G, e1);
    e3 = dnext(G, e2);
    s = orient(A, B, C);
    if (s >= 0) {
        x.b = e1;
        x.t = e2 ^ 1;
    } else {
        x.b = e3 ^ 1;
        x.t = e3;
    }
    return x;
}

// The merge of a node's two triangulated halves
// (TriangulateHorizontalSerial / TriangulateVerticalSerial,
// grid_triangulation.cpp:417-578): common tangent, zipper, new extremes.
__device__ inline Ext merge_halves(const TinGraph &G, bool horiz, Ext L, Ext R, Alloc &a,
                                   long long bound) {
    long long steps = 0;
    // the tangent walk from the facing extremes: p on the left (bottom) half,
    // q on the right (top) one
    int p = horiz ? L.r : L.t, q = horiz ? R.l : R.b;
    {
        int4 P = rec(G, p), Pt_ = rec(G, p ^ 1), Q = rec(G, q), Qt = rec(G, q ^ 1);
        for (;;) {
            if (!step_ok(G, steps, bound)) return L;
            if (orient(pt_of(P), pt_of(Pt_), pt_of(Q)) > 0) {
                p = Pt_.y ^ 1;       // twin(oprev(twin(p)))
                P = rec(G, p);
                Pt_ = rec(G, p ^ 1);
            } else if (orient(pt_of(Q), pt_of(Qt), pt_of(P)) < 0) {
                q = Q.x;             // dnext(q)
                Q = rec(G, q);
                Qt = rec(G, q ^ 1);
            } else {
                break;
            }
        }
    }
    const int first = bridge(G, a, oprev(G, q), dnext(G, p ^ 1));
    Ext x;
    if (horiz) {
        if (same(orig(G, p), orig(G, L.l))) L.l = first ^ 1;
        if (same(orig(G, q), orig(G, R.r))) R.r = first;
        const int last = zipper(G, a, first, steps, bound);
        x.l = L.l;
        x.r = R.r;
        int t = first ^ 1;
        while (less_yx(orig(G, t), dest(G, t)) && step_ok(G, steps, bound)) t = oprev(G, t);
        t = dnext(G, t);
        while (less_yx(dest(G, t), orig(G, t)) && step_ok(G, steps, bound)) t = dnext(G, t);
        x.b = t;
        t = last ^ 1;
        while (less_yx(dest(G, t), orig(G, t)) && step_ok(G, steps, bound)) t = dnext(G, t ^ 1) ^ 1;
        t = oprev(G, t ^ 1) ^ 1;
        while (less_yx(orig(G, t), dest(G, t)) && step_ok(G, steps, bound)) t = oprev(G, t ^ 1) ^ 1;
        x.t = t;
    } else {
        if (same(orig(G, p), orig(G, L.b))) L.b = first ^ 1;
        if (same(orig(G, q), orig(G, R.t))) R.t = first;
        const int last = zipper(G, a, first, steps, bound);
        x.b = L.b;
        x.t = R.t;
        int t = first;
        while (less_xy(dest(G, t), orig(G, t)) && step_ok(G, steps, bound)) t = dnext(G, t ^ 1) ^ 1;
        t = oprev(G, t ^ 1) ^ 1;
        while (less_xy(orig(G, t), dest(G, t)) && step_ok(G, steps, bound)) t = oprev(G, t ^ 1) ^ 1;
        x.r = t;
        t = last;
        while (less_xy(orig(G, t), dest(G, t)) && step_ok(G, steps, bound)) t = oprev(G, t);
        t = dnext(G, t);
        while (less_xy(dest(G, t), orig(G, t)) && step_ok(G, steps, bound)) t = dnext(G, t);
        x.l = t;
    }
    return x;
}

// A subtree of fewer than 100 points (TriangulateHorizontalSerial /
// TriangulateVerticalSerial): the reference recurses without splitting its
// edge list, so the whole subtree draws from one allocator stack, children
// before parents, left before right.
__device__ inline Ext serial_subtree(const TinGraph &G, const int2 *pts, int lo, int cnt, bool horiz,
                                     Alloc &a, long long bound) {
    struct Frame {
        int lo, cnt, state;
        Ext left;
    };
    Frame f[8];   // 99 points: halved at most six times
    int sp = 0;
    f[0].lo = lo;
    f[0].cnt = cnt;
    f[0].state = 0;
    Ext ret{0, 0, 0, 0};
    while (sp >= 0) {
        Frame &F = f[sp];
        if (F.cnt < 4) {
            ret = base_case(G, pts + F.lo, F.cnt, a);
            --sp;
            continue;
        }
        const int mid = F.cnt / 2;
        if (F.state == 2) {
            ret = merge_halves(G, horiz != (bool)(sp & 1), F.left, ret, a, bound);
            --sp;
            continue;
        }
        Frame &C = f[sp + 1];
        C.state = 0;
        if (F.state == 0) {
            C.lo = F.lo;
            C.cnt = mid;
        } else {
            F.left = ret;
            C.lo = F.lo + mid;
            C.cnt = F.cnt - mid;
        }
        ++F.state;
        ++sp;
    }
    return ret;
}

// The triangles around a point (Grid::GetAllTris, grid.cpp:16-51, and
// AdjTriIter, grid_iterators.hpp:63-110): counter-clockwise from the first
// face that is a triangle at or after its stored edge `e`, those of which it
// is the (col, row)-smallest vertex, passed to emit(e0, e1, e2), the edges out
// of its vertices.  Points of degree <= 2 whose edges are collinear have none.
template <class Emit>
__device__ inline void point_tris(const TinGraph &G, int e, long long bound, Emit emit) {
    if (e < 0) return;
    const int g = dnext(G, e ^ 1);
    const int f = dnext(G, g ^ 1);
    const Pt p1 = orig(G, e), p2 = dest(G, e), p3 = dest(G, g);
    const bool collinear = (p1.c - p2.c) * (p1.r - p3.r) == (p1.r - p2.r) * (p1.c - p3.c);
    if (f == e && collinear) return;
    long long steps = 0;
    int start = e;
    while (dnext(G, dnext(G, dnext(G, start))) != start && step_ok(G, steps, bound))
        start = dnext(G, start ^ 1);
    int cur = start;
    do {
        const int4 E0 = rec(G, cur);
        const int e1 = E0.x;
        const int4 E1 = rec(G, e1);
        const int e2 = E1.x;
        const Pt q0 = pt_of(E0), q1 = pt_of(E1), q2 = orig(G, e2);
        if (less_xy(q0, q1) && less_xy(q0, q2)) emit(cur, e1, e2);
        cur = dnext(G, cur ^ 1);
        while (dnext(G, dnext(G, dnext(G, cur))) != cur && step_ok(G, steps, bound))
            cur = dnext(G, cur ^ 1);
    } while (cur != start && step_ok(G, steps, bound));
}

}  // namespace tin
}  // namespace vll
