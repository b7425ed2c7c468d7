// gjk_pool.cuh -- the FP64 GJK over a pool of pairs per block.
//
// What bounds it: the FP64 pipe, which takes one warp instruction per 16
// cycles of an SM (64 from a single warp) however few lanes are active, and
// the length of a pair's chain of iterations (19 on average, ~75 at most).
// With one lane per pair the lanes of a warp sit in different support
// functions, simplex sizes and Voronoi regions: 7.9 of 32 lanes did FP64 work
// per instruction, and towards the end of a batch every round still paid for
// the two supports and up to four tetrahedron faces of its pairs one after
// the other.
//
// Here a block keeps one pair per thread in shared memory and runs its pairs
// in rounds of one iteration each.  A round is three phases, each of them a
// list of small tasks that any warp takes in chunks of one kind, so that the
// lanes of a warp run the same code on different pairs:
//
//   supports  one task per pair and side, listed by collider type (a box or a
//             hull finds its vertex through the FP32 filter, a hull with the
//             whole warp); the ends of the last round's finished pairs
//             (closest points, checks, outputs) are listed with them
//   advance   the pair's new Minkowski point and its clipping test, one thread
//             per pair; the pairs listed by simplex size
//   solve     tetrahedra sixteen per chunk: four lanes test the four planes of
//             one, then the faces that see the origin, one per lane; triangles,
//             segments and points one per lane; the solving lane also ends the
//             iteration (finish_step)
//
// The simplex rows never move: a pair's four logical rows map to four places
// through two bits each, so compaction is integer work; a row's place stays
// untouched while any logical row, live or stale, names it (the outputs hold
// the reference's stale rows).
//
// Every value is computed by the expressions of jolt.cuh, so the results are
// the reference's bit for bit, whichever lane computes them.
#pragma once

#include "gjk_out.cuh"
#include "jolt.cuh"
#include "persist.cuh"

namespace d3d {
namespace pool {

constexpr unsigned kAll = 0xffffffffu;
constexpr int kTypes = 10;
constexpr int kEndBin = 2 * kTypes;  // after the collider types, each without and with a margin
constexpr int kBins = kEndBin + 1;
constexpr int kHullChunk = 4;    // hulls a warp scans one after the other
constexpr int kTetraChunk = 16;  // tetrahedra per chunk: ~27 of their faces see the origin
constexpr int kEndMin = 32;      // finished pairs that make an end chunk worth running
constexpr int kFetch = 32;       // pairs a warp claims from the order at a time

enum { kFree = 0, kLive = 1, kEnding = 2, kSpare = 3 };  // kSpare: beyond the share (persist.cuh)

// a pair's state word
__device__ __forceinline__ unsigned pack_meta(unsigned perm, int n, int fresh, int state, int gstate = 0,
                                              int status = 0) {
    return perm | ((unsigned)n << 8) | ((unsigned)fresh << 11) | ((unsigned)state << 13) | ((unsigned)gstate << 15) |
           ((unsigned)status << 17);
}
__device__ __forceinline__ int meta_n(unsigned m) { return (m >> 8) & 7; }
__device__ __forceinline__ int meta_fresh(unsigned m) { return (m >> 11) & 3; }
__device__ __forceinline__ int meta_state(unsigned m) { return (m >> 13) & 3; }
__device__ __forceinline__ int meta_gstate(unsigned m) { return (m >> 15) & 3; }
__device__ __forceinline__ int meta_status(unsigned m) { return (m >> 17) & 15; }
__device__ __forceinline__ int place_of(unsigned m, int row) { return (m >> (2 * row)) & 3; }

// The place that no logical row other than n names, for the row pushed next.
__device__ __forceinline__ int free_place(unsigned perm, int n) {
    unsigned used = 0;
#pragma unroll
    for (int r = 0; r < 4; ++r)
        if (r != n) used |= 1u << ((perm >> (2 * r)) & 3u);
    return __ffs(~used) - 1;
}

// A block's shared memory for S pairs.  PQ rows of support points per pair:
// four for the distance (its closest points need them), one for the
// intersection test.
template <int S, int PQ>
struct Mem {
    double Y[12 * S];  // coordinate c of place r of slot s at [(3 r + c) S + s]
    double P[3 * PQ * S], Q[3 * PQ * S];
    double dir[3 * S];
    double vl[S], prev[S];
    int col[2 * S];  // collider of side k at [k S + s]
    int pid[S];
    int it[S];
    unsigned meta[S];
    unsigned short list[2 * S];   // support and end tasks by bin: slot << 1 | side
    unsigned short solve[4 * S];  // slots to solve by size (tetrahedra first)
    int cnt[2][kBins];
    int scnt[2][4];
    int next[2][2];
    unsigned char task[S / 32][4 * kTetraChunk];

    __device__ d3 row(const double* a, int r, int s) const {
        return mk(a[(3 * r) * S + s], a[(3 * r + 1) * S + s], a[(3 * r + 2) * S + s]);
    }
    __device__ void put(double* a, int r, int s, d3 v) {
        a[(3 * r) * S + s] = v.x;
        a[(3 * r + 1) * S + s] = v.y;
        a[(3 * r + 2) * S + s] = v.z;
    }
    __device__ d3 y(unsigned m, int row_, int s) const { return row(Y, place_of(m, row_), s); }
    __device__ d3 direction(int s) const { return mk(dir[s], dir[S + s], dir[2 * S + s]); }
    // the support point of side `side` along the pair's direction
    __device__ void put_support(int s, int side, d3 x) {
        put(side ? Q : P, PQ == 4 ? meta_fresh(meta[s]) : 0, s, x);
    }
};

// P and Q rows of a pair for closest_points
template <int S, int PQ>
struct PoolRows {
    const Mem<S, PQ>* m;
    unsigned meta;
    int s;
    __device__ __forceinline__ d3 p(int k) const { return m->row(m->P, place_of(meta, k), s); }
    __device__ __forceinline__ d3 q(int k) const { return m->row(m->Q, place_of(meta, k), s); }
};

// order-preserving key of a float (not NaN)
__device__ __forceinline__ unsigned key32(float x) {
    const unsigned u = __float_as_uint(x);
    return (u >> 31) ? ~u : (u | 0x80000000u);
}
__device__ __forceinline__ float unkey32(unsigned k) { return __uint_as_float((k >> 31) ? (k & 0x7fffffffu) : ~k); }

// Ordering key of a support product: unsigned order equals the order of the
// doubles (-0 as +0); a NaN is 0, below every number.
__device__ __forceinline__ unsigned long long product_key(double x) {
    const unsigned long long u = (unsigned long long)__double_as_longlong(x);
    if ((u << 1) > 0xffe0000000000000ull) return 0ull;
    if ((u << 1) == 0ull) return 0x8000000000000000ull;
    return (u >> 63) ? ~u : (u | 0x8000000000000000ull);
}

// hull_argmax_filtered with the 32 lanes of the warp on one hull: the first
// maximum of V . d, or the first vertex if its product is NaN.
__device__ __forceinline__ int warp_argmax(const d3d_store& st, int off, int nv, d3 d, Filter32 f) {
    if (nv <= 1) return 0;
    const int ln = threadIdx.x & 31;
    float lo = -INFINITY, top = -INFINITY, second = -INFINITY;
    int ti = 0;
    bool fin = isfinite(f.dabs);
    // the loads of four rounds together
    const float4* const v = reinterpret_cast<const float4*>(st.verts32) + off;
#pragma unroll 1
    for (int k0 = ln; k0 < nv; k0 += 128) {
        float4 x[4];
#pragma unroll
        for (int h = 0; h < 4; ++h)
            if (k0 + 32 * h < nv) x[h] = __ldg(v + k0 + 32 * h);
#pragma unroll
        for (int h = 0; h < 4; ++h) {
            if (k0 + 32 * h >= nv) continue;
            const float2 se = filter_product(x[h], f);
            fin &= isfinite(se.x) && isfinite(se.y);
            lo = fmaxf(lo, se.x - se.y);
            const float up = se.x + se.y;
            if (up > top) {
                second = top;
                top = up;
                ti = k0 + 32 * h;
            } else {
                second = fmaxf(second, up);
            }
        }
    }
    const bool finite = __all_sync(kAll, fin);
    const float L = unkey32(__reduce_max_sync(kAll, key32(lo)));
    const unsigned cand = __ballot_sync(kAll, top >= L);
    const bool many = __any_sync(kAll, second >= L);
    if (finite && !many && __popc(cand) == 1) return __shfl_sync(kAll, ti, __ffs(cand) - 1);
    unsigned long long bk = 0ull;
    int bi = 0x7fffffff;
    bool nan0 = false;
#pragma unroll 1
    for (int k = ln; k < nv; k += 32) {
        const float2 se = filter_product(st.verts32, off + k, f);
        if (!finite || se.x + se.y >= L) {
            const d3 w = load_vertex(st.verts64, off + k);
            const unsigned long long key = product_key(dot102(w.x, w.y, w.z, d.x, d.y, d.z));
            if (k == 0 && key == 0ull) nan0 = true;
            if (key > bk) {
                bk = key;
                bi = k;
            }
        }
    }
    const unsigned hi = __reduce_max_sync(kAll, (unsigned)(bk >> 32));
    const unsigned low = __reduce_max_sync(kAll, (unsigned)(bk >> 32) == hi ? (unsigned)bk : 0u);
    const unsigned long long best = ((unsigned long long)hi << 32) | low;
    const unsigned i = __reduce_min_sync(kAll, bk == best ? (unsigned)bi : 0xffffffffu);
    return (__any_sync(kAll, nan0) || i >= (unsigned)nv) ? 0 : (int)i;
}

// Up to kHullChunk listed hulls (m.list[first ...]: slot << 1 | side), the
// whole warp on one at a time.  The pool m gives `list`, the colliders
// col[side S + slot], direction(slot) and put_support(slot, side, point).
template <int S, typename M>
__device__ __forceinline__ void hull_supports(M& m, const d3d_store& st, int first, int count) {
    const int ln = threadIdx.x & 31;
    const int e = m.list[first + (ln < count ? ln : count - 1)];
    const int slot = e >> 1, side = e & 1;
    const int ci = m.col[side * S + slot];
    int type, nv, off;
    load_meta(st, ci, type, nv, off);
    d3 d = m.direction(slot);
    if (side) d = -d;
    const Filter32 f = filter32(d);
    int win = 0;
#pragma unroll 1
    for (int j = 0; j < count; ++j) {
        Filter32 g;
        g.dx = __shfl_sync(kAll, f.dx, j);
        g.dy = __shfl_sync(kAll, f.dy, j);
        g.dz = __shfl_sync(kAll, f.dz, j);
        g.dabs = __shfl_sync(kAll, f.dabs, j);
        const d3 dj = mk(__shfl_sync(kAll, d.x, j), __shfl_sync(kAll, d.y, j), __shfl_sync(kAll, d.z, j));
        const int k = warp_argmax(st, __shfl_sync(kAll, off, j), __shfl_sync(kAll, nv, j), dj, g);
        if (ln == j) win = k;
    }
    if (ln < count) {
        d3 x = nv < 1 ? mk(double(NAN), double(NAN), double(NAN)) : load_vertex(st.verts64, off + win);
        Col<double> c;
        load_meta(st, ci, c);
        c.m = c.wrapped ? __ldg(st.rec64 + (size_t)ci * 16 + 15) : 0.0;
        m.put_support(slot, side, add_margin(c, x, d));
    }
}

// The listed support e (slot << 1 | side) of any type but a hull, by one lane.
template <int S, typename M>
__device__ __forceinline__ void lane_support(M& m, const d3d_store& st, int e) {
    const int s = e >> 1, side = e & 1;
    Col<double> c;
    load_col(st, m.col[side * S + s], c);
    d3 d = m.direction(s);
    if (side) d = -d;
    m.put_support(s, side, support(c, st, d));
}

// The rest of gjk_step after its solve (distance) or of the intersection test's
// iteration (gjk_intersection_jolt, _gjk_jolt.py:29-135), for slot s and the
// result of its solve; ysq(r) is |Y|^2 of place r.  Returns the intersection
// form's outcome, -1 while it runs.
template <int S, int PQ, typename Ysq>
__device__ __forceinline__ int finish_step(Mem<S, PQ>& m, int s, bool closer, d3 nv, double nl, int set, double tol_sq,
                                           int max_iter, const JoltEps<double>& E, Ysq ysq) {
    constexpr bool kDistance = PQ == 4;
    unsigned mt = m.meta[s];
    unsigned perm = mt & 0xffu;
    int n = meta_n(mt);
    d3 dir;
    double vl;
    if (closer) {
        dir = nv;
        vl = nl;
    } else {
        if (!kDistance) return 0;
        --n;
        set = (1 << n) - 1;
        dir = mk(m.dir[s], m.dir[S + s], m.dir[2 * S + s]);
        vl = m.vl[s];
    }
    if (!kDistance && (set == 15 || le_sq(vl, tol_sq))) return 1;
    int ending = -1;  // GjkEnd
    if (set == 15) {
        ending = GJK_INTERSECTION;
    } else {
        if (!kDistance) {
            // max |Y|^2 over the rows before compaction
            double y = ysq(place_of(mt, 0));
            for (int r = 1; r < n; ++r) {
                const double l = ysq(place_of(mt, r));
                if (lt_sq(y, l)) y = l;
            }
            if (le_sq(vl, E.isect * y)) return 1;
            dir = -dir;
            const double prev = m.prev[s];
            if (le(prev - vl, E.conv * prev)) return 0;
        }
        // keep the rows whose bit is set, in order
        int k = 0;
        unsigned np = perm;
#pragma unroll
        for (int r = 0; r < 4; ++r)
            if (r < n && ((set >> r) & 1)) {
                np = (np & ~(3u << (2 * k))) | (((perm >> (2 * r)) & 3u) << (2 * k));
                ++k;
            }
        perm = np;
        n = k;
        if (kDistance) {
            bool touch = le_sq(vl, tol_sq);
            if (!touch) {
                double y = ysq(place_of(perm, 0));
                for (int r = 1; r < n; ++r) {
                    const double l = ysq(place_of(perm, r));
                    if (lt_sq(y, l)) y = l;
                }
                touch = le_sq(vl, E.isect * y);
            }
            if (touch) {
                ending = GJK_INTERSECTION;
            } else {
                dir = -dir;
                const double prev = m.prev[s];
                if (le(prev - vl, E.conv * prev)) ending = GJK_NO_INTERSECTION;
            }
        }
    }
    int status = D3D_STATUS_OK;
    if (ending < 0) {
        m.prev[s] = vl;
        if (m.it[s] >= max_iter) {  // the bound, tested before the next iteration
            if (!kDistance) return 2;
            ending = GJK_NO_INTERSECTION;
            status = D3D_STATUS_MAX_ITER;
        }
    } else if (ending == GJK_INTERSECTION) {
        vl = 0.0;
    }
    m.vl[s] = vl;
    m.dir[s] = dir.x;
    m.dir[S + s] = dir.y;
    m.dir[2 * S + s] = dir.z;
    m.meta[s] = ending < 0 ? pack_meta(perm, n, free_place(perm, n), kLive)
                           : pack_meta(perm, n, 0, kEnding, ending, status);
    return -1;
}

template <int S, int PQ>
__device__ __forceinline__ int finish_step(Mem<S, PQ>& m, int s, bool closer, d3 nv, double nl, int set, double tol_sq,
                                           int max_iter, const JoltEps<double>& E) {
    return finish_step(m, s, closer, nv, nl, set, tol_sq, max_iter, E, [&](int r) {
        const d3 v = m.row(m.Y, r, s);
        return dot(v, v);
    });
}

// The pair of slot s has ended in the intersection form.
template <int S, int PQ>
__device__ __forceinline__ void put_hit(Mem<S, PQ>& m, int s, int hit, int8_t* hits, int8_t* status) {
    if (PQ == 4 || hit < 0) return;
    const int pid = m.pid[s];
    hits[pid] = (int8_t)(hit == 1);
    status[pid] = (int8_t)(hit == 2 ? D3D_STATUS_MAX_ITER : D3D_STATUS_OK);
    m.meta[s] = 0;
}

// cp_triangle with its regions merged: every value the regions share is
// computed once for all lanes, and the point on an edge takes the same
// division and the same products whichever edge it is.  The lanes of a warp
// sit in different regions, so the branches of cp_triangle were paid for one
// after the other: three edges and the face with six divisions in all.
__device__ __forceinline__ d3 flat_triangle(d3 a, d3 b, d3 c, const JoltEps<double>& E, int& set) {
    const d3 ab = b - a, ac = c - a, bc = c - b;
    const bool shorter = lt_sq(dot(bc, bc), dot(ac, ac));
    const d3 n = cross(ab, mk(shorter ? bc.x : ac.x, shorter ? bc.y : ac.y, shorter ? bc.z : ac.z));
    const double nl = dot(n, n);
    if (lt_sq(nl, E.sq)) return cp_triangle(a, b, c, E, set);  // degenerate
    const double d1 = dot(ab, -a), d2 = dot(ac, -a), d3_ = dot(ab, -b), d4 = dot(ac, -b), d5 = dot(ab, -c),
                 d6 = dot(ac, -c);
    const double vc = d1 * d4 - d3_ * d2, vb = d5 * d2 - d1 * d6, va = d3_ * d6 - d5 * d4;
    const double d43 = d4 - d3_, d56 = d5 - d6;
    const bool d3up = not_below0(d3_), d6up = not_below0(d6);
    if (not_above0(d1) && not_above0(d2))
        set = 1;
    else if (d3up && le(d4, d3_))
        set = 2;
    else if (not_above0(vc) && not_below0(d1) && not_above0(d3_))
        set = 3;
    else if (d6up && le(d5, d6))
        set = 4;
    else if (not_above0(vb) && not_below0(d2) && not_above0(d6))
        set = 5;
    else if (not_above0(va) && not_below0(d43) && not_below0(d56))
        set = 6;
    else
        set = 7;
    d3 r = set == 2 ? b : (set == 4 ? c : a);
    if (set == 3 || set >= 5) {
        // edges: base + edge * (num / (num + rest)); the face: n * s / den per component
        double num = set == 3 ? d1 : (set == 5 ? d2 : d43);
        double den = num + (set == 3 ? -d3_ : (set == 5 ? -d6 : d56));
        double s = 0.0;
        if (set == 7) {
            s = dot((a + b) + c, n);
            den = 3.0 * nl;
            num = n.x * s;
        }
        const double q = num / den;
        if (set == 7) {
            r = mk(q, n.y * s / den, n.z * s / den);
        } else {
            const d3 e = set == 3 ? ab : (set == 5 ? ac : bc);
            r = (set == 6 ? b : a) + e * q;
        }
    }
    return r;
}

// Up to kTetraChunk tetrahedra (m.solve[first ...]): closest_to_origin with
// four lanes on the planes of one tetrahedron and one lane per tested face.
template <int S, int PQ>
__device__ __forceinline__ void solve_tetrahedra(Mem<S, PQ>& m, int first, int count, double tol_sq, int max_iter,
                                                 const JoltEps<double>& E, int8_t* hits, int8_t* status) {
    const int ln = threadIdx.x & 31;
    unsigned char* const task = m.task[threadIdx.x >> 5];
    unsigned vis[kTetraChunk / 8];
    int T = 0;
    // outside_planes, plane j = lane & 3 of tetrahedron lane >> 2 of each eight
#pragma unroll
    for (int h = 0; h < kTetraChunk / 8; ++h) {
        vis[h] = 0;
        if (8 * h >= count) continue;
        const int i = 8 * h + (ln >> 2), j = ln & 3;
        const bool on = i < count;
        double sp = 0.0, sd = 0.0;
        if (on) {
            const int s = m.solve[first + i];
            const unsigned mt = m.meta[s];
            // planes: a, ab x ac, ad;  a, ac x ad, ab;  a, ad x ab, ac;  b, bd x bc, -ab
            const d3 a = m.y(mt, 0, s);
            const d3 o = j == 3 ? m.y(mt, 1, s) : a;
            const d3 e1 = m.y(mt, j == 0 ? 1 : (j == 1 ? 2 : 3), s) - o;
            const d3 e2 = m.y(mt, j == 0 ? 2 : (j == 1 ? 3 : (j == 2 ? 1 : 2)), s) - o;
            const d3 e3 = m.y(mt, j == 0 ? 3 : (j == 2 ? 2 : 1), s) - a;
            const d3 c = cross(e1, e2);
            sp = dot(o, c);
            sd = dot(e3, c);
            if (j == 3) sd = -sd;
        }
        const int q = ln & ~3;
        const bool up = ((__ballot_sync(kAll, on && above0(sd)) >> q) & 15u) == 15u;
        const bool down = ((__ballot_sync(kAll, on && below0(sd)) >> q) & 15u) == 15u;
        const bool out = up ? le(-E.plane, sp) : (down ? le(sp, E.plane) : true);
        vis[h] = __ballot_sync(kAll, on && out);
        if (on && out) task[T + __popc(vis[h] & ((1u << ln) - 1u))] = (unsigned char)(32 * h + ln);
        T += __popc(vis[h]);
    }
    __syncwarp();
    // the faces abc, acd, adb, bdc that were listed, one per lane; lane i keeps the best of tetrahedron i
    d3 bv = mk(0.0, 0.0, 0.0);
    double bd = DBL_MAX, bl = 0.0;
    int bs = 15;
#pragma unroll 1
    for (int base = 0; base < T; base += 32) {
        d3 r = mk(0.0, 0.0, 0.0);
        double d2 = 0.0;
        int set = 0;
        if (base + ln < T) {
            const int x = task[base + ln];
            const int f = x & 3;
            const int s = m.solve[first + (x >> 2)];
            const unsigned mt = m.meta[s];
            const int i0 = f == 3 ? 1 : 0;
            const int i1 = f == 0 ? 1 : (f == 1 ? 2 : 3);
            const int i2 = f == 0 ? 2 : (f == 1 ? 3 : (f == 2 ? 1 : 2));
            int ns;
            r = flat_triangle(m.y(mt, i0, s), m.y(mt, i1, s), m.y(mt, i2, s), E, ns);
            d2 = dot(r, r);
            set = ((ns & 1) << i0) | (((ns >> 1) & 1) << i1) | (((ns >> 2) & 1) << i2);
        }
        // tetrahedron ln: faces in order, the first taken as it is, later ones if strictly closer
        const int below = 4 * (ln & 7);
#pragma unroll
        for (int f = 0; f < 4; ++f) {
            unsigned v = 0;
            int rank = -base;
#pragma unroll
            for (int h = 0; h < kTetraChunk / 8; ++h) {
                if (h < (ln >> 3)) rank += __popc(vis[h]);
                if (h == (ln >> 3)) v = vis[h];
            }
            const int bit = below + f;
            rank += __popc(v & ((1u << bit) - 1u));
            const bool mine = ln < kTetraChunk && ((v >> bit) & 1u) && rank >= 0 && rank < 32;
            const int src = mine ? rank : 0;
            const double fd = __shfl_sync(kAll, d2, src);
            const d3 fv = mk(__shfl_sync(kAll, r.x, src), __shfl_sync(kAll, r.y, src), __shfl_sync(kAll, r.z, src));
            const int fs = __shfl_sync(kAll, set, src);
            if (mine && (f == 0 || lt_sq(fd, bd))) {
                bd = bl = fd;
                bv = fv;
                bs = fs;
            }
        }
    }
    if (ln < count) {
        const int s = m.solve[first + ln];
        put_hit(m, s, finish_step(m, s, lt_sq(bl, m.prev[s]), bv, bl, bs, tol_sq, max_iter, E), hits, status);
    }
    __syncwarp();  // the task list is rewritten by the warp's next chunk
}

__device__ __forceinline__ double shfl8(double x, int j) { return __shfl_sync(kAll, x, j, 8); }
__device__ __forceinline__ d3 shfl8(d3 v, int j) { return mk(shfl8(v.x, j), shfl8(v.y, j), shfl8(v.z, j)); }
__device__ __forceinline__ double coord(d3 v, int j) { return j == 0 ? v.x : (j == 1 ? v.y : v.z); }

// One triangle or tetrahedron by the whole warp, where a block has no more of
// them than warps: the length of the chain counts then, not the pipe.  Eight
// lanes take each face of a tetrahedron (a triangle has one), tested by its
// plane or not, and spread the independent products of flat_triangle: the six
// corner dots and two edge lengths on a lane each, the normal's and the
// closest point's components on three, so that a solve is ~45 dependent FP64
// instructions instead of ~150.  The values are flat_triangle's and
// outside_planes', operation by operation.  1,000 primitive pairs: 609 -> 505 us.
template <int S, int PQ>
__device__ __forceinline__ void solve_wide(Mem<S, PQ>& m, int s, double tol_sq, int max_iter, const JoltEps<double>& E,
                                           int8_t* hits, int8_t* status) {
    const int ln = threadIdx.x & 31, f = ln >> 3, j = ln & 7;
    const unsigned mt = m.meta[s];
    const bool tetra = meta_n(mt) == 4;
    const int i0 = f == 3 ? 1 : 0;
    const int i1 = f == 0 ? 1 : (f == 1 ? 2 : 3);
    const int i2 = f == 0 ? 2 : (f == 1 ? 3 : (f == 2 ? 1 : 2));
    const d3 a = m.y(mt, i0, s), b = m.y(mt, i1, s), c = m.y(mt, i2, s);
    // lanes 0-5: d1 .. d6 (ab or ac against -a, -b, -c), 6: bc . bc, 7: ac . ac
    const bool toc = j == 1 || j == 3 || j >= 5;
    const d3 e = (toc ? c : b) - (j == 6 ? b : a);
    const d3 u = j < 2 ? -a : (j < 4 ? -b : (j < 6 ? -c : e));
    const double dj = dot(e, u);
    const double d1 = shfl8(dj, 0), d2 = shfl8(dj, 1), d3_ = shfl8(dj, 2), d4 = shfl8(dj, 3), d5 = shfl8(dj, 4),
                 d6 = shfl8(dj, 5);
    const d3 ab = shfl8(e, 0), ac = shfl8(e, 1), bc = shfl8(e, 6);
    const bool shorter = lt_sq(shfl8(dj, 6), shfl8(dj, 7));
    const d3 x = shorter ? bc : ac;
    // lanes 0-2: the normal ab x (bc or ac), 3-5: vc, vb, va
    double n1 = 0.0, n2 = 0.0, n3 = 0.0, n4 = 0.0;
    if (j < 3) {
        const int k = j == 2 ? 0 : j + 1, l = j == 0 ? 2 : j - 1;
        n1 = coord(ab, k);
        n2 = coord(x, l);
        n3 = coord(ab, l);
        n4 = coord(x, k);
    } else if (j < 6) {
        n1 = j == 3 ? d1 : (j == 4 ? d5 : d3_);
        n2 = j == 3 ? d4 : (j == 4 ? d2 : d6);
        n3 = j == 3 ? d3_ : (j == 4 ? d1 : d5);
        n4 = j == 3 ? d2 : (j == 4 ? d6 : d4);
    }
    const double pj = n1 * n2 - n3 * n4;
    const d3 n = mk(shfl8(pj, 0), shfl8(pj, 1), shfl8(pj, 2));
    const double vc = shfl8(pj, 3), vb = shfl8(pj, 4), va = shfl8(pj, 5);
    // the plane of the face (tetrahedra): normal ab x ac, and the fourth corner's edge from corner 0
    d3 cr = n, e3 = n;
    if (tetra) {
        const int k = j == 2 ? 0 : j + 1, l = j == 0 ? 2 : j - 1;
        const double cj = coord(ab, k) * coord(ac, l) - coord(ab, l) * coord(ac, k);
        const double ej = coord(m.y(mt, f == 0 ? 3 : (f == 2 ? 2 : 1), s), j) - coord(m.y(mt, 0, s), j);
        cr = mk(shfl8(cj, 0), shfl8(cj, 1), shfl8(cj, 2));
        e3 = mk(shfl8(ej, 0), shfl8(ej, 1), shfl8(ej, 2));
    }
    // lanes 0-2: (a + b) + c, 3: d43 + d56, 5: d1 - d3, 6: d2 - d6
    const double s1 = j < 3 ? coord(a, j) : (j == 3 ? d4 : (j == 4 ? d5 : (j == 5 ? d1 : d2)));
    const double s2 = j < 3 ? coord(b, j) : (j == 3 || j == 5 ? -d3_ : -d6);
    const double sj = s1 + s2;
    const double d43 = shfl8(sj, 3), d56 = shfl8(sj, 4), e13 = shfl8(sj, 5), e26 = shfl8(sj, 6);
    const double tj = (j < 3 ? sj : d43) + (j < 3 ? coord(c, j) : d56);
    const d3 sum = mk(shfl8(tj, 0), shfl8(tj, 1), shfl8(tj, 2));
    const double e46 = shfl8(tj, 3);
    // lane 0: |n|^2, 1: (a + b + c) . n, 2: the origin's side of the plane, 3: the fourth corner's
    const double uj = dot(j == 0 ? n : (j == 1 ? sum : (j == 2 ? a : e3)), j < 2 ? n : cr);
    const double nl = shfl8(uj, 0), sn = shfl8(uj, 1), sp = shfl8(uj, 2);
    double sd = shfl8(uj, 3);
    if (f == 3) sd = -sd;
    // flat_triangle's region tests, one value per lane: bit i of a mask is d(i + 1)'s, vc's .. va's
    // sit at bits 3 - 5, d43's and d56's at 3 and 4
    const int sh = 8 * f;
    const unsigned dn = __ballot_sync(kAll, not_above0(dj)) >> sh, du = __ballot_sync(kAll, not_below0(dj)) >> sh;
    const unsigned pn = __ballot_sync(kAll, not_above0(pj)) >> sh, su = __ballot_sync(kAll, not_below0(sj)) >> sh;
    const unsigned ord = __ballot_sync(kAll, le(j == 0 ? d4 : d5, j == 0 ? d3_ : d6)) >> sh;  // d4 <= d3, d5 <= d6
    int set = 7;
    if ((pn & 32u) && (su & 24u) == 24u) set = 6;
    if ((pn & 16u) && (du & 2u) && (dn & 32u)) set = 5;
    if ((du & 32u) && (ord & 2u)) set = 4;
    if ((pn & 8u) && (du & 1u) && (dn & 4u)) set = 3;
    if ((du & 4u) && (ord & 1u)) set = 2;
    if ((dn & 3u) == 3u) set = 1;
    const bool line = set == 3 || set == 5 || set == 6;
    const double mj = (j < 3 ? coord(n, j) : 3.0) * (j < 3 ? sn : nl);
    const double den7 = shfl8(mj, 3);
    double r1 = coord(set == 2 || set == 6 ? b : (set == 4 ? c : a), j);
    if (line || set == 7) {
        const double num = set == 7 ? mj : (set == 3 ? d1 : (set == 5 ? d2 : d43));
        const double den = set == 7 ? den7 : (set == 3 ? e13 : (set == 5 ? e26 : e46));
        const double q = num / den;
        r1 = line ? r1 + coord(set == 3 ? ab : (set == 5 ? ac : bc), j) * q : q;
    }
    __syncwarp();
    d3 r = mk(shfl8(r1, 0), shfl8(r1, 1), shfl8(r1, 2));
    if (lt_sq(nl, E.sq)) r = cp_triangle(a, b, c, E, set);  // degenerate
    const double l = dot(r, r);
    set = ((set & 1) << i0) | (((set >> 1) & 1) << i1) | (((set >> 2) & 1) << i2);
    // the faces that see the origin (a triangle's own)
    const bool up = (__ballot_sync(kAll, above0(sd)) & 0x01010101u) == 0x01010101u;
    const bool down = (__ballot_sync(kAll, below0(sd)) & 0x01010101u) == 0x01010101u;
    const bool out = tetra ? (up ? le(-E.plane, sp) : (down ? le(sp, E.plane) : true)) : f == 0;
    const unsigned vis = __ballot_sync(kAll, out);
    // place ln's |Y|^2 for the end of the iteration
    const d3 yv = m.row(m.Y, ln & 3, s);
    const double yy = dot(yv, yv);
    // the first face as it is (a NaN included), a later one if strictly closer: the smallest |r|^2,
    // then the lowest face
    const unsigned long long lb = (unsigned long long)__double_as_longlong(l);
    const bool in = j == 0 && out && (f == 0 || lb < 0x7fefffffffffffffull);
    const unsigned long long key = f == 0 && lb > 0x7ff0000000000000ull ? 0ull : lb;
    const unsigned khi = __reduce_min_sync(kAll, in ? (unsigned)(key >> 32) : 0xffffffffu);
    const unsigned klo = __reduce_min_sync(kAll, in && (unsigned)(key >> 32) == khi ? (unsigned)key : 0xffffffffu);
    const unsigned win = __ballot_sync(kAll, in && key == (((unsigned long long)khi << 32) | klo));
    const int from = win ? __ffs(win) - 1 : 0;
    d3 bv = mk(__shfl_sync(kAll, r.x, from), __shfl_sync(kAll, r.y, from), __shfl_sync(kAll, r.z, from));
    double bl = __shfl_sync(kAll, l, from);
    int bs = __shfl_sync(kAll, set, from);
    if (!win) {
        bv = mk(0.0, 0.0, 0.0);
        bl = 0.0;
        bs = 15;
    }
    const double y0 = __shfl_sync(kAll, yy, 0), y1 = __shfl_sync(kAll, yy, 1), y2 = __shfl_sync(kAll, yy, 2),
                 y3 = __shfl_sync(kAll, yy, 3);
    if (ln == 0)
        put_hit(m, s,
                finish_step(m, s, lt_sq(bl, m.prev[s]), bv, bl, bs, tol_sq, max_iter, E,
                            [=](int p) { return p == 0 ? y0 : (p == 1 ? y1 : (p == 2 ? y2 : y3)); }),
                hits, status);
}

// The pairs of a batch dealt to the blocks in runs of 1 << run: the lanes that
// want one take the block's next, counted in *dealt (shared memory).
__device__ __forceinline__ unsigned dealt_slot(unsigned* dealt, bool want, int run) {
    const unsigned w = __ballot_sync(kAll, want);
    if (!w) return 0u;
    const int ln = threadIdx.x & 31, leader = __ffs(w) - 1;
    unsigned x = 0;
    if (ln == leader) x = atomicAdd(dealt, (unsigned)__popc(w));
    x = __shfl_sync(kAll, x, leader) + __popc(w & ((1u << ln) - 1u));
    return ((x >> run) * gridDim.x + blockIdx.x << run) | (x & ((1u << run) - 1u));
}

// The FP64 GJK distance (PQ = 4) or intersection test (PQ = 1) of the pairs
// order[k] (or k), k < n (or *n_dev): see the top of this file.  S threads
// and pairs per block.  The distances' blocks claim pairs from *cursor.  The
// intersection test takes no memory but its arguments (null order, n_dev and
// cursor): the pairs are dealt to the blocks in input order, and a block counts
// its own in shared memory.
template <int S, int PQ>
__global__ void __launch_bounds__(S, 512 / S) k_gjk_pool(d3d_store st, const int32_t* __restrict__ i1,
                                                         const int32_t* __restrict__ i2,
                                                         const int32_t* __restrict__ order, int64_t n,
                                                         const unsigned long long* __restrict__ n_dev,
                                                         unsigned long long* __restrict__ cursor, d3d_gjk_options opt,
                                                         DistanceOut o, int8_t* __restrict__ hits) {
    constexpr bool kDistance = PQ == 4;
    extern __shared__ __align__(16) unsigned char pool_smem[];
    Mem<S, PQ>& m = *reinterpret_cast<Mem<S, PQ>*>(pool_smem);
    const int t = threadIdx.x, ln = t & 31;
    if (n_dev) n = (int64_t)*n_dev;
    const JoltEps<double> E = reference_eps<double>();
    const double tol_sq = opt.tolerance * opt.tolerance;
    // a batch that does not fill every block is spread evenly over them
    const long long share = (n + gridDim.x - 1) / gridDim.x;
    const long long split = share < S ? 0 : n;
    bool exhausted = kDistance ? share == 0 : t >= share;
    WarpChunk32 chunk;
    __shared__ unsigned dealt;
    if (!kDistance && t == 0) dealt = 0u;
    m.meta[t] = !exhausted && t >= share ? pack_meta(0, 0, 0, kSpare) : 0;
    if (!exhausted && t >= share) m.it[t] = spare_rounds(t, share);
    if (t < kBins) m.cnt[0][t] = m.cnt[1][t] = 0;
    if (t < 4) m.scnt[0][t] = m.scnt[1][t] = m.next[t >> 1][t & 1] = 0;
    int type0 = 0, type1 = 0;
    __syncthreads();
    for (int par = 0;; par ^= 1) {
        // ---- free slots take new pairs
        int state = meta_state(m.meta[t]);
        const bool want = state == kFree && !exhausted;
        const long long slot = kDistance ? fetch_slot_chunked(cursor, want, chunk, kAll, kFetch, split)
                                         : (long long)dealt_slot(&dealt, want, share < S ? 0 : 5);
        if (want) {
            if (slot >= n) {
                exhausted = true;
            } else {
                const int pid = order ? order[slot] : (int)slot;
                const int a = i1[pid], b = i2[pid];
                if (!pair_ok(st, a, b)) {  // reported at once, no record read
                    if (kDistance) {
                        store_bad_index(o, pid);
                    } else {
                        hits[pid] = 0;
                        o.status[pid] = (int8_t)D3D_STATUS_BAD_INDEX;
                    }
                } else {
                    const int4 ma = __ldg(reinterpret_cast<const int4*>(st.meta) + a);
                    const int4 mb = __ldg(reinterpret_cast<const int4*>(st.meta) + b);
                    type0 = 2 * min(max(ma.x, 0), kTypes - 1) + (ma.w ? 1 : 0);
                    type1 = 2 * min(max(mb.x, 0), kTypes - 1) + (mb.w ? 1 : 0);
                    m.col[t] = a;
                    m.col[S + t] = b;
                    m.pid[t] = pid;
                    m.it[t] = 0;
                    for (int k = 0; k < 12; ++k) m.Y[k * S + t] = 0.0;
                    m.dir[t] = 1.0;
                    m.dir[S + t] = m.dir[2 * S + t] = 0.0;
                    m.vl[t] = 1.0;
                    m.prev[t] = DBL_MAX;
                    m.meta[t] = pack_meta(0xe4u, 0, 0, kLive);  // rows 0-3 in places 0-3
                    state = kLive;
                }
            }
        }
        // ---- list the supports and the ends
        int pos[2];
#pragma unroll
        for (int k = 0; k < 2; ++k) {
            const int bin = state == kLive ? (k ? type1 : type0) : (state == kEnding && k == 0 ? kEndBin : -1);
            const unsigned same = __match_any_sync(kAll, bin);
            const int leader = __ffs(same) - 1;
            int base = 0;
            if (ln == leader && bin >= 0) base = atomicAdd(&m.cnt[par][bin], __popc(same));
            pos[k] = __shfl_sync(kAll, base, leader) + __popc(same & ((1u << ln) - 1u));
        }
        if (!__syncthreads_or(state == kFree ? !exhausted : state != kSpare)) break;
        // bin ln of the list: its first task and first chunk; the finished pairs wait until they
        // fill a warp, or no pair is left to iterate
        const int size = (ln >> 1) == D3D_HULL ? kHullChunk : 32;
        int c = ln < kBins ? m.cnt[par][ln] : 0;
        const unsigned iterating = __ballot_sync(kAll, c > 0) & ((1u << kEndBin) - 1u);
        if (ln == kEndBin && c < kEndMin && iterating) c = 0;
        const bool ends = __shfl_sync(kAll, c, kEndBin) > 0;
        int tasks = c, chunks = (c + size - 1) / size;
#pragma unroll
        for (int k = 1; k < 32; k <<= 1) {
            const int a = __shfl_up_sync(kAll, tasks, k), b = __shfl_up_sync(kAll, chunks, k);
            if (ln >= k) {
                tasks += a;
                chunks += b;
            }
        }
        const int total = __shfl_sync(kAll, chunks, 31);
        const int task0 = tasks - c;
        {
            const int p0 = __shfl_sync(kAll, task0, state == kEnding ? kEndBin : type0) + pos[0];
            const int p1 = __shfl_sync(kAll, task0, type1) + pos[1];
            if (state == kLive || (state == kEnding && ends)) m.list[p0] = (unsigned short)(2 * t);
            if (state == kLive) m.list[p1] = (unsigned short)(2 * t + 1);
        }
        __syncthreads();
        // ---- supports and ends
        while (true) {
            int x = 0;
            if (ln == 0) x = atomicAdd(&m.next[par][0], 1);
            x = __shfl_sync(kAll, x, 0);
            if (x >= total) break;
            x = total - 1 - x;  // the ends and the long supports first
            const int bin = __popc(__ballot_sync(kAll, chunks <= x));
            const int csize = (bin >> 1) == D3D_HULL ? kHullChunk : 32;
            const int cbin = __shfl_sync(kAll, c, bin);
            const int k0 = (x - __shfl_sync(kAll, chunks, bin) + (cbin + csize - 1) / csize) * csize;
            const int first = __shfl_sync(kAll, task0, bin) + k0;
            const int count = min(csize, cbin - k0);
            if ((bin >> 1) == D3D_HULL) {
                hull_supports<S>(m, st, first, count);
            } else if (ln < count) {
                const int e = m.list[first + ln];
                const int s = e >> 1;
                if (bin == kEndBin) {
                    if (kDistance) {
                        const unsigned mt = m.meta[s];
                        GjkLoop<double, PoolRows<S, PQ>> g;
                        g.S.R.m = &m;
                        g.S.R.meta = mt;
                        g.S.R.s = s;
                        g.S.n = meta_n(mt);
#pragma unroll
                        for (int r = 0; r < 4; ++r) g.S.Y[r] = m.y(mt, r, s);
                        g.dir = mk(m.dir[s], m.dir[S + s], m.dir[2 * S + s]);
                        g.vl = m.vl[s];
                        g.it = m.it[s];
                        g.state = meta_gstate(mt);
                        g.status = meta_status(mt);
                        GjkResult<double> r;
                        gjk_end(g, opt.sanity_check, E, r);
                        store_result(o, m.pid[s], r, g.S);
                        m.meta[s] = 0;
                    }
                } else {
                    lane_support<S>(m, st, e);
                }
            }
            __syncwarp();
        }
        __syncthreads();
        // ---- advance: the new Minkowski point (gjk_step between its supports and its solve)
        int cls = -1;
        if (state == kLive) {
            const unsigned mt = m.meta[t];
            const int f = meta_fresh(mt), rows = meta_n(mt);
            const int r = kDistance ? f : 0;
            const d3 w = m.row(m.P, r, t) - m.row(m.Q, r, t);
            const double dd = dot(mk(m.dir[t], m.dir[S + t], m.dir[2 * S + t]), w);
            m.it[t] += 1;
            if (!kDistance && lt(dd, -E.conv)) {
                put_hit(m, t, 0, hits, o.status);
            } else if (kDistance && below0(dd) && lt(m.vl[t] * opt.max_distance_squared, dd * dd)) {
                m.meta[t] = pack_meta(mt & 0xffu, rows, 0, kEnding, GJK_CLIPPED, D3D_STATUS_OK);
            } else {
                m.put(m.Y, f, t, w);
                const unsigned perm = (mt & 0xffu & ~(3u << (2 * rows))) | ((unsigned)f << (2 * rows));
                m.meta[t] = pack_meta(perm, rows + 1, 0, kLive);
                cls = 3 - rows;  // 0: tetrahedron .. 3: point
            }
        } else if (kDistance && state == kSpare) {
            exhausted = slots_claimed(cursor, n);
            if (exhausted || --m.it[t] == 0) m.meta[t] = 0;
        }
        {
            unsigned mine = 0;
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const unsigned b = __ballot_sync(kAll, cls == k);
                if (cls == k) mine = b;
                if (ln == k) pos[0] = b ? atomicAdd(&m.scnt[par][k], __popc(b)) : 0;
            }
            const int p = __shfl_sync(kAll, pos[0], cls >= 0 ? cls : 0) + __popc(mine & ((1u << ln) - 1u));
            if (cls >= 0) m.solve[cls * S + p] = (unsigned short)t;
        }
        // the other parity's counters, free since the last round
        if (t < kBins) m.cnt[par ^ 1][t] = 0;
        if (t < 4) m.scnt[par ^ 1][t] = 0;
        if (t < 2) m.next[par ^ 1][t] = 0;
        __syncthreads();
        // ---- solve
        const int n4 = m.scnt[par][0], n3 = m.scnt[par][1], n2 = m.scnt[par][2], n1 = m.scnt[par][3];
        const bool wide = n4 + n3 <= S / 32;  // no more than warps: each by a whole warp
        const int c4 = wide ? n4 + n3 : (n4 + kTetraChunk - 1) / kTetraChunk, c3 = wide ? 0 : (n3 + 31) / 32,
                  c2 = (n2 + 31) / 32, c1 = (n1 + 31) / 32;
        while (true) {
            int x = 0;
            if (ln == 0) x = atomicAdd(&m.next[par][1], 1);
            x = __shfl_sync(kAll, x, 0);
            if (x >= c4 + c3 + c2 + c1) break;
            if (x < c4 && wide) {
                solve_wide(m, m.solve[x < n4 ? x : S + x - n4], tol_sq, opt.max_iterations, E, hits, o.status);
                continue;
            }
            if (x < c4) {
                solve_tetrahedra(m, kTetraChunk * x, min(kTetraChunk, n4 - kTetraChunk * x), tol_sq, opt.max_iterations,
                                 E, hits, o.status);
                continue;
            }
            x -= c4;
            const int k = x < c3 ? 1 : (x < c3 + c2 ? 2 : 3);
            const int i = 32 * (k == 1 ? x : (k == 2 ? x - c3 : x - c3 - c2)) + ln;
            if (i < (k == 1 ? n3 : (k == 2 ? n2 : n1))) {
                const int s = m.solve[k * S + i];
                const unsigned mt = m.meta[s];
                d3 r = m.y(mt, 0, s);
                int set = 1;
                if (k == 1)
                    r = flat_triangle(r, m.y(mt, 1, s), m.y(mt, 2, s), E, set);
                else if (k == 2)
                    r = cp_line(r, m.y(mt, 1, s), E, set);
                const double l = dot(r, r);
                put_hit(m, s, finish_step(m, s, lt_sq(l, m.prev[s]), r, l, set, tol_sq, opt.max_iterations, E), hits,
                        o.status);
            }
        }
        __syncthreads();
    }
}

}  // namespace pool
}  // namespace d3d
