// epa_warp.cu -- mixed-precision EPA, the lanes of a warp on a pair.
//
// The search is the mixed EPA of epa_mixed.cu (FP32 polytope search on the
// FP32 mirror, validation with an FP64 fallback); this file lays it out for
// the GPU.  Each pair's polytope lives in shared memory and the lanes share
// the work of every expansion (epa.py:59-74).  k_epa_segments gives a pair 8,
// 16 or 32 lanes of a warp (FP32, up to 255 face slots), k_epa_warp a whole
// warp (FP64, and FP32 with more slots):
//
//   closest face      lanes scan strided face slots, warp min-reduction
//   support           the two colliders on the two half warps; box / hull
//                     argmax split across a half warp's lanes (first
//                     maximum, as np.argmax)
//   visible faces     breadth-first search from the closest face over the
//                     face adjacency with the reference's visibility test
//                     (epa.py:157-165)
//   horizon           edges of visible faces whose neighbour is not visible,
//                     gathered by a warp prefix sum (epa.py:167-187)
//   validation        every horizon vertex starts and ends exactly one edge,
//                     and the edges form one loop (pointer jumping): the
//                     visible faces are a disk, so the new faces close the
//                     surface again
//   new faces         one per horizon edge, in the slots the visible faces
//                     freed (then fresh slots), with their adjacency set from
//                     the loop order (epa.py:126-146)
//
// Faces keep their three vertex ids, unit normal and offset, and the ids of
// the faces across their three edges; winding is outward by construction, as
// in epa_mixed.cu.  A pair whose polytope fails validation (degenerate face,
// horizon not one loop, more horizon edges than max_loose_edges) goes to the
// fallback list.  The converged face is refined along its FP32 normal with
// FP64 supports in a second pass, the supports listed by type (k_epa_refine).
//
// The same search is instantiated with an FP64 polytope and exact FP64
// supports.  It takes the FP32 search's fallback pairs: the plane tests
// behind a pinched horizon are FP32 noise on nearly coplanar faces, which
// FP64 resolves.  Its own fallback pairs go to the serial FP64 EPA (the
// reference's arithmetic).  Compiled with -fmad=true.
#define D3D_FP_COMPARES  // see d3d_device.cuh
#include "capi_util.h"
#include "epa_mixed.cuh"
#include "epa_mixed.h"
#include "persist.cuh"
#include "scratch.h"

namespace {

using namespace d3d;

constexpr unsigned kFull = 0xffffffffu;
constexpr unsigned kDead = 0xffffffffu;  // vertex word of a free face slot

// xyz + w of the polytope's precision (16-byte aligned)
template <typename T>
struct alignas(16) Q4 {
    T x, y, z, w;
};

template <typename T>
__device__ __forceinline__ Q4<T> q4(T x, T y, T z, T w) {
    return Q4<T>{x, y, z, w};
}

template <typename T>
__device__ __forceinline__ T eps_of();
template <>
__device__ __forceinline__ float eps_of<float>() { return FLT_EPSILON; }
template <>
__device__ __forceinline__ double eps_of<double>() { return DBL_EPSILON; }

// Storage bounds of one polytope.  The search adds one vertex per iteration
// (nv <= max_iterations + 4) and keeps a closed triangulated surface (the
// visible faces are validated to be a disk), so its live faces number
// 2 V - 4 <= 2 nv - 4 for its V <= nv vertices in use (Euler), and a horizon
// loop visits distinct vertices (ne <= nv).  The face slots and horizon
// edges are bounded by those numbers as well as by max_faces and
// max_loose_edges; the search checks both bounds before it writes.
__host__ __device__ inline int vertex_cap(const d3d_epa_options& o) { return o.max_iterations + 4; }
__host__ __device__ inline int face_cap(const d3d_epa_options& o) {
    const int euler = 2 * vertex_cap(o) - 4;
    return o.max_faces < euler ? o.max_faces : euler;
}
__host__ __device__ inline int edge_cap(const d3d_epa_options& o) {
    const int e = o.max_loose_edges < vertex_cap(o) ? o.max_loose_edges : vertex_cap(o);
    return e > 0 ? e : 1;
}

// Byte offsets of one warp's polytope in shared memory.
struct Layout {
    int vy, fn, fv, adj, hz, freel, vis, se, ee, bytes;
};

template <typename T>
__host__ __device__ inline Layout layout_for(const d3d_epa_options& o) {
    const int nv = vertex_cap(o), F = face_cap(o), E = edge_cap(o);
    const int q = (int)sizeof(Q4<T>);
    Layout L;
    int p = 0;
    L.vy = p;
    p += q * nv;
    L.fn = p;
    p += q * F;
    L.adj = p;
    p += 8 * F;
    L.hz = p;
    p += 8 * E;
    L.fv = p;
    p += 4 * F;
    L.vis = p;
    p += 4 * F;
    L.freel = p;
    p += 2 * F;
    L.se = p;
    p += nv;
    L.ee = p;
    p += nv;
    L.bytes = (p + 15) & ~15;
    return L;
}

template <typename T>
struct Poly {
    Q4<T>* vy;             // vertex y.xyz
    Q4<T>* fn;             // unit normal .xyz, w = offset n . y_a
    ushort4* adj;          // faces across edges (a,b), (b,c), (c,a)
    int2* hz;              // horizon edge e: x = a | b << 8 | k << 16 (edge k of g faces it), y = g
    unsigned* fv;          // a | b << 8 | c << 16, kDead for a free slot
    unsigned short* freel; // free face slots (stack)
    int* vis;              // iteration stamp of the faces found visible
    unsigned char* se;     // horizon edge that starts at vertex v
    unsigned char* ee;     // horizon edge that ends at vertex v
};

template <typename T>
__device__ __forceinline__ Poly<T> poly_at(unsigned char* base, const Layout& L) {
    Poly<T> P;
    P.vy = reinterpret_cast<Q4<T>*>(base + L.vy);
    P.fn = reinterpret_cast<Q4<T>*>(base + L.fn);
    P.adj = reinterpret_cast<ushort4*>(base + L.adj);
    P.hz = reinterpret_cast<int2*>(base + L.hz);
    P.fv = reinterpret_cast<unsigned*>(base + L.fv);
    P.freel = reinterpret_cast<unsigned short*>(base + L.freel);
    P.vis = reinterpret_cast<int*>(base + L.vis);
    P.se = base + L.se;
    P.ee = base + L.ee;
    return P;
}

__device__ __forceinline__ int lane_id() { return threadIdx.x & 31; }

template <typename T>
__device__ __forceinline__ V3<T> yv(const Poly<T>& P, int v) {
    const Q4<T> a = P.vy[v];
    return mk(a.x, a.y, a.z);
}

// Index of the first maximum of V . d over a polytope's vertices, the 16
// lanes of a half warp (mask hm) taking every 16th vertex (same products as
// hull_argmax, same winner).
template <typename T>
__device__ __forceinline__ int half_argmax(const T* verts, int off, int nv, V3<T> d, unsigned hm) {
    T best = T(0);
    int bi = -1;
    for (int k = lane_id() & 15; k < nv; k += 16) {
        const V3<T> v = load_vertex(verts, off + k);
        const T s = dot102(v.x, v.y, v.z, d.x, d.y, d.z);
        if (bi < 0 || s > best) {
            best = s;
            bi = k;
        }
    }
#pragma unroll
    for (int m = 8; m; m >>= 1) {
        const T ob = __shfl_xor_sync(hm, best, m);
        const int oi = __shfl_xor_sync(hm, bi, m);
        if (oi >= 0 && (bi < 0 || ob > best || (ob == best && oi < bi))) {
            best = ob;
            bi = oi;
        }
    }
    return bi;
}

// The FP32 instance with two warp reductions on order-preserving keys: the
// largest product, then the lowest index holding it (-0 counts as +0; a NaN
// product loses to every number).
template <>
__device__ __forceinline__ int half_argmax<float>(const float* verts, int off, int nv, f3 d, unsigned hm) {
    unsigned best = 0u;
    int bi = 0x7fffffff;
    bool any = false;
    for (int k = lane_id() & 15; k < nv; k += 16) {
        const f3 v = load_vertex(verts, off + k);
        const float x = dot102(v.x, v.y, v.z, d.x, d.y, d.z);
        const unsigned u = x == 0.f ? 0u : __float_as_uint(x);
        const unsigned key = x != x ? 0u : ((u & 0x80000000u) ? ~u : (u | 0x80000000u));
        if (!any || key > best) {
            best = key;
            bi = k;
            any = true;
        }
    }
    const unsigned m = __reduce_max_sync(hm, any ? best : 0u);
    return (int)__reduce_min_sync(hm, (any && best == m) ? (unsigned)bi : 0xffffffffu);
}

__device__ __forceinline__ unsigned half_mask() { return (lane_id() & 16) ? 0xffff0000u : 0x0000ffffu; }

// FastSupport, the sphere's roundings written out: x and y fused, z only
// in the kernels for stores with meshes (left to the compiler they depend on
// the code around).
template <bool MESH>
__device__ __forceinline__ f3 search_support(const Col<float>& c, const d3d_store& st, f3 d) {
    if (c.type != D3D_SPHERE) return FastSupportT<MESH>::eval(c, st, d);
    const f3 ctr = mk(c.t[0], c.t[1], c.t[2]);
    const float n2 = dot(d, d);
    const float f = c.p[0] * rsqrtf(n2);
    const float z = MESH ? fmaf(d.z, f, ctr.z) : __fadd_rn(ctr.z, __fmul_rn(d.z, f));
    return margin_fast(st, c,
                       n2 == 0.f ? ctr + mk(0.f, 0.f, c.p[0]) : mk(fmaf(d.x, f, ctr.x), fmaf(d.y, f, ctr.y), z), d);
}

// w = s_a(d) - s_b(-d) in FP32: the lower half warp evaluates collider a, the
// upper half collider b, together; every lane returns w.
template <bool MESH>
__device__ __forceinline__ f3 minkowski32(const d3d_store& st, int a, int b, f3 d) {
    const bool up = lane_id() & 16;
    Col<float> c;
    load_col(st, up ? b : a, c);
    const f3 dd = up ? -d : d;
    f3 s;
    if (c.type == D3D_BOX || c.type == D3D_HULL) {
        if (c.nv < 1)
            s = mk(NAN, NAN, NAN);
        else
            s = margin_fast(st, c, load_vertex(st.verts32, c.off + (c.nv == 1 ? 0 : half_argmax(st.verts32, c.off, c.nv, dd, half_mask()))), dd);
    } else {
        s = search_support<MESH>(c, st, dd);
    }
    const f3 o = mk(__shfl_xor_sync(kFull, s.x, 16), __shfl_xor_sync(kFull, s.y, 16), __shfl_xor_sync(kFull, s.z, 16));
    return up ? o - s : s - o;
}

// w in FP64 with the reference's supports (the polytope argmax in FP64), for
// the FP64 polytope.
__device__ __forceinline__ d3 minkowski64_exact(const d3d_store& st, int a, int b, d3 d) {
    const bool up = lane_id() & 16;
    Col<double> c;
    load_col(st, up ? b : a, c);
    const d3 dd = up ? -d : d;
    d3 s;
    if (c.type == D3D_BOX || c.type == D3D_HULL) {
        if (c.nv < 1)
            s = mk(double(NAN), double(NAN), double(NAN));
        else
            s = add_margin(c, load_vertex(st.verts64, c.off + (c.nv == 1 ? 0 : half_argmax(st.verts64, c.off, c.nv, dd, half_mask()))), dd);
    } else {
        s = support(c, st, dd);
    }
    const d3 o = mk(__shfl_xor_sync(kFull, s.x, 16), __shfl_xor_sync(kFull, s.y, 16), __shfl_xor_sync(kFull, s.z, 16));
    return up ? o - s : s - o;
}

// The polytope's precision: FP32 search on the FP32 mirror, or FP64 with the
// reference's supports.
template <bool MESH>
__device__ __forceinline__ f3 minkowski_of(const d3d_store& st, int a, int b, f3 d);
template <bool MESH>
__device__ __forceinline__ d3 minkowski_of(const d3d_store& st, int a, int b, d3 d) {
    return minkowski64_exact(st, a, b, d);
}

// exclusive prefix sum over lanes
__device__ __forceinline__ int warp_excl(int x) {
    int s = x;
#pragma unroll
    for (int m = 1; m < 32; m <<= 1) {
        const int t = __shfl_up_sync(kFull, s, m);
        if (lane_id() >= m) s += t;
    }
    return s - x;
}

template <bool MESH>
__device__ __forceinline__ f3 minkowski_of(const d3d_store& st, int a, int b, f3 d) {
    return minkowski32<MESH>(st, a, b, d);
}

// unit normal and offset of face (a, b, c); false if degenerate
template <typename T>
__device__ __forceinline__ bool plane_of(const Poly<T>& P, int a, int b, int c, Q4<T>& out) {
    const V3<T> ya = yv(P, a), yb = yv(P, b), yc = yv(P, c);
    V3<T> n = cross(yb - ya, yc - ya);
    const T l = sqrt_t(dot(n, n));
    if (!(l > T(0))) return false;
    n = n * (T(1) / l);
    out = q4(n.x, n.y, n.z, dot(ya, n));
    return true;
}

__device__ __forceinline__ unsigned pack3(int a, int b, int c) { return (unsigned)a | ((unsigned)b << 8) | ((unsigned)c << 16); }
__device__ __forceinline__ int vid(unsigned w, int j) { return (int)((w >> (8 * j)) & 0xffu); }
__device__ __forceinline__ int adj_at(ushort4 g, int j) { return j == 0 ? g.x : (j == 1 ? g.y : g.z); }

// Closest live face: (offset, slot), ties to the lower slot.
template <typename T>
__device__ __forceinline__ int closest_face(const Poly<T>& P, int nslots) {
    T bd = T(0);
    int bs = -1;
    for (int f = lane_id(); f < nslots; f += 32) {
        if (P.fv[f] == kDead) continue;
        const T d = P.fn[f].w;
        if (bs < 0 || d < bd) {
            bd = d;
            bs = f;
        }
    }
#pragma unroll
    for (int m = 16; m; m >>= 1) {
        const T od = __shfl_xor_sync(kFull, bd, m);
        const int os = __shfl_xor_sync(kFull, bs, m);
        if (os >= 0 && (bs < 0 || od < bd || (od == bd && os < bs))) {
            bd = od;
            bs = os;
        }
    }
    return bs;
}

// The same for the FP32 polytope with two warp reductions (REDUX) on
// order-preserving 32-bit keys of the offsets instead of five shuffle rounds:
// the smallest key, then the lowest slot holding it.  (-0 counts as +0; a NaN
// offset loses to every number.)
template <>
__device__ __forceinline__ int closest_face<float>(const Poly<float>& P, int nslots) {
    unsigned best = 0xffffffffu;
    int bs = 0x7fffffff;
    for (int f = lane_id(); f < nslots; f += 32) {
        if (P.fv[f] == kDead) continue;
        const float d = P.fn[f].w;
        const unsigned u = d == 0.f ? 0u : __float_as_uint(d);
        const unsigned key = d != d ? 0xfffffffeu : ((u & 0x80000000u) ? ~u : (u | 0x80000000u));
        if (key < best) {
            best = key;
            bs = f;
        }
    }
    const unsigned m = __reduce_min_sync(kFull, best);
    if (m == 0xffffffffu) return -1;
    return (int)__reduce_min_sync(kFull, best == m ? (unsigned)bs : 0xffffffffu);
}

// Outcome of the FP32 search for one pair.
struct Search {
    int status;   // a D3D status, or kEpaFallback
    int closest;  // face slot refined for OK / NOT_CONVERGED
    int nslots;
    int live;
};

// The expanding-polytope search for one pair in the polytope's precision T
// (uniform across the warp).
template <typename T, bool MESH>
__device__ Search search_pair(const Poly<T>& P, const d3d_store& st, int a, int b, const double* simplex,
                              const d3d_epa_options& o) {
    const int ln = lane_id();
    Search R{kEpaFallback, 0, 0, 0};
    // starting tetrahedron: the FP64 simplex (rounded to T)
    T scale = T(0);
    if (ln < 4) {
        const V3<T> y = mk((T)simplex[3 * ln], (T)simplex[3 * ln + 1], (T)simplex[3 * ln + 2]);
        P.vy[ln] = q4(y.x, y.y, y.z, T(0));
        scale = sqrt_t(dot(y, y));
    }
#pragma unroll
    for (int m = 16; m; m >>= 1) scale = maxf2(scale, (T)__shfl_xor_sync(kFull, scale, m));
    __syncwarp();
    // faces ABC, ACD, ADB, BDC, each wound away from the vertex it leaves out
    bool bad = false;
    if (ln < 4) {
        const int t = ln == 0 ? 0x3210 : (ln == 1 ? 0x1320 : (ln == 2 ? 0x2130 : 0x0231));
        int fa = t & 15, fb = (t >> 4) & 15;
        const int fc = (t >> 8) & 15, fd = (t >> 12) & 15;
        Q4<T> pl;
        if (!plane_of(P, fa, fb, fc, pl)) {
            bad = true;
        } else {
            const V3<T> yd = yv(P, fd) - yv(P, fa);
            if (pl.x * yd.x + pl.y * yd.y + pl.z * yd.z > T(0)) {
                const int s = fa;
                fa = fb;
                fb = s;
                pl = q4(-pl.x, -pl.y, -pl.z, -pl.w);
            }
            P.fv[ln] = pack3(fa, fb, fc);
            P.fn[ln] = pl;
            P.vis[ln] = 0;
        }
    }
    if (__any_sync(kFull, bad)) return R;
    __syncwarp();
    // adjacency of the tetrahedron: the face across (u, v) holds (v, u)
    if (ln < 12) {
        const int f = ln / 3, j = ln % 3;
        const unsigned w = P.fv[f];
        const int u = vid(w, j), v = vid(w, (j + 1) % 3);
        int g = -1;
        for (int h = 0; h < 4; ++h) {
            if (h == f) continue;
            const unsigned x = P.fv[h];
            for (int i = 0; i < 3; ++i)
                if (vid(x, i) == v && vid(x, (i + 1) % 3) == u) g = h;
        }
        if (g < 0) {
            bad = true;
        } else {
            unsigned short* ap = reinterpret_cast<unsigned short*>(&P.adj[f]);
            ap[j] = (unsigned short)g;
        }
    }
    if (__any_sync(kFull, bad)) return R;
    __syncwarp();

    const T vis_eps = (T)o.epsilon;  // the reference's visibility test
    int nslots = 4, nfree = 0, live = 4, nv = 4, it = 0;
    while (true) {
        const int cf = closest_face(P, nslots);
        R.closest = cf;
        R.nslots = nslots;
        R.live = live;
        if (cf < 0) {
            R.status = D3D_STATUS_EPA_DEGENERATE;
            return R;
        }
        if (it >= o.max_iterations) {
            R.status = D3D_STATUS_EPA_NOT_CONVERGED;
            return R;
        }
        ++it;
        const Q4<T> cn = P.fn[cf];
        const V3<T> sd = mk(cn.x, cn.y, cn.z);
        const V3<T> w = minkowski_of<MESH>(st, a, b, sd);
        scale = maxf2(scale, sqrt_t(dot(w, w)));
        const T eps = maxf2((T)o.epsilon, T(kSearchUlps) * eps_of<T>() * scale);
        if (dot(w, sd) - cn.w < eps) {
            R.status = D3D_STATUS_OK;
            return R;
        }
        if (nv >= o.max_iterations + 4) {
            R.status = D3D_STATUS_EPA_NOT_CONVERGED;
            return R;
        }
        const int vn = nv++;
        const int stamp = it;
        // Faces that see w: breadth first from the closest face over the
        // adjacency.  The visible faces are listed where they are about to
        // go, on the free list above its current top.
        unsigned short* const vl = P.freel + nfree;
        if (ln == 0) {
            P.vy[vn] = q4(w.x, w.y, w.z, T(0));
            P.vis[cf] = stamp;
            vl[0] = (unsigned short)cf;
        }
        __syncwarp();
        int head = 0, nvis = 1;
        while (head < nvis) {
            const int nc = 3 * (nvis - head);
            int added = 0;
            for (int i0 = 0; i0 < nc; i0 += 32) {
                const int i = i0 + ln;
                bool take = false;
                int g = 0;
                if (i < nc) {
                    g = adj_at(P.adj[vl[head + i / 3]], i % 3);
                    if (P.vis[g] != stamp) {
                        // w above the face's plane: n . w - n . y_a (the offset kept with the normal)
                        const Q4<T> pl = P.fn[g];
                        if (dot(mk(pl.x, pl.y, pl.z), w) - pl.w > vis_eps)
                            take = atomicExch(&P.vis[g], stamp) != stamp;
                    }
                }
                const unsigned m = __ballot_sync(kFull, take);
                if (take) vl[nvis + added + __popc(m & ((1u << ln) - 1u))] = (unsigned short)g;
                added += __popc(m);
            }
            __syncwarp();
            head = nvis;
            nvis += added;
        }
        // horizon: edges of visible faces whose neighbour is not visible (a
        // single visible face: its own three edges, in order)
        int ne = 3;
        if (nvis == 1) {
            if (3 > o.max_loose_edges) return R;
            if (ln < 3) {
                const unsigned fw = P.fv[cf];
                const int h = adj_at(P.adj[cf], ln);
                const ushort4 gh = P.adj[h];
                const int k = gh.x == cf ? 0 : (gh.y == cf ? 1 : 2);
                P.hz[ln] = make_int2(vid(fw, ln) | (vid(fw, (ln + 1) % 3) << 8) | (k << 16), h);
            }
        } else {
            int ne_l = 0;
            for (int i = ln; i < 3 * nvis; i += 32) ne_l += P.vis[adj_at(P.adj[vl[i / 3]], i % 3)] != stamp;
            int eb = warp_excl(ne_l);
            ne = __shfl_sync(kFull, eb + ne_l, 31);
            // more than edge_cap(o) < max_loose_edges edges: not one loop
            if (ne > o.max_loose_edges || ne > edge_cap(o) || ne < 3) return R;
            for (int i = ln; i < 3 * nvis; i += 32) {
                const int f = vl[i / 3], j = i % 3;
                const int h = adj_at(P.adj[f], j);
                if (P.vis[h] == stamp) continue;
                const unsigned fw = P.fv[f];
                const ushort4 gh = P.adj[h];
                const int k = gh.x == f ? 0 : (gh.y == f ? 1 : 2);
                P.hz[eb++] = make_int2(vid(fw, j) | (vid(fw, (j + 1) % 3) << 8) | (k << 16), h);
            }
        }
        __syncwarp();
        for (int i = ln; i < nvis; i += 32) P.fv[vl[i]] = kDead;
        __syncwarp();
        // The horizon must be one loop.  A single visible face gives its own
        // three edges, in order.  Otherwise: unique start and end per vertex ...
        if (nvis > 1) {
            for (int e = ln; e < ne; e += 32) {
                const int x = P.hz[e].x;
                P.se[x & 0xff] = (unsigned char)e;
                P.ee[(x >> 8) & 0xff] = (unsigned char)e;
            }
            __syncwarp();
            bool ok = true;
            for (int e = ln; e < ne; e += 32) {
                const int x = P.hz[e].x;
                const int nx = P.se[(x >> 8) & 0xff];
                ok &= P.se[x & 0xff] == e && P.ee[(x >> 8) & 0xff] == e && nx < ne &&
                      (P.hz[nx].x & 0xff) == ((x >> 8) & 0xff);
            }
            if (!__all_sync(kFull, ok)) return R;
            // ... and following next(e) from edge 0 visits every edge once
            if (ne <= 32) {
                int nxt = ln < ne ? P.se[(P.hz[ln].x >> 8) & 0xff] : ln;
                int lab = ln < ne ? ln : 0;
#pragma unroll
                for (int r = 0; r < 5; ++r) {
                    lab = min(lab, __shfl_sync(kFull, lab, nxt));
                    nxt = __shfl_sync(kFull, nxt, nxt);
                }
                ok = lab == 0;
            } else {
                int steps = 0, cur = 0;
                if (ln == 0) {
                    do {
                        cur = P.se[(P.hz[cur].x >> 8) & 0xff];
                        ++steps;
                    } while (cur != 0 && steps <= ne);
                }
                ok = __shfl_sync(kFull, steps == ne && cur == 0, 0);
            }
            if (!__all_sync(kFull, ok)) return R;
        }
        const int nlive = live - nvis + ne;
        if (nlive > o.max_faces) {
            R.status = D3D_STATUS_EPA_FACE_OVERFLOW;
            R.live = live - nvis;
            return R;
        }
        // new faces (a, b, w): slots from the top of the free list, then fresh
        const int nft = nfree + nvis;
        if (ne > nft && nslots + (ne - nft) > face_cap(o)) return R;  // beyond the Euler bound: never for a closed surface
        for (int e = ln; e < ne; e += 32) {
            const int2 h = P.hz[e];
            const int ea = h.x & 0xff, eb2 = (h.x >> 8) & 0xff, k = (h.x >> 16) & 3;
            const int nx = nvis == 1 ? (e == 2 ? 0 : e + 1) : P.se[eb2];
            const int pv = nvis == 1 ? (e == 0 ? 2 : e - 1) : P.ee[ea];
            const int s = e < nft ? P.freel[nft - 1 - e] : nslots + (e - nft);
            const int sn = nx < nft ? P.freel[nft - 1 - nx] : nslots + (nx - nft);
            const int sp = pv < nft ? P.freel[nft - 1 - pv] : nslots + (pv - nft);
            Q4<T> pl;
            if (!plane_of(P, ea, eb2, vn, pl)) bad = true;
            P.fn[s] = pl;
            P.fv[s] = pack3(ea, eb2, vn);
            P.adj[s] = make_ushort4((unsigned short)h.y, (unsigned short)sn, (unsigned short)sp, 0);
            P.vis[s] = 0;
            reinterpret_cast<unsigned short*>(&P.adj[h.y])[k] = (unsigned short)s;
        }
        if (__any_sync(kFull, bad)) return R;
        nslots = ne > nft ? nslots + (ne - nft) : nslots;
        nfree = ne < nft ? nft - ne : 0;
        live = nlive;
        __syncwarp();
    }
}

// Resident warps per SM the register budget is set for: the FP32 search runs
// 32 (64 registers, a few spilled: latency hiding outweighs the spills), the
// FP64 search, which takes few pairs, 16.
template <typename T>
constexpr int kWarpsPerSm = sizeof(T) == 4 ? 32 : 16;

template <typename T, int WARPS, bool MESH>
__global__ void __launch_bounds__(32 * WARPS, kWarpsPerSm<T> / WARPS) k_epa_warp(d3d_store st, const int32_t* __restrict__ i1,
                                                          const int32_t* __restrict__ i2,
                                                          const int32_t* __restrict__ list, int64_t n,
                                                          const unsigned long long* __restrict__ n_dev,
                                                          unsigned long long* __restrict__ cursor,
                                                          const double* __restrict__ simplex, d3d_epa_options o,
                                                          double* __restrict__ mtv, int8_t* __restrict__ status,
                                                          int32_t* __restrict__ n_faces, double* __restrict__ faces,
                                                          int32_t* __restrict__ fallback,
                                                          unsigned long long* __restrict__ n_fallback,
                                                          int32_t* __restrict__ refine,
                                                          unsigned long long* __restrict__ n_refine) {
    extern __shared__ __align__(16) unsigned char smem[];
    const Layout L = layout_for<T>(o);
    const Poly<T> P = poly_at<T>(smem + (threadIdx.x >> 5) * L.bytes, L);
    const int ln = lane_id();
    if (n_dev) n = (int64_t)*n_dev;
    while (true) {
        long long slot = 0;
        if (ln == 0) slot = (long long)atomicAdd(cursor, 1ull);
        slot = __shfl_sync(kFull, slot, 0);
        if (slot >= n) break;
        const int64_t k = list ? list[slot] : slot;
        const int a = i1[k], b = i2[k];
        if (!pair_ok(st, a, b)) {  // the same for every lane
            if (ln == 0) epa_store_bad_index(mtv, status, n_faces, k);
            __syncwarp();
            continue;
        }
        const double* sx = simplex + 12 * k;
        const Search R = search_pair<T, MESH>(P, st, a, b, sx, o);
        if (R.status == kEpaFallback) {
            if (ln == 0) fallback[atomicAdd(n_fallback, 1ull)] = (int32_t)k;
            __syncwarp();
            continue;
        }
        d3 m = mk(double(NAN), double(NAN), double(NAN));
        const bool ended = R.status == D3D_STATUS_OK || R.status == D3D_STATUS_EPA_NOT_CONVERGED;
        if (ended) {
            const Q4<T> q = P.fn[R.closest];
            m = mk((double)q.x, (double)q.y, (double)q.z);
            if (sizeof(T) == 8) {
                // mtv = n (n . w(n)), the reference's expression at convergence (epa.py:69)
                const d3 w = minkowski64_exact(st, a, b, m);
                m = m * dot(w, m);
            }  // FP32: the face's normal now, the FP64 depth along it in k_epa_refine
        }
        const int nf = R.status == D3D_STATUS_EPA_DEGENERATE ? 0 : R.live;
        if (ln == 0) {
            mtv[3 * k] = m.x;
            mtv[3 * k + 1] = m.y;
            mtv[3 * k + 2] = m.z;
            status[k] = (int8_t)R.status;
            n_faces[k] = nf;
            if (sizeof(T) == 4 && ended) refine[atomicAdd(n_refine, 1ull)] = (int32_t)k;
        }
        if (faces && nf > 0) {
            // live faces in slot order: three vertices and the normal
            double* out = faces + k * 12 * (int64_t)o.max_faces;
            int base = 0;
            for (int f0 = 0; f0 < R.nslots; f0 += 32) {
                const int f = f0 + ln;
                const bool live = f < R.nslots && P.fv[f] != kDead;
                const unsigned mask = __ballot_sync(kFull, live);
                if (live) {
                    double* q = out + 12 * (base + __popc(mask & ((1u << ln) - 1u)));
                    const unsigned fw = P.fv[f];
#pragma unroll
                    for (int j = 0; j < 3; ++j) {
                        const Q4<T> yy = P.vy[vid(fw, j)];
                        q[3 * j] = yy.x;
                        q[3 * j + 1] = yy.y;
                        q[3 * j + 2] = yy.z;
                    }
                    const Q4<T> pl = P.fn[f];
                    q[9] = pl.x;
                    q[10] = pl.y;
                    q[11] = pl.z;
                }
                base += __popc(mask);
            }
        }
        __syncwarp();
    }
}

// ---- the FP32 search, several pairs to a warp
//
// The search above spends its issue slots on steps that are alike for every
// expansion and busy few lanes (an expansion sees ~4 faces and adds ~6): one
// warp per pair kept 71 % of the issue slots busy.  Here a segment of W lanes
// takes a pair and the segments of a warp step together, an ended one fetching
// its next pair, so that the steps are issued once for 32 / W pairs.  Control
// flow is the warp's, collectives are full-warp and a segment takes its own
// part.  Three passes go: the horizon is collected by the flood fill itself
// (an edge whose far face does not see w), faces carry the order-preserving
// key of their offset, which the closest-face scan reads and which marks free
// slots, and a face's visited flag rides in its adjacency word.  A lane keeps
// its collider in registers.  The list comes in the type-sorted order of GJK
// where there is one and a warp claims 4 slots of it at a time, so that its
// segments run through few kinds of support.  Vertex, face and edge order,
// and with them every tie, are those of the search above.  Face ids are bytes:
// polytopes of up to 255 face slots.  Before -> now: 310,000 pairs, 256 faces
// 4,820 -> 3,360 us; scene of 131,072, 64 faces 635 -> 430 us; robot batch
// 200 -> 106 us; 900 pairs 116 -> 101 us.  1.18e9 -> 7.6e8 warp instructions
// for 77,500 pairs before the list was sorted and the passes merged.
constexpr int kSegChunk = 4;  // list slots a warp claims at a time

// Resident warps per SM the register budget is set for.
__host__ __device__ constexpr int seg_warps(int w) { return w == 8 ? 20 : 24; }

template <int W>
struct Seg {
    static_assert(W == 8 || W == 16 || W == 32, "8, 16 or 32 lanes");
    static constexpr int kPairs = 32 / W;
    static constexpr unsigned kBits = W == 32 ? kFull : (1u << (W & 31)) - 1u;
    static __device__ __forceinline__ int lane() { return lane_id() & (W - 1); }
    static __device__ __forceinline__ int index() { return lane_id() / W; }
    // the segment's lanes, and those below the caller
    static __device__ __forceinline__ unsigned own() { return kBits << (lane_id() & (32 - W)); }
    static __device__ __forceinline__ unsigned below() { return own() & ((1u << lane_id()) - 1u); }
    template <int N>
    static __device__ __forceinline__ unsigned min_over(unsigned x) {
        if (N == 32) return __reduce_min_sync(kFull, x);
#pragma unroll
        for (int m = N / 2; m; m >>= 1) x = min(x, __shfl_xor_sync(kFull, x, m));
        return x;
    }
};

// Order-preserving key of an offset (-0 counts as +0, a NaN is above every
// number), and back.
constexpr unsigned kFreeKey = 0xffffffffu;

__device__ __forceinline__ unsigned offset_key(float d) {
    const unsigned u = d == 0.f ? 0u : __float_as_uint(d);
    return d != d ? 0xfffffffeu : ((u & 0x80000000u) ? ~u : (u | 0x80000000u));
}
__device__ __forceinline__ float key_offset(unsigned k) {
    return __uint_as_float((k & 0x80000000u) ? k ^ 0x80000000u : ~k);
}

constexpr unsigned kSeen = 0x80000000u;  // flag of an adjacency word

// One pair's polytope: vertex y.xyz with horizon word e in the unused w of
// vertex e, face normal .xyz with the offset's key in w.
struct BytePoly {
    float4* vy;
    float4* fn;
    unsigned* adj;         // faces across edges (a,b), (b,c), (c,a), a byte each, and kSeen
    unsigned* fv;          // a | b << 8 | c << 16
    unsigned char* freel;  // free face slots (stack)
    unsigned char* se;
    unsigned char* ee;
    __device__ __forceinline__ unsigned hz(int e) const { return __float_as_uint(vy[e].w); }
    __device__ __forceinline__ f3 y(int v) const { return mk(vy[v].x, vy[v].y, vy[v].z); }
};

__host__ __device__ inline int byte_poly_bytes(const d3d_epa_options& o) {
    const int nv = vertex_cap(o), F = face_cap(o);
    return (16 * nv + 25 * F + 2 * nv + 15) & ~15;
}

// unit normal and offset key of face (a, b, c); false if degenerate
__device__ __forceinline__ bool byte_plane(const BytePoly& P, int a, int b, int c, float4& out, float& off) {
    const f3 ya = P.y(a), yb = P.y(b), yc = P.y(c);
    f3 n = cross(yb - ya, yc - ya);
    const float l = sqrt_t(dot(n, n));
    if (!(l > 0.f)) return false;
    n = n * (1.f / l);
    off = dot(ya, n);
    out = make_float4(n.x, n.y, n.z, 0.f);
    return true;
}

template <int W, int WARPS, bool MESH>
__global__ void __launch_bounds__(32 * WARPS, seg_warps(W) / WARPS) k_epa_segments(
    d3d_store st, const int32_t* __restrict__ i1, const int32_t* __restrict__ i2, const int32_t* __restrict__ list,
    int64_t n, const unsigned long long* __restrict__ n_dev, unsigned long long* __restrict__ cursor,
    const double* __restrict__ simplex, d3d_epa_options o, double* __restrict__ mtv, int8_t* __restrict__ status,
    int32_t* __restrict__ n_faces, double* __restrict__ faces, int32_t* __restrict__ fallback,
    unsigned long long* __restrict__ n_fallback, int32_t* __restrict__ refine,
    unsigned long long* __restrict__ n_refine, int64_t lo, int64_t hi) {
    using S = Seg<W>;
    static_assert(kSegChunk >= S::kPairs, "a claim serves every segment that asks");
    constexpr int H = W / 2;        // lanes per collider
    constexpr int kRun = -1000;     // no outcome yet
    extern __shared__ __align__(16) unsigned char smem[];
    const int sl = S::lane();
    const unsigned own = S::own(), below = S::below();
    const int cap_v = vertex_cap(o), cap_f = face_cap(o), cap_e = edge_cap(o);
    BytePoly P;
    {
        unsigned char* base = smem + (threadIdx.x / W) * byte_poly_bytes(o);
        P.vy = reinterpret_cast<float4*>(base);
        P.fn = P.vy + cap_v;
        P.adj = reinterpret_cast<unsigned*>(P.fn + cap_f);
        P.fv = P.adj + cap_f;
        P.freel = reinterpret_cast<unsigned char*>(P.fv + cap_f);
        P.se = P.freel + cap_f;
        P.ee = P.se + cap_v;
    }
    if (n_dev) n = (int64_t)*n_dev;
    if (n < lo || n >= hi) return;  // another form's batch
    // a batch of fewer pairs than segments takes warps before segments
    bool done = S::index() > 0 && n <= (int64_t)S::index() * gridDim.x * WARPS;
    bool run = false;
    WarpChunk chunk;
    const long long split = n - 2ll * S::kPairs * WARPS * gridDim.x;
    int64_t k = 0;
    int a = 0, b = 0;
    Col<float> c;  // the lane's collider
    c.type = -1;
    c.nv = 0;
    int nslots = 0, nfree = 0, live = 0, nv = 0, it = 0;
    float scale = 0.f;
    const float vis_eps = (float)o.epsilon;  // the reference's visibility test
    const int mine = sl / 3, j = sl - 3 * mine;  // of W / 3 visible faces and their edges, the lane's
    while (true) {
        // ---- segments without a pair fetch one
        if (__any_sync(kFull, !run && !done)) {
            const bool want = !run && !done;
            long long slot = fetch_slot_chunked(cursor, want && sl == 0, chunk, kFull, kSegChunk, split);
            slot = __shfl_sync(kFull, slot, 0, W);
            bool begin = false;
            if (want) {
                if (slot >= n) {
                    done = true;
                } else {
                    k = list ? list[slot] : slot;
                    a = i1[k];
                    b = i2[k];
                    begin = pair_ok(st, a, b);
                    if (!begin && sl == 0) epa_store_bad_index(mtv, status, n_faces, k);
                }
            }
            if (__all_sync(kFull, done)) break;
            // starting tetrahedron: the FP64 simplex rounded to FP32
            float ys = 0.f;
            if (begin && sl < 4) {
                const double* x = simplex + 12 * k + 3 * sl;
                const f3 y = mk((float)x[0], (float)x[1], (float)x[2]);
                P.vy[sl] = make_float4(y.x, y.y, y.z, 0.f);
                ys = sqrt_t(dot(y, y));
            }
#pragma unroll
            for (int m = W / 2; m; m >>= 1) ys = maxf2(ys, __shfl_xor_sync(kFull, ys, m));
            __syncwarp();
            // faces ABC, ACD, ADB, BDC, each wound away from the vertex it leaves out
            bool bad = false;
            if (begin && sl < 4) {
                const int t = sl == 0 ? 0x3210 : (sl == 1 ? 0x1320 : (sl == 2 ? 0x2130 : 0x0231));
                int fa = t & 15, fb = (t >> 4) & 15;
                const int fc = (t >> 8) & 15, fd = (t >> 12) & 15;
                float4 pl;
                float off;
                if (!byte_plane(P, fa, fb, fc, pl, off)) {
                    bad = true;
                } else {
                    const f3 yd = P.y(fd) - P.y(fa);
                    if (pl.x * yd.x + pl.y * yd.y + pl.z * yd.z > 0.f) {
                        const int s = fa;
                        fa = fb;
                        fb = s;
                        pl = make_float4(-pl.x, -pl.y, -pl.z, 0.f);
                        off = -off;
                    }
                    pl.w = __uint_as_float(offset_key(off));
                    P.fv[sl] = pack3(fa, fb, fc);
                    P.fn[sl] = pl;
                    P.adj[sl] = 0u;
                }
            }
            bad = (__ballot_sync(kFull, bad) & own) != 0;
            __syncwarp();
            // adjacency of the tetrahedron: the face across (u, v) holds (v, u)
            if (begin && !bad) {
                for (int i0 = sl; i0 < 12; i0 += W) {
                    const int f = i0 / 3, j = i0 % 3;
                    const unsigned w = P.fv[f];
                    const int u = vid(w, j), v = vid(w, j == 2 ? 0 : j + 1);
                    int g = -1;
                    for (int h = 0; h < 4; ++h) {
                        if (h == f) continue;
                        const unsigned x = P.fv[h];
                        for (int i = 0; i < 3; ++i)
                            if (vid(x, i) == v && vid(x, (i + 1) % 3) == u) g = h;
                    }
                    if (g < 0)
                        bad = true;
                    else
                        reinterpret_cast<unsigned char*>(P.adj + f)[j] = (unsigned char)g;
                }
            }
            bad = (__ballot_sync(kFull, bad) & own) != 0;
            __syncwarp();
            if (begin) {
                if (bad) {
                    if (sl == 0) fallback[atomicAdd(n_fallback, 1ull)] = (int32_t)k;
                } else {
                    run = true;
                    load_col(st, (sl & H) ? b : a, c);
                    scale = ys;
                    nslots = live = nv = 4;
                    nfree = it = 0;
                }
            }
            if (!__any_sync(kFull, run)) continue;
        }
        // ---- closest face: (offset, slot), ties to the lower slot
        int end = kRun;
        int cf = -1;
        {
            unsigned best = kFreeKey, bs = 0xffffffffu;
            if (run) {
                for (int f = sl; f < nslots; f += W) {
                    const unsigned key = __float_as_uint(P.fn[f].w);
                    if (key < best) {
                        best = key;
                        bs = f;
                    }
                }
            }
            const unsigned m = S::template min_over<W>(best);
            cf = (int)S::template min_over<W>(best == m ? bs : 0xffffffffu);
        }
        if (run) {
            if (cf < 0)
                end = D3D_STATUS_EPA_DEGENERATE;
            else if (it >= o.max_iterations)
                end = D3D_STATUS_EPA_NOT_CONVERGED;
            else
                ++it;
        }
        bool act = run && end == kRun;
        // ---- support: a collider on each half of the segment
        f3 sd = mk(0.f, 0.f, 0.f), w = mk(0.f, 0.f, 0.f);
        float cw = 0.f;
        if (act) {
            const float4 cn = P.fn[cf];
            sd = mk(cn.x, cn.y, cn.z);
            cw = key_offset(__float_as_uint(cn.w));
        }
        {
            const bool up = sl & H;
            const f3 dd = up ? -sd : sd;
            const bool poly = act && (c.type == D3D_BOX || c.type == D3D_HULL);
            int vi = 0;
            if (__any_sync(kFull, poly && c.nv > 1)) {
                // first maximum of V . d, the lanes of the half taking every H-th vertex
                unsigned best = 0u, bi = 0x7fffffffu;
                bool any = false;
                if (poly && c.nv > 1) {
                    for (int q = sl & (H - 1); q < c.nv; q += H) {
                        const f3 v = load_vertex(st.verts32, c.off + q);
                        const float x = dot102(v.x, v.y, v.z, dd.x, dd.y, dd.z);
                        const unsigned u = x == 0.f ? 0u : __float_as_uint(x);
                        const unsigned key = x != x ? 0u : ((u & 0x80000000u) ? ~u : (u | 0x80000000u));
                        if (!any || key > best) {
                            best = key;
                            bi = q;
                            any = true;
                        }
                    }
                }
                const unsigned m = ~S::template min_over<H>(~best);
                bi = S::template min_over<H>(any && best == m ? bi : 0x7fffffffu);
                if (poly && c.nv > 1) vi = (int)bi;
            }
            f3 s = mk(0.f, 0.f, 0.f);
            if (act) {
                if (poly) {
                    if (c.nv < 1)
                        s = mk(NAN, NAN, NAN);
                    else
                        s = margin_fast(st, c, load_vertex(st.verts32, c.off + vi), dd);
                } else {
                    s = search_support<MESH>(c, st, dd);
                }
            }
            __syncwarp();
            const f3 t = mk(__shfl_xor_sync(kFull, s.x, H), __shfl_xor_sync(kFull, s.y, H),
                            __shfl_xor_sync(kFull, s.z, H));
            w = up ? t - s : s - t;
        }
        if (act) {
            scale = maxf2(scale, sqrt_t(dot(w, w)));
            const float eps = maxf2((float)o.epsilon, (float)kSearchUlps * FLT_EPSILON * scale);
            if (dot(w, sd) - cw < eps)
                end = D3D_STATUS_OK;
            else if (nv >= o.max_iterations + 4)
                end = D3D_STATUS_EPA_NOT_CONVERGED;
            act = end == kRun;
        }
        // ---- faces that see w, breadth first from the closest face over the
        // adjacency, and the horizon on the way.  The visible faces are listed
        // where they are about to go, on the free list above its current top.
        unsigned char* const vl = P.freel + nfree;
        const int vn = nv;
        int head = 0, nvis = 0, ne = 0;
        if (act) {
            ++nv;
            nvis = 1;
            if (sl == 0) {
                P.vy[vn] = make_float4(w.x, w.y, w.z, 0.f);
                P.adj[cf] |= kSeen;
                vl[0] = (unsigned char)cf;
            }
        }
        __syncwarp();
        while (__any_sync(kFull, head < nvis)) {
            bool take = false, rim = false;
            int g = 0;
            unsigned word = 0;
            if (sl < W / 3 * 3 && head + mine < nvis) {
                const int f = vl[head + mine];
                g = (P.adj[f] >> (8 * j)) & 0xff;
                const unsigned gw = P.adj[g];
                if (!(gw & kSeen)) {
                    // w above the face's plane: n . w - n . y_a (the offset kept with the normal)
                    const float4 pl = P.fn[g];
                    if (dot(mk(pl.x, pl.y, pl.z), w) - key_offset(__float_as_uint(pl.w)) > vis_eps) {
                        take = !(atomicOr(P.adj + g, kSeen) & kSeen);
                    } else {
                        rim = true;
                        const unsigned fw = P.fv[f];
                        const unsigned e = (gw & 0xff) == f ? 0u : (((gw >> 8) & 0xff) == f ? 1u : 2u);
                        word = vid(fw, j) | (vid(fw, j == 2 ? 0 : j + 1) << 8) | (g << 16) | (e << 24);
                    }
                }
            }
            const unsigned mt = __ballot_sync(kFull, take) & own, mr = __ballot_sync(kFull, rim) & own;
            if (take) vl[nvis + __popc(mt & below)] = (unsigned char)g;
            const int e = ne + __popc(mr & below);
            if (rim && e < cap_e) P.vy[e].w = __uint_as_float(word);
            head = min(head + W / 3, nvis);
            nvis += __popc(mt);
            ne += __popc(mr);
            __syncwarp();
        }
        bool fail = act && (ne > o.max_loose_edges || ne > cap_e || ne < 3);
        const bool wide = act && !fail && 3 * nvis > 32;
        if (__any_sync(kFull, wide)) {
            // many visible faces: the horizon in the order of 32 strided lanes
            int base = 0;
            for (int v0 = 0; v0 < 32; v0 += W) {
                int cnt = 0;
                if (wide)
                    for (int i = v0 + sl; i < 3 * nvis; i += 32)
                        cnt += !(P.adj[(P.adj[vl[i / 3]] >> (8 * (i % 3))) & 0xff] & kSeen);
                int sum = cnt;
#pragma unroll
                for (int m = 1; m < W; m <<= 1) {
                    const int t = __shfl_up_sync(kFull, sum, m, W);
                    if (sl >= m) sum += t;
                }
                int e = base + sum - cnt;
                if (wide)
                    for (int i = v0 + sl; i < 3 * nvis; i += 32) {
                        const int f = vl[i / 3], j = i % 3;
                        const int g = (P.adj[f] >> (8 * j)) & 0xff;
                        const unsigned gw = P.adj[g];
                        if (gw & kSeen) continue;
                        const unsigned fw = P.fv[f];
                        const unsigned x = (gw & 0xff) == f ? 0u : (((gw >> 8) & 0xff) == f ? 1u : 2u);
                        P.vy[e++].w = __uint_as_float(vid(fw, j) | (vid(fw, (j + 1) % 3) << 8) | (g << 16) | (x << 24));
                    }
                base += __shfl_sync(kFull, sum, W - 1, W);
            }
        }
        __syncwarp();
        if (act)
            for (int i = sl; i < nvis; i += W) P.fn[vl[i]].w = __uint_as_float(kFreeKey);
        // ---- the horizon must be one loop.  A single visible face gives its
        // own three edges, in order.  Otherwise: unique start and end per
        // vertex, and following next(e) from edge 0 visits every edge once.
        const bool loop = act && !fail && nvis > 1;
        if (__any_sync(kFull, loop)) {
            const bool many = __any_sync(kFull, loop && ne > W);
            const bool in = loop && sl < ne;
            const unsigned x = in ? P.hz(sl) : 0u;
            const int xa = x & 0xff, xb = (x >> 8) & 0xff;
            if (in) {
                P.se[xa] = (unsigned char)sl;
                P.ee[xb] = (unsigned char)sl;
            }
            if (many && loop)
                for (int e = sl + W; e < ne; e += W) {
                    const unsigned y = P.hz(e);
                    P.se[y & 0xff] = (unsigned char)e;
                    P.ee[(y >> 8) & 0xff] = (unsigned char)e;
                }
            __syncwarp();
            bool ok = true;
            int nxt = sl;
            if (in) {
                nxt = P.se[xb];
                ok = P.se[xa] == sl && P.ee[xb] == sl && nxt < ne && (P.hz(nxt < ne ? nxt : 0) & 0xff) == xb;
            }
            if (many && loop)
                for (int e = sl + W; e < ne; e += W) {
                    const unsigned y = P.hz(e);
                    const unsigned yb = (y >> 8) & 0xff;
                    const int nx = P.se[yb];
                    ok &= P.se[y & 0xff] == e && P.ee[yb] == e && nx < ne && (P.hz(nx < ne ? nx : 0) & 0xff) == yb;
                }
            {
                // the lowest edge on each edge's loop, by pointer jumping
                int lab = in && ne <= W ? sl : 0;
                nxt &= W - 1;
#pragma unroll
                for (int r = 1; r < W; r <<= 1) {
                    lab = min(lab, __shfl_sync(kFull, lab, nxt, W));
                    nxt = __shfl_sync(kFull, nxt, nxt, W);
                }
                ok = ok && lab == 0;
            }
            ok = (__ballot_sync(kFull, !ok) & own) == 0;
            if (many) {
                int steps = 0, cur = 0;
                const bool walk = loop && ok && ne > W;
                if (walk && sl == 0) {
                    do {
                        cur = P.se[(P.hz(cur) >> 8) & 0xff];
                        ++steps;
                    } while (cur != 0 && steps <= ne);
                }
                __syncwarp();
                const bool one = __shfl_sync(kFull, (int)(steps == ne && cur == 0), 0, W);
                if (walk) ok = one;
            }
            if (loop && !ok) fail = true;
        }
        const int nft = nfree + nvis;
        if (act && !fail) {
            if (live - nvis + ne > o.max_faces) {
                end = D3D_STATUS_EPA_FACE_OVERFLOW;
                live -= nvis;
            } else if (ne > nft && nslots + (ne - nft) > cap_f) {
                fail = true;  // beyond the Euler bound: never for a closed surface
            }
        }
        __syncwarp();
        // ---- new faces (a, b, w): slots from the top of the free list, then fresh
        bool bad = false;
        if (act && !fail && end == kRun) {
            const bool single = nvis == 1;
            for (int e = sl; e < ne; e += W) {
                const unsigned x = P.hz(e);
                const int ea = x & 0xff, eb = (x >> 8) & 0xff, g = (x >> 16) & 0xff;
                const int nx = single ? (e == 2 ? 0 : e + 1) : P.se[eb];
                const int pv = single ? (e == 0 ? 2 : e - 1) : P.ee[ea];
                const int s = e < nft ? P.freel[nft - 1 - e] : nslots + (e - nft);
                const int sn = nx < nft ? P.freel[nft - 1 - nx] : nslots + (nx - nft);
                const int sp = pv < nft ? P.freel[nft - 1 - pv] : nslots + (pv - nft);
                float4 pl;
                float off = 0.f;
                if (!byte_plane(P, ea, eb, vn, pl, off)) bad = true;
                pl.w = __uint_as_float(offset_key(off));
                P.fn[s] = pl;
                P.fv[s] = pack3(ea, eb, vn);
                P.adj[s] = (unsigned)g | ((unsigned)sn << 8) | ((unsigned)sp << 16);
                reinterpret_cast<unsigned char*>(P.adj + g)[x >> 24] = (unsigned char)s;
            }
        }
        bad = (__ballot_sync(kFull, bad) & own) != 0;
        if (act && end == kRun) {
            if (fail || bad) {
                end = kEpaFallback;
            } else {
                nslots = ne > nft ? nslots + (ne - nft) : nslots;
                nfree = ne < nft ? nft - ne : 0;
                live += ne - nvis;
            }
        }
        __syncwarp();
        // ---- ended pairs
        if (!__any_sync(kFull, end != kRun)) continue;
        const bool fin = end != kRun && end != kEpaFallback;
        const int nf = fin && end != D3D_STATUS_EPA_DEGENERATE ? live : 0;
        if (sl == 0 && end == kEpaFallback) fallback[atomicAdd(n_fallback, 1ull)] = (int32_t)k;
        if (sl == 0 && fin) {
            d3 m = mk(double(NAN), double(NAN), double(NAN));
            if (end == D3D_STATUS_OK || end == D3D_STATUS_EPA_NOT_CONVERGED) {
                // the face's normal now; the FP64 depth along it in k_epa_refine
                const float4 q = P.fn[cf];
                m = mk((double)q.x, (double)q.y, (double)q.z);
                refine[atomicAdd(n_refine, 1ull)] = (int32_t)k;
            }
            mtv[3 * k] = m.x;
            mtv[3 * k + 1] = m.y;
            mtv[3 * k + 2] = m.z;
            status[k] = (int8_t)end;
            n_faces[k] = nf;
        }
        if (faces) {
            // live faces in slot order: three vertices and the normal
            double* out = faces + k * 12 * (int64_t)o.max_faces;
            int base = 0;
            for (int f0 = 0; __any_sync(kFull, nf > 0 && f0 < nslots); f0 += W) {
                const int f = f0 + sl;
                const bool on = nf > 0 && f < nslots && __float_as_uint(P.fn[f < nslots ? f : 0].w) != kFreeKey;
                const unsigned mask = (__ballot_sync(kFull, on) & own);
                if (on) {
                    double* q = out + 12 * (base + __popc(mask & below));
                    const unsigned fw = P.fv[f];
#pragma unroll
                    for (int j = 0; j < 3; ++j) {
                        const f3 yy = P.y(vid(fw, j));
                        q[3 * j] = yy.x;
                        q[3 * j + 1] = yy.y;
                        q[3 * j + 2] = yy.z;
                    }
                    const float4 pl = P.fn[f];
                    q[9] = pl.x;
                    q[10] = pl.y;
                    q[11] = pl.z;
                }
                base += __popc(mask);
            }
        }
        if (end != kRun) run = false;
        __syncwarp();
    }
}

// The FP64 refinement of the FP32 search's converged faces: the unit normal
// the search left in mtv, renormalised in FP64, and mtv = n (n . w(n)) with
// RefineSupport (the reference's expression at convergence, epa.py:69).
// n . w(n) is the support depth h(n), an upper bound on the penetration depth
// for every n, and the FP32 normal of the converged face is within the
// search's tolerance of the optimal direction.  In the search kernel the whole
// warp waited on each pair's FP64 support chain.  A block lists the two supports of its pairs by
// collider type (typelist.cuh); with a pair per thread the lanes of a warp ran
// through all types (6.3 lanes per FP64 instruction).  Converged pairs of the
// bench workload (310k): 210 -> 110 us.
constexpr int kRefine = 128;

template <bool MESH>
__global__ void __launch_bounds__(kRefine) k_epa_refine(d3d_store st, const int32_t* __restrict__ i1,
                                                        const int32_t* __restrict__ i2,
                                                        const int32_t* __restrict__ list,
                                                        const unsigned long long* __restrict__ n_dev,
                                                        double* __restrict__ mtv) {
    __shared__ double dir[3 * kRefine], sup[2][3 * kRefine];
    __shared__ int col[2 * kRefine];
    __shared__ unsigned short task[2 * kRefine];  // thread << 1 | side
    __shared__ int cnt[kSupportBins], next;
    const int64_t n = (int64_t)*n_dev;
    const int t = threadIdx.x, ln = lane_id();
    // fewer pairs per block where full blocks would leave SMs idle
    const int64_t share = (n + gridDim.x - 1) / gridDim.x;
    const int per = share < 16 ? 16 : (share > kRefine ? kRefine : (int)share);
    for (int64_t base = (int64_t)blockIdx.x * per; base < n; base += (int64_t)gridDim.x * per) {
        __syncthreads();  // the last round's reads
        if (t < kSupportBins) cnt[t] = 0;
        if (t == kSupportBins) next = 0;
        __syncthreads();
        const bool on = t < per && base + t < n;
        int64_t k = 0;
        d3 nrm = mk(0.0, 0.0, 0.0);
        int bin[2] = {0, 0}, pos[2] = {0, 0};
        if (on) {
            k = list[base + t];
            nrm = mk(mtv[3 * k], mtv[3 * k + 1], mtv[3 * k + 2]);
            nrm = nrm * (1.0 / sqrt(dot(nrm, nrm)));
            dir[t] = nrm.x;
            dir[kRefine + t] = nrm.y;
            dir[2 * kRefine + t] = nrm.z;
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int c = (h ? i2 : i1)[k];
                col[h * kRefine + t] = c;
                const int4 m = __ldg(reinterpret_cast<const int4*>(st.meta) + c);
                bin[h] = m.x == D3D_HULL ? kSearchBin : support_bin(m.x, m.w);
                pos[h] = atomicAdd(cnt + bin[h], 1);
            }
        }
        __syncthreads();
        const Chunks ch = chunks_of(cnt, kSupportBins, ln == kSearchBin ? 4 : 32);
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int p = ch.start(bin[h]) + pos[h];
            if (on) task[p] = (unsigned short)(2 * t + h);
        }
        __syncthreads();
        int cb, first, num;
        while (ch.take(&next, cb, first, num)) {
            const bool mine = ln < num;
            const int e = task[first + (mine ? ln : 0)];
            const int u = e >> 1, h = e & 1;
            const int c = col[h * kRefine + u];
            d3 d = mk(dir[u], dir[kRefine + u], dir[2 * kRefine + u]);
            if (h) d = -d;
            int vi = -1;
            const f3 f = RefineSupportT<MESH>::rounded(d);
            if (cb == kSearchBin) {  // the hulls, each by the whole warp
                int type, nv, off;
                load_meta(st, c, type, nv, off);
                for (int q = 0; q < num; ++q) {
                    const int w = warp_hull_argmax(
                        st.verts32, __shfl_sync(kFull, off, q), max(__shfl_sync(kFull, nv, q), 1),
                        mk(__shfl_sync(kFull, f.x, q), __shfl_sync(kFull, f.y, q), __shfl_sync(kFull, f.z, q)));
                    if (ln == q) vi = w;
                }
            }
            if (mine) {
                Col<double> cl;
                load_col(st, c, cl);
                const d3 x = RefineSupportT<MESH>::eval_at(cl, st, d, f, vi);
                sup[h][u] = x.x;
                sup[h][kRefine + u] = x.y;
                sup[h][2 * kRefine + u] = x.z;
            }
            __syncwarp();
        }
        __syncthreads();
        if (on) {
            const d3 p = mk(sup[0][t], sup[0][kRefine + t], sup[0][2 * kRefine + t]);
            const d3 q = mk(sup[1][t], sup[1][kRefine + t], sup[1][2 * kRefine + t]);
            const d3 m = nrm * dot(p - q, nrm);
            mtv[3 * k] = m.x;
            mtv[3 * k + 1] = m.y;
            mtv[3 * k + 2] = m.z;
        }
    }
}

}  // namespace

namespace {

int prepare_smem(const void* fn, int smem) {
    cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(fn, cudaFuncAttributePreferredSharedMemoryCarveout,
                                 (int)cudaSharedmemCarveoutMaxShared);
    if (e == cudaSuccess) return D3D_SUCCESS;
    set_error("d3d_epa (mixed): %s", cudaGetErrorString(e));
    return D3D_ERR_CUDA;
}

int sm_count() {
    int dev = 0, sms = 1;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    return sms;
}

template <int W, int WARPS, bool MESH>
int launch_segments(const d3d_store& store, const int32_t* i1, const int32_t* i2, const int32_t* list, int64_t n,
                    const unsigned long long* n_dev, unsigned long long* cursor, const double* simplex,
                    const d3d_epa_options& o, double* mtv, int8_t* status, int32_t* n_faces, double* faces,
                    int32_t* fallback, unsigned long long* n_fallback, int32_t* refine, unsigned long long* n_refine,
                    int64_t lo, int64_t hi, cudaStream_t stream) {
    const void* fn = (const void*)k_epa_segments<W, WARPS, MESH>;
    const int smem = byte_poly_bytes(o) * WARPS * Seg<W>::kPairs;
    int rc = prepare_smem(fn, smem);
    if (rc) return rc;
    k_epa_segments<W, WARPS, MESH><<<persistent_blocks(fn, 32 * WARPS, launch_items(n * 32, n * W / 4), 0, smem), 32 * WARPS, smem,
                                     stream>>>(store, i1, i2, list, n, n_dev, cursor, simplex, o, mtv, status, n_faces,
                                               faces, fallback, n_fallback, refine, n_refine, lo, hi);
    return check_launch("d3d_epa (mixed)");
}

// The FP32 search's form by its number of pairs and the bytes of a polytope.
// Up to two pairs per resident warp the batch takes as long as its longest
// pairs, which a whole warp each steps fastest; above that the issue slots
// decide, which 8 lanes per pair save most while 20 warps of four pairs fit in
// an SM's shared memory, and 16 lanes otherwise.  Measured with 32, 16, 8
// lanes, us: 64 faces (2,824 bytes): 900 pairs 101, 125, 142; 6,667 pairs 156,
// 179, 194; 13,333 pairs 376, 233, 241; 33,333 pairs 611, 436, 365.  256 faces
// (4,528 bytes): 6,667 pairs 212, 247, 279; 13,333 pairs 450, 284, 307;
// 310,000 pairs 4,939, 3,357, 3,736.  Beside other batches (shared_gpu) the form
// of a whole warp is left out, and the grid holds a quarter of n, about the
// pairs that intersect (16 server slots: 51.3 M pairs/s; an eighth 49.2, all of
// n 45.5).
template <int WARPS, bool MESH>
int launch_search(const d3d_store& store, const int32_t* i1, const int32_t* i2, const int32_t* list, int64_t n,
                  const unsigned long long* n_dev, unsigned long long* cursor, const double* simplex,
                  const d3d_epa_options& o, double* mtv, int8_t* status, int32_t* n_faces, double* faces,
                  int32_t* fallback, unsigned long long* n_fallback, int32_t* refine, unsigned long long* n_refine,
                  cudaStream_t stream) {
    const int64_t few = shared_gpu() ? 0 : 2 * seg_warps(32) * (int64_t)sm_count() + 1;
    // with the count on the device the forms of both sides are launched and one returns at once
    if (few && (n_dev || n < few)) {
        const int rc = launch_segments<32, WARPS, MESH>(store, i1, i2, list, n < few ? n : few, n_dev, cursor, simplex,
                                                        o, mtv, status, n_faces, faces, fallback, n_fallback, refine,
                                                        n_refine, 0, few, stream);
        if (rc || n < few) return rc;
    }
    const int per_sm = 228 * 1024 - 1024 * (seg_warps(8) / WARPS);  // 1 KB of a block is the system's
    if (byte_poly_bytes(o) * Seg<8>::kPairs * (seg_warps(8) / WARPS * WARPS) <= per_sm)
        return launch_segments<8, WARPS, MESH>(store, i1, i2, list, n, n_dev, cursor, simplex, o, mtv, status,
                                               n_faces, faces, fallback, n_fallback, refine, n_refine, few, INT64_MAX,
                                               stream);
    return launch_segments<16, WARPS, MESH>(store, i1, i2, list, n, n_dev, cursor, simplex, o, mtv, status, n_faces,
                                            faces, fallback, n_fallback, refine, n_refine, few, INT64_MAX, stream);
}

template <typename T, int WARPS, bool MESH>
int launch_warp(const d3d_store& store, const int32_t* i1, const int32_t* i2, const int32_t* list, int64_t n,
                const unsigned long long* n_dev, unsigned long long* cursor, const double* simplex,
                const d3d_epa_options& o, double* mtv, int8_t* status, int32_t* n_faces, double* faces,
                int32_t* fallback, unsigned long long* n_fallback, int32_t* refine, unsigned long long* n_refine,
                cudaStream_t stream) {
    int rc;
    if (sizeof(T) == 4 && face_cap(o) <= 255) {
        rc = launch_search<WARPS, MESH>(store, i1, i2, list, n, n_dev, cursor, simplex, o, mtv, status, n_faces, faces,
                                        fallback, n_fallback, refine, n_refine, stream);
    } else {
        const void* fn = (const void*)k_epa_warp<T, WARPS, MESH>;
        const int smem = layout_for<T>(o).bytes * WARPS;
        rc = prepare_smem(fn, smem);
        if (rc) return rc;
        k_epa_warp<T, WARPS, MESH><<<persistent_blocks(fn, 32 * WARPS, n * 32, 0, smem), 32 * WARPS, smem, stream>>>(
            store, i1, i2, list, n, n_dev, cursor, simplex, o, mtv, status, n_faces, faces, fallback, n_fallback,
            refine, n_refine);
        rc = check_launch("d3d_epa (mixed)");
    }
    if (rc || sizeof(T) == 8) return rc;
    const void* kr = (const void*)k_epa_refine<MESH>;
    k_epa_refine<MESH><<<persistent_blocks(kr, kRefine, launch_items(8 * n, n)), kRefine, 0, stream>>>(store, i1, i2, refine, n_refine, mtv);
    return check_launch("d3d_epa (mixed, refinement)");
}

// The kernels without the MeshGraph branch serve stores without meshes.
template <typename T, int WARPS>
int launch_warp(const d3d_store& store, const int32_t* i1, const int32_t* i2, const int32_t* list, int64_t n,
                const unsigned long long* n_dev, unsigned long long* cursor, const double* simplex,
                const d3d_epa_options& o, double* mtv, int8_t* status, int32_t* n_faces, double* faces,
                int32_t* fallback, unsigned long long* n_fallback, int32_t* refine, unsigned long long* n_refine,
                cudaStream_t stream) {
    if (store.n_links > 0)
        return launch_warp<T, WARPS, true>(store, i1, i2, list, n, n_dev, cursor, simplex, o, mtv, status, n_faces,
                                           faces, fallback, n_fallback, refine, n_refine, stream);
    return launch_warp<T, WARPS, false>(store, i1, i2, list, n, n_dev, cursor, simplex, o, mtv, status, n_faces,
                                        faces, fallback, n_fallback, refine, n_refine, stream);
}

}  // namespace

namespace d3d {

constexpr int64_t kSmemPerBlock = 227 * 1024;

bool epa_warp_supported(const d3d_epa_options& o, bool fp64) {
    if (o.max_iterations > 250 || o.max_loose_edges > 255 || o.max_faces > 65535) return false;
    const int bytes = fp64 ? layout_for<double>(o).bytes : layout_for<float>(o).bytes;
    return (int64_t)bytes * 2 <= kSmemPerBlock;
}

int epa_warp_count(const d3d_tuning& t, const d3d_epa_options& o, bool fp64) {
    const int64_t bytes = fp64 ? layout_for<double>(o).bytes : layout_for<float>(o).bytes;
    int w = t.epa_warps;
    while (w > 2 && bytes * w > kSmemPerBlock) w /= 2;
    return w;
}

int epa_warp_launch(const d3d_store& store, const int32_t* i1, const int32_t* i2, const int32_t* list, int64_t n,
                    const unsigned long long* n_dev, unsigned long long* cursor, const double* simplex,
                    const d3d_epa_options& o, double* mtv, int8_t* status, int32_t* n_faces, double* faces,
                    int32_t* fallback, unsigned long long* n_fallback, cudaStream_t stream, bool fp64,
                    int32_t* refine, unsigned long long* n_refine) {
    const int w = epa_warp_count(tuning(), o, fp64);
#define D3D_WARP_LAUNCH(T, W)                                                                                      \
    return launch_warp<T, W>(store, i1, i2, list, n, n_dev, cursor, simplex, o, mtv, status, n_faces, faces, fallback, \
                             n_fallback, refine, n_refine, stream)
    if (fp64) {
        refine = nullptr;  // the FP64 search refines with exact supports itself
        if (w == 2) D3D_WARP_LAUNCH(double, 2);
        if (w == 8) D3D_WARP_LAUNCH(double, 8);
        D3D_WARP_LAUNCH(double, 4);
    }
    if (w == 2) D3D_WARP_LAUNCH(float, 2);
    if (w == 8) D3D_WARP_LAUNCH(float, 8);
    D3D_WARP_LAUNCH(float, 4);
#undef D3D_WARP_LAUNCH
}

}  // namespace d3d
