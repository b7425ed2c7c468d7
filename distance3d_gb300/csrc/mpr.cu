// mpr.cu -- Minkowski portal refinement (MPR), the plain FP64 drop-in for
// distance3d's mpr_intersection and mpr_penetration (mpr.py:21-110).
// Compiled with -fmad=false: every step is the reference's
// rounding sequence (NumPy orders as in d3d_device.cuh), so flags, depths,
// directions and contact positions are the reference's bit for bit.
//
// Like the FP64 GJK (gjk_pool.cuh), bound by the FP64 pipe and by the length
// of a pair's chain: a block keeps one pair per thread in shared memory and
// runs rounds of one support evaluation each, listing the supports by collider
// type, the centers of hulls and meshes (the vertices summed in order, one
// component per lane), the steps of the state machine of mpr.cuh by phase, and
// the finished pairs' penetration results, so that a warp runs one of them at
// a time.  One pair per lane had 4.6 lanes per FP64 instruction: 50,021 pairs
// of the ten types 2.21 ms (1.53 with the integer compares), now 0.78 ms.
// The refinement loop of the reference has no bound; here it stops after
// `refine_limit` expansions with status D3D_STATUS_MAX_ITER.  d3d_mpr also
// dispatches the mixed form (mpr_mixed.cu).
#include "capi_util.h"
#include "gjk_pool.cuh"
#include "mpr.cuh"
#include "mpr_impl.h"
#include "persist.cuh"
#include "scratch.h"
#include "typelist.cuh"

namespace {

using namespace d3d;

constexpr int kSlots = 256;  // pairs (and threads) per block
constexpr unsigned kAll = 0xffffffffu;
constexpr int kCenterBin = 2 * kSupportTypes;  // bins after the supports: centers of hulls and meshes, finished pairs
constexpr int kEndBin = kCenterBin + 1;
constexpr int kBins = kEndBin + 1;
constexpr int kInit = 5;  // phase of a pair whose portal is not begun
constexpr int kPhases = 6;

using PortalT = mpr::Portal<double, kSlots, true>;
enum { kFree = 0, kLive = 1, kEnding = 2, kSpare = 3 };  // kSpare: beyond the share (persist.cuh)

struct Mem {
    double rows[PortalT::kWords * kSlots];
    double dir[3 * kSlots];
    double sup[2][3 * kSlots];
    int col[2 * kSlots];
    int pid[kSlots];
    int it[kSlots];
    int meta[kSlots];  // state | phase << 2 | outcome << 5
    unsigned short list[2 * kSlots];        // slot << 1 | side, by bin
    unsigned short step[kPhases * kSlots];  // slots by phase
    int cnt[2][kBins];
    int scnt[2][kPhases];
    int next[2][2];

    __device__ d3 direction(int s) const { return mk(dir[s], dir[kSlots + s], dir[2 * kSlots + s]); }
    __device__ void put_direction(int s, d3 d) {
        dir[s] = d.x;
        dir[kSlots + s] = d.y;
        dir[2 * kSlots + s] = d.z;
    }
    __device__ d3 point(int side, int s) const {
        return mk(sup[side][s], sup[side][kSlots + s], sup[side][2 * kSlots + s]);
    }
    __device__ void put_support(int s, int side, d3 x) {
        sup[side][s] = x.x;
        sup[side][kSlots + s] = x.y;
        sup[side][2 * kSlots + s] = x.z;
    }
    __device__ PortalT portal(int s) { return PortalT{rows + s}; }
};

// mpr::collider_center of up to ten listed hulls or meshes, three lanes each.
__device__ __forceinline__ void centers(Mem& m, const d3d_store& st, int first, int count) {
    const int ln = threadIdx.x & 31;
    const int g = ln / 3, i = ln - 3 * g;
    const bool on = g < count;
    const int e = m.list[first + (on ? g : 0)];
    const int s = e >> 1, side = e & 1;
    Col<double> c;
    load_meta(st, m.col[side * kSlots + s], c);
    double x = 0.0;
    if (on && c.nv >= 1) {
        const double* v = st.verts64 + (size_t)c.off * 4 + i;
        x = __ldg(v);
#pragma unroll 8
        for (int k = 1; k < c.nv; ++k) x = x + __ldg(v + 4 * (size_t)k);
        x = x / (double)c.nv;
    }
    const d3 mean = mk(__shfl_sync(kAll, x, 3 * g), __shfl_sync(kAll, x, 3 * g + 1 < 32 ? 3 * g + 1 : 31),
                       __shfl_sync(kAll, x, 3 * g + 2 < 32 ? 3 * g + 2 : 31));
    if (!on) return;
    if (c.nv < 1) {
        x = NAN;
    } else if (c.type == D3D_MESH) {
        const double* r = st.rec64 + (size_t)c.idx * 16;
        x = __ldg(r + 9 + i) +
            dot102(__ldg(r + 3 * i), __ldg(r + 3 * i + 1), __ldg(r + 3 * i + 2), mean.x, mean.y, mean.z);
    }
    m.portal(s).at(1 + side, 0, i) = x;
}

// The FP64 MPR of pairs order[slot] (or slot), slot < n; with n_dev, the pair
// count is read on the device (the mixed form's fallback list).
__global__ void __launch_bounds__(kSlots, 2) k_mpr(d3d_store st, const int32_t* __restrict__ i1,
                                                   const int32_t* __restrict__ i2, const int32_t* __restrict__ order,
                                                   int64_t n, const unsigned long long* __restrict__ n_dev,
                                                   unsigned long long* __restrict__ cursor, d3d_mpr_options opt,
                                                   mpr::Out o) {
    extern __shared__ __align__(16) unsigned char mpr_smem[];
    Mem& m = *reinterpret_cast<Mem*>(mpr_smem);
    const int t = threadIdx.x, ln = t & 31;
    if (n_dev) n = (int64_t)*n_dev;
    const d3 nan3 = mk(double(NAN), double(NAN), double(NAN));
    // a batch that does not fill every block is spread evenly over them
    const long long share = (n + gridDim.x - 1) / gridDim.x;
    const long long split = share < kSlots ? 0 : n;
    bool exhausted = share == 0;
    WarpChunk chunk;
    m.meta[t] = !exhausted && t >= share ? kSpare : kFree;
    if (!exhausted && t >= share) m.it[t] = spare_rounds(t, share);
    if (t < kBins) m.cnt[0][t] = m.cnt[1][t] = 0;
    if (t < kPhases) m.scnt[0][t] = m.scnt[1][t] = 0;
    if (t < 2) m.next[0][t] = m.next[1][t] = 0;
    int type[2] = {0, 0};
    __syncthreads();
    for (int par = 0;; par ^= 1) {
        // ---- free slots take new pairs
        int meta = m.meta[t];
        const bool want = (meta & 3) == kFree && !exhausted;
        const long long slot = fetch_slot_chunked(cursor, want, chunk, kAll, 32, split);
        if (want) {
            if (slot >= n) {
                exhausted = true;
            } else {
                const int pid = order ? order[slot] : (int)slot;
                const int c[2] = {i1[pid], i2[pid]};
                if (!pair_ok(st, c[0], c[1])) {
                    mpr::store(o, pid, false, D3D_STATUS_BAD_INDEX, opt.penetration, NAN, nan3, nan3);
                } else {
                    m.pid[t] = pid;
                    m.it[t] = 0;
#pragma unroll
                    for (int k = 0; k < 2; ++k) {
                        const int4 q = __ldg(reinterpret_cast<const int4*>(st.meta) + c[k]);
                        type[k] = support_bin(q.x, q.w);
                        m.col[k * kSlots + t] = c[k];
                        if (q.x != D3D_HULL && q.x != D3D_MESH)
                            m.portal(t).put(1 + k, 0, mpr::collider_center<double>(st, c[k]));
                    }
                    meta = kLive | (kInit << 2);
                    m.meta[t] = meta;
                }
            }
        }
        // ---- list the supports, the centers and the ends
        const int state = meta & 3, phase = (meta >> 2) & 7;
        int bin[2], pos[2];
#pragma unroll
        for (int k = 0; k < 2; ++k) {
            const bool poly = (type[k] >> 1) == D3D_HULL || (type[k] >> 1) == D3D_MESH;
            bin[k] = state == kLive ? (phase == kInit ? (poly ? kCenterBin : -1) : type[k])
                                    : (state == kEnding && k == 0 ? kEndBin : -1);
            const unsigned same = __match_any_sync(kAll, bin[k]);
            const int leader = __ffs(same) - 1;
            int base = 0;
            if (ln == leader && bin[k] >= 0) base = atomicAdd(&m.cnt[par][bin[k]], __popc(same));
            pos[k] = __shfl_sync(kAll, base, leader) + __popc(same & ((1u << ln) - 1u));
        }
        const int running = __syncthreads_or(((state == kFree ? !exhausted : state != kSpare) ? 1 : 0) | (state == kLive ? 2 : 0));
        if (!running) break;
        // the finished pairs wait until they fill a warp, or no pair is left to iterate
        const bool ends = m.cnt[par][kEndBin] >= 32 || !(running & 2);
        const Chunks ch = chunks_of(m.cnt[par], ends ? kBins : kEndBin,
                                    (ln >> 1) == D3D_HULL ? pool::kHullChunk : (ln == kCenterBin ? 10 : 32));
#pragma unroll
        for (int k = 0; k < 2; ++k) {
            const int p = ch.start(bin[k] >= 0 ? bin[k] : 0) + pos[k];
            if (bin[k] >= 0 && (bin[k] != kEndBin || ends)) m.list[p] = (unsigned short)(2 * t + k);
        }
        __syncthreads();
        int cb, first, count;
        while (ch.take(&m.next[par][0], cb, first, count)) {
            if ((cb >> 1) == D3D_HULL) {
                pool::hull_supports<kSlots>(m, st, first, count);
            } else if (cb == kCenterBin) {
                centers(m, st, first, count);
            } else if (ln < count) {
                const int e = m.list[first + ln];
                if (cb == kEndBin) {
                    const int s = e >> 1;
                    double depth;
                    d3 dir, cp;
                    mpr::penetration((m.meta[s] >> 5) & 3, m.portal(s), depth, dir, cp);
                    mpr::store(o, m.pid[s], true, D3D_STATUS_OK, true, depth, dir, cp);
                    m.meta[s] = 0;
                } else {
                    pool::lane_support<kSlots>(m, st, e);
                }
            }
            __syncwarp();
        }
        __syncthreads();
        // ---- list the pairs by phase
        {
            const int cls = state == kLive ? phase : -1;
            unsigned mine = 0;
            int base = 0;
#pragma unroll
            for (int k = 0; k < kPhases; ++k) {
                const unsigned b = __ballot_sync(kAll, cls == k);
                if (cls == k) mine = b;
                if (ln == k) base = b ? atomicAdd(&m.scnt[par][k], __popc(b)) : 0;
            }
            const int p = __shfl_sync(kAll, base, cls >= 0 ? cls : 0) + __popc(mine & ((1u << ln) - 1u));
            if (cls >= 0) m.step[cls * kSlots + p] = (unsigned short)t;
        }
        if (state == kSpare) {
            exhausted = slots_claimed(cursor, n);
            if (exhausted || --m.it[t] == 0) m.meta[t] = kFree;
        }
        // the other parity's counters, free since the last round
        if (t < kBins) m.cnt[par ^ 1][t] = 0;
        if (t < kPhases) m.scnt[par ^ 1][t] = 0;
        if (t < 2) m.next[par ^ 1][t] = 0;
        __syncthreads();
        // ---- one step of every pair
        const Chunks ph = chunks_of(m.scnt[par], kPhases, 32);
        while (ph.take(&m.next[par][1], cb, first, count)) {
            const int k = first - ph.start(cb) + ln;
            if (ln < count) {
                const int s = m.step[cb * kSlots + k];
                const PortalT P = m.portal(s);
                mpr::Lane<double> L;
                L.it = m.it[s];
                int status = D3D_STATUS_OK, r = mpr::kRunning;
                if (cb == kInit) {
                    mpr::begin(P, L, P.a(0), P.b(0));
                } else {
                    L.phase = cb;
                    L.d = m.direction(s);
                    r = mpr::round(P, L, m.point(0, s), m.point(1, s), opt, status);
                }
                if (r == mpr::kRunning) {
                    m.it[s] = L.it;
                    m.put_direction(s, L.d);
                    m.meta[s] = kLive | (L.phase << 2);
                } else if (r != mpr::kMiss && opt.penetration) {
                    m.meta[s] = kEnding | (r << 5);
                } else {
                    mpr::store(o, m.pid[s], r != mpr::kMiss, status, opt.penetration, NAN, nan3, nan3);
                    m.meta[s] = 0;
                }
            }
            __syncwarp();
        }
        __syncthreads();
    }
}

}  // namespace

namespace d3d {

int mpr_f64_launch(const d3d_store& store, const int32_t* i1, const int32_t* i2, const int32_t* order, int64_t n,
                   const unsigned long long* n_dev, unsigned long long* cursor, const d3d_mpr_options& opt,
                   const mpr::Out& o, cudaStream_t stream) {
    const void* fn = (const void*)k_mpr;
    const int smem = (int)sizeof(Mem);
    cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(fn, cudaFuncAttributePreferredSharedMemoryCarveout,
                                 (int)cudaSharedmemCarveoutMaxShared);
    if (e != cudaSuccess) {
        set_error("d3d_mpr: %s", cudaGetErrorString(e));
        return D3D_ERR_CUDA;
    }
    const int blocks = persistent_blocks(fn, kSlots, n * kSlots, 0, smem);
    k_mpr<<<blocks, kSlots, smem, stream>>>(store, i1, i2, order, n, n_dev, cursor, opt, o);
    return check_launch("d3d_mpr");
}

}  // namespace d3d

extern "C" int d3d_mpr(const d3d_store* store, const int32_t* i1, const int32_t* i2, int64_t n,
                       const d3d_mpr_options* opt, int8_t* hit, double* depth, double* dir, double* pos,
                       int8_t* status, void* stream) {
    int rc = d3d::check_store(store, "d3d_mpr");
    if (rc) return rc;
    D3D_REQUIRE(opt, "d3d_mpr: null options");
    D3D_REQUIRE(n >= 0, "d3d_mpr: n < 0");
    D3D_REQUIRE(opt->max_iterations >= 0 && opt->refine_limit >= 0, "d3d_mpr: negative iteration bound");
    D3D_REQUIRE(opt->tolerance >= 0.0, "d3d_mpr: negative tolerance");
    D3D_REQUIRE(opt->precision == D3D_PRECISION_FP64 || opt->precision == D3D_PRECISION_MIXED,
                "d3d_mpr: unknown precision %d", opt->precision);
    if (n == 0) return D3D_SUCCESS;
    D3D_REQUIRE(i1 && i2 && hit && status, "d3d_mpr: null pointer");
    D3D_REQUIRE(n <= INT32_MAX, "d3d_mpr: more than 2^31 pairs");
    cudaStream_t st = d3d::as_stream(stream);
    const bool mixed = opt->precision == D3D_PRECISION_MIXED;
    void* scratch = nullptr;
    rc = d3d::scratch_alloc(&scratch, d3d::mpr_scratch_bytes(n, mixed), st);
    if (rc) return rc;
    d3d::mpr::Out o{hit, depth, dir, pos, status};
    rc = mixed ? d3d::mpr_mixed_run(*store, i1, i2, n, *opt, o, scratch, st)
               : d3d::mpr_f64_run(*store, i1, i2, n, *opt, o, scratch, st);
    d3d::scratch_free(scratch, st);
    return rc;
}

namespace d3d {

size_t mpr_scratch_bytes(int64_t n, bool mixed) {
    const size_t order = (sizeof(int32_t) * (size_t)n + 255) & ~size_t(255);
    size_t bytes = 256 + order + pair_order_temp_bytes(n);
    if (mixed) bytes += mpr_mixed_extra_bytes(n);
    return bytes;
}

int mpr_f64_run(const d3d_store& store, const int32_t* i1, const int32_t* i2, int64_t n, const d3d_mpr_options& opt,
                const mpr::Out& o, void* scratch, cudaStream_t st) {
    const bool sched = n >= tuning().sort_min;
    unsigned long long* cursor = static_cast<unsigned long long*>(scratch);
    const size_t order_bytes = (sizeof(int32_t) * (size_t)n + 255) & ~size_t(255);
    int32_t* order = sched ? reinterpret_cast<int32_t*>(static_cast<char*>(scratch) + 256) : nullptr;
    cudaError_t e = cudaMemsetAsync(cursor, 0, sizeof(unsigned long long), st);
    if (e != cudaSuccess) {
        set_error("d3d_mpr: %s", cudaGetErrorString(e));
        return D3D_ERR_CUDA;
    }
    int rc = D3D_SUCCESS;
    if (sched)
        rc = pair_order(store, i1, i2, n, order, static_cast<char*>(scratch) + 256 + order_bytes,
                        pair_order_temp_bytes(n), st);
    if (!rc) rc = mpr_f64_launch(store, i1, i2, order, n, nullptr, cursor, opt, o, st);
    return rc;
}

}  // namespace d3d
