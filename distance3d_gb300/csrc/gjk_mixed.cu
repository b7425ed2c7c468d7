// gjk_mixed.cu -- mixed-precision GJK distance.
//
// Five kernels, over the pairs in type-sorted order where the batch fills phase
// A's grid (mixed_sorted), else in input order:
//
// A  runs the Jolt loop in FP32 on the FP32 mirror of the store, with
//    thresholds scaled to single precision, hands each pair's outcome, final
//    closest point and the search direction of each final simplex row on
//    (80 bytes/pair) and appends clipped and unconverged pairs to the
//    fallback list.
// R  (the refinement pass) lists the rows of a block's pairs by collider type,
//    so that a warp's lanes evaluate the same supports.
//    The final simplex rows are re-evaluated in FP64 along their
//    FP32 directions (polytope supports choose their vertex by an FP32 argmax
//    and return the FP64 vertex) and, for a separated pair, one more support
//    pair along -v, the closest point A ended on.  A separated pair whose
//    origin projection lies inside its FP64 feature and whose duality gap
//    brackets the distance within 1e-6 of itself (or 1e-9 of the scene's
//    scale) is done there, closest points from the projection's barycentric
//    coordinates; so is a touching pair whose FP64 tetrahedron encloses the
//    origin.  Every other separated or touching pair is flagged, its FP64 rows
//    in its record, and a stable compaction (CUB) lists the flagged pairs in
//    the order of the slots.
// B  continues the reference's loop (_gjk_jolt.py:224-288) in FP64 for the
//    listed pairs, a pool of pairs per block: the first round solves the
//    handed rows, later rounds add a support pair along -v, until the duality
//    gap closes as in R.  A pair whose loop ends leaves its simplex in the
//    outputs and the rest of its state in its record.
// E  (the end pass) computes the closest points and the checks of B's
//    finished pairs (pb_end), every lane on a finished pair.
// C  is the plain FP64 kernel over the fallback list (the reference's
//    arithmetic; CLIPPED and MAX_ITER keep their FP64 meaning).
//
// FP64 instructions cost the GB300's FP64 pipe the same however few lanes of
// a warp are active, so the FP64 work sits where lanes are busy: R runs the
// same support code on every lane of a warp and a short per-lane solve, and
// only the pairs R cannot finish (those whose gap or feature check fails)
// pay for B's loop.  A pair goes to the fallback list only if its result fails
// the consistency check (closest points vs |v|) or the sanity check in E, or
// hits the iteration bound in B.
//
// On the six-type workloads A takes ~11 FP32 iterations and R evaluates ~3
// rows plus the gap row, against ~17-19 FP64 iterations for the plain form.
// Compiled with -fmad=true: the tests bound its error against the FP64
// oracle.
#define D3D_FP_COMPARES  // see d3d_device.cuh
#include <cub/cub.cuh>

#include "capi_util.h"
#include "gjk_impl.h"
#include "gjk_mixed.cuh"
#include "gjk_out.cuh"
#include "gjk_pool.cuh"
#include "persist.cuh"
#include "scratch.h"

namespace {

using namespace d3d;


// Per-call counters (one 256-byte block): cursors of A, B and C, then the
// lengths of the fallback, finished and run lists.
enum { kCurA = 0, kCurB, kCurC, kNumFallback, kNumEnd, kNumRun, kCounters };

struct Lists {
    int32_t* fallback;
    int32_t* ends;         // pairs whose FP64 loop ended in B, for the end pass
    EndRecord* records;    // by pair: R's FP64 rows for B, B's end state for E
    int8_t* run_flag;      // by slot of the order: R left the pair to B
    int32_t* run_pid;      // by slot of the order: the pair
    int32_t* run;          // the flagged pairs in the order (B's work list)
    unsigned long long* ctr;
};

// slots a warp claims from the type-sorted order at a time
constexpr int kChunk = 32;

// Lanes per warp that take pairs where n pairs are spread over the whole grid.
__device__ __forceinline__ long long spread_lanes(long long n, int block) {
    const long long warps = (long long)gridDim.x * (block / 32);
    return n >= 32 * warps ? 32 : (n + warps - 1) / warps;
}

// Phase A's register budget: 16 resident warps per SM (128 registers), its
// simplex P/Q rows in shared memory (ARows).  At 1M pairs: 3.9 ms for the
// mixed GJK, against 4.2 with 12 warps and the rows in registers, 4.2 with 20
// warps and 4.9 with 24 (more spilled registers).
template <int BLOCK>
constexpr int phase_a_min_blocks() { return 512 / BLOCK; }

// A batch that does not fill the grid (spread_lanes below) runs in
// k_gjk_mixed_a_spread: a few lanes of every warp take pairs, so that their
// different supports and simplex sizes cost little, and the others help to
// scan their hulls.  3,000 six-type pairs: 203 -> 91 us; a full grid stays
// with k_gjk_mixed_a (1M pairs: 2.09 ms, 2.36 in the spread form).
template <int BLOCK, bool MESH>
__global__ void __launch_bounds__(BLOCK, phase_a_min_blocks<BLOCK>()) k_gjk_mixed_a_spread(
    d3d_store s, const int32_t* __restrict__ i1, const int32_t* __restrict__ i2, const int32_t* __restrict__ order,
    int64_t n, const int64_t* __restrict__ n_dev, float tol_sq, float max_d2, int max_iter,
    Handoff* __restrict__ hand, DistanceOut out, Lists lists) {
    constexpr unsigned kAll = 0xffffffffu;
    if (n_dev) n = *n_dev;
    __shared__ float4 arows[4 * BLOCK];
    PhaseALoop<ARows<BLOCK>> L;
    L.S.R.base = arows + threadIdx.x;
    int64_t pid = 0;
    int a = 0, b = 0;
    const long long lanes = spread_lanes(n, BLOCK);
    bool have = false, bad = false, exhausted = false;
    // rounds the lane sits out (persist.cuh)
    int spare = (int)(threadIdx.x & 31) >= lanes && lanes ? spare_rounds(threadIdx.x & 31, lanes) : 0;
    WarpChunk chunk;
    while (true) {
        __syncwarp();
        const bool want = !have && !exhausted && spare == 0;
        const long long slot = fetch_slot_chunked(lists.ctr + kCurA, want, chunk, kAll, kChunk, 0);
        if (want) {
            if (slot >= n) {
                exhausted = true;
            } else {
                pid = order ? order[slot] : slot;
                a = i1[pid];
                b = i2[pid];
                bad = !pair_ok(s, a, b);
                pa_begin(L);
                have = true;
            }
        }
        if (!__any_sync(kAll, have)) break;
        int o = pa_step<MESH, true>(L, have && !bad, s, a, b, tol_sq, max_d2, max_iter);
        if (have && bad) o = PA_BAD_INDEX;
        const bool done = have && o >= 0;
        if (done) {
            hand[pid] = pa_handoff(L, o);
            if (bad) store_bad_index(out, pid);
            have = false;
        }
        if (spare) {
            exhausted = slots_claimed(lists.ctr + kCurA, n);
            spare = exhausted ? 0 : spare - 1;
        }
        __syncwarp();
        append_lanes(kAll, lists.fallback, lists.ctr + kNumFallback, done && (o == PA_CLIPPED || o == PA_FAILED),
                     (int32_t)pid);
    }
}

template <int BLOCK, bool MESH>
__global__ void __launch_bounds__(BLOCK, phase_a_min_blocks<BLOCK>()) k_gjk_mixed_a(d3d_store s, const int32_t* __restrict__ i1,
                                                        const int32_t* __restrict__ i2,
                                                        const int32_t* __restrict__ order, int64_t n,
                                                        const int64_t* __restrict__ n_dev, float tol_sq,
                                                        float max_d2, int max_iter, Handoff* __restrict__ hand,
                                                        DistanceOut out, Lists lists) {
    if (n_dev) n = *n_dev;
    __shared__ float4 arows[4 * BLOCK];
    PhaseALoop<ARows<BLOCK>> L;
    L.S.R.base = arows + threadIdx.x;
    int64_t pid = 0;
    int a = 0, b = 0;
    bool need = true, bad = false;
    unsigned live = __activemask();  // the warp's lanes still in the loop
    WarpChunk chunk;
    // per-lane claims for the last slots: the pairs are short, and slots left in a busy warp's chunk
    // would hold up the end of the launch
    const long long split = n - 2LL * gridDim.x * blockDim.x;
    while (true) {
        __syncwarp(live);
        const long long slot = fetch_slot_chunked(lists.ctr + kCurA, need, chunk, live, kChunk, split);
        const bool quit = need && slot >= n;
        live = __ballot_sync(live, !quit);
        if (quit) break;
        if (need) {
            pid = order ? order[slot] : slot;
            a = i1[pid];
            b = i2[pid];
            bad = !pair_ok(s, a, b);
            pa_begin(L);
            need = false;
        }
        __syncwarp(live);  // the round starts converged (pa_step keeps it so through the solve)
        // a pair with an out-of-range index ends at once; R skips it (its outcome is neither
        // separated nor touching) and it joins no list
        const int o = bad ? PA_BAD_INDEX : pa_step<MESH, false>(L, true, s, a, b, tol_sq, max_d2, max_iter);
        const bool done = o >= 0;
        if (done) {
            hand[pid] = pa_handoff(L, o);
            if (bad) store_bad_index(out, pid);
        }
        append_lanes(live, lists.fallback, lists.ctr + kNumFallback, done && (o == PA_CLIPPED || o == PA_FAILED),
                     (int32_t)pid);
        need = done;
    }
}

// R's checks and outputs for one pair, its FP64 rows at my[(6 j + e) BLOCK]
// (the rows of separated pairs end with the gap row).  Run by the thread the
// block's regrouping gave the pair, which may not be the one that read it.
template <int BLOCK>
__device__ __forceinline__ void r_finish(const double* my, int nr, bool sep, bool touch, float4 v, int it_a,
                                         int32_t pid, int64_t slot, const d3d_gjk_options& opt, const DistanceOut& o,
                                         const Lists& lists) {
    const bool rows_ok = sep || touch;
    auto row_p = [&](int j) { return mk(my[(6 * j) * BLOCK], my[(6 * j + 1) * BLOCK], my[(6 * j + 2) * BLOCK]); };
    auto row_q = [&](int j) {
        return mk(my[(6 * j + 3) * BLOCK], my[(6 * j + 4) * BLOCK], my[(6 * j + 5) * BLOCK]);
    };
    bool done = false;
    d3 cp1 = mk(0.0, 0.0, 0.0), cp2 = cp1;
    double dist = 0.0;
    d3 w[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) w[j] = (j < nr && rows_ok) ? row_p(j) - row_q(j) : mk(0.0, 0.0, 0.0);
    if (sep) {
        d3 vv;
        double lam[3];
        const bool inside = feature_point(w, nr, vv, lam);
        const double vl = dot(vv, vv);
        const d3 wg = row_p(nr) - row_q(nr);
        const d3 u = mk((double)v.x, (double)v.y, (double)v.z);
        // distance in [u.wg / |u|, |vv|] (wg is the support of the Minkowski difference along -u)
        const double upper = sqrt(vl);
        const double lower = dot(u, wg) / sqrt(dot(u, u));
        const double gap = upper - lower;
        double ymax = dot(w[0], w[0]);
#pragma unroll
        for (int j = 1; j < 3; ++j)
            if (j < nr) ymax = maxf2(ymax, dot(w[j], w[j]));
        const double tol_sq = opt.tolerance * opt.tolerance;
        // touching in FP64 (B's test) is B's to decide
        const bool apart = vl > tol_sq && vl > DBL_EPSILON * ymax;
        const bool closed = gap <= kMixedRelGap * upper || gap * gap <= kMixedAbsGap2 * maxf2(1.0, dot(wg, wg));
        if (inside && apart && closed) {
            cp1 = row_p(0) * lam[0];
            cp2 = row_q(0) * lam[0];
#pragma unroll
            for (int j = 1; j < 3; ++j) {
                if (j < nr) {
                    cp1 = cp1 + row_p(j) * lam[j];
                    cp2 = cp2 + row_q(j) * lam[j];
                }
            }
            dist = upper;
            const d3 ab = cp1 - cp2;
            // pb_end's consistency check
            done = abs_t(sqrt(dot(ab, ab)) - dist) <= 1e-10 * maxf2(dist, 1.0);
        }
    } else if (touch) {
        if (outside_planes(w[0], w[1], w[2], w[3], reference_eps<double>()) == 0) {
            // the origin inside the FP64 tetrahedron: closest points as gjk_end takes them
            // (bary_tetra, then merged at distance 0)
            double o4[4];
            bary_tetra(w[0], w[1], w[2], w[3], o4);
            const d3 pa = ((row_p(0) * o4[0] + row_p(1) * o4[1]) + row_p(2) * o4[2]) + row_p(3) * o4[3];
            const d3 pb = ((row_q(0) * o4[0] + row_q(1) * o4[1]) + row_q(2) * o4[2]) + row_q(3) * o4[3];
            cp1 = cp2 = (pa + pb) * 0.5;
            done = true;
        }
    }
    if (done) {
        o.dist[pid] = dist;
        o.cp1[3 * (int64_t)pid] = cp1.x;
        o.cp1[3 * (int64_t)pid + 1] = cp1.y;
        o.cp1[3 * (int64_t)pid + 2] = cp1.z;
        o.cp2[3 * (int64_t)pid] = cp2.x;
        o.cp2[3 * (int64_t)pid + 1] = cp2.y;
        o.cp2[3 * (int64_t)pid + 2] = cp2.z;
        double* sp = o.simplex + 12 * (int64_t)pid;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            sp[3 * j] = w[j].x;
            sp[3 * j + 1] = w[j].y;
            sp[3 * j + 2] = w[j].z;
        }
        o.n_simplex[pid] = (int8_t)nr;
        o.status[pid] = (int8_t)D3D_STATUS_OK;
        // the gap row counts as the FP64 iteration that closed the bracket
        if (o.iterations) o.iterations[pid] = it_a + (sep ? 1 : 0);
    } else {
        EndRecord& e = lists.records[pid];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            if (j < nr && rows_ok) {
                const d3 p = row_p(j), q = row_q(j);
                e.pq[j][0] = p.x;
                e.pq[j][1] = p.y;
                e.pq[j][2] = p.z;
                e.pq[j][3] = q.x;
                e.pq[j][4] = q.y;
                e.pq[j][5] = q.z;
            }
        }
        e.n = rows_ok ? nr : 0;
    }
    lists.run_flag[slot] = (int8_t)(!done);
    lists.run_pid[slot] = pid;
}

// R, one lane per slot of the order (see the top of this file), `per` slots
// per block.  The grid covers the capacity; slots at and beyond the pair count
// are flagged 0.  The block lists every row's two supports by collider type
// (typelist.cuh) and its warps evaluate them 32 of a type at a time, the hulls
// of the gap rows, whose vertex has to be searched, one per warp.  (One lane
// per pair evaluated its rows in turn: 20 lanes per FP64 instruction in the
// type-sorted order, 8.6 in a batch too small to be sorted.  1M pairs 1.00 ->
// 0.86 ms, 300,032 robot pairs 270 -> 187 us, 3,000 pairs 65 -> 20 us.)  The checks that
// follow run in different branches for touching pairs and for separated pairs
// of one, two and three rows, so the block regroups them: the pairs are sorted
// by that class (counting sort over the block, the rows staying where they are
// in shared memory) and thread t runs the t-th pair's checks (r_finish).
constexpr int kRowTasks = 10;  // rows x sides of a pair

template <int BLOCK, bool MESH>
__global__ void __launch_bounds__(BLOCK) k_gjk_mixed_r(d3d_store s, const int32_t* __restrict__ i1,
                                                        const int32_t* __restrict__ i2,
                                                        const int32_t* __restrict__ order, int64_t cap, int per,
                                                        const int64_t* __restrict__ n_dev, d3d_gjk_options opt,
                                                        const Handoff* __restrict__ hand, DistanceOut o, Lists lists) {
    constexpr int W = BLOCK / 32;
    constexpr unsigned kAll = 0xffffffffu;
    // p and q of up to five rows per lane: element e of row j at [(6 j + e) BLOCK]
    __shared__ double rows[30 * BLOCK];
    __shared__ float4 tv[BLOCK];       // the handoff's v of each lane's pair
    __shared__ int tpid[BLOCK], tita[BLOCK], tcls[BLOCK];
    __shared__ int col[2 * BLOCK];
    __shared__ unsigned short list[kRowTasks * BLOCK];  // thread * kRowTasks + 2 row + side
    __shared__ int tcnt[kSupportBins], next;
    __shared__ unsigned short tperm[BLOCK];
    __shared__ int cnt[4 * W];
    const int64_t n = n_dev ? *n_dev : cap;
    const int64_t slot0 = (int64_t)blockIdx.x * per;
    const int64_t slot = slot0 + threadIdx.x;
    const bool in = (int)threadIdx.x < per && slot < cap;
    const int ln = threadIdx.x & 31, wp = threadIdx.x >> 5;
    if (threadIdx.x < kSupportBins) tcnt[threadIdx.x] = 0;
    if (threadIdx.x == kSupportBins) next = 0;
    int32_t pid = 0;
    int outcome = PA_FAILED, nr = 0, it_a = 0;
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    if (in && slot < n) {
        pid = order ? order[slot] : (int32_t)slot;
        v = hand[pid].v;
        outcome = __float_as_int(v.w) & 0xff;
        nr = (__float_as_int(v.w) >> 8) & 0xff;
        it_a = handoff_iters(v);
    }
    const bool mine = outcome == PA_SEPARATED || outcome == PA_TOUCHING;  // R or B finishes it
    const bool rows_ok = mine && nr >= 1 && nr <= 4;
    const bool sep = rows_ok && outcome == PA_SEPARATED && nr <= 3;
    const bool touch = rows_ok && outcome == PA_TOUCHING && nr == 4;
    // the rows in FP64, then the gap row of a separated pair along -v
    const int count = rows_ok ? nr + (sep ? 1 : 0) : 0;
    double* my = rows + threadIdx.x;
    tv[threadIdx.x] = v;
    tpid[threadIdx.x] = pid;
    __syncthreads();
    int bin[2] = {0, 0}, pos[2] = {0, 0}, found[2] = {0, 0};
    bool search[2] = {false, false};
    if (rows_ok) {
#pragma unroll
        for (int k = 0; k < 2; ++k) {
            const int c = (k ? i2 : i1)[pid];
            col[k * BLOCK + threadIdx.x] = c;
            const int4 m = __ldg(reinterpret_cast<const int4*>(s.meta) + c);
            bin[k] = support_bin(m.x, m.w);
            search[k] = sep && m.x == D3D_HULL;
            pos[k] = atomicAdd(tcnt + bin[k], search[k] ? count - 1 : count);
            if (search[k]) found[k] = atomicAdd(tcnt + kSearchBin, 1);
        }
    }
    __syncthreads();
    const Chunks ch = chunks_of(tcnt, kSupportBins, ln == kSearchBin ? 2 : 32);
#pragma unroll
    for (int k = 0; k < 2; ++k) {
        const int p0 = ch.start(bin[k]) + pos[k], p1 = ch.start(kSearchBin) + found[k];
        const unsigned short t = (unsigned short)(threadIdx.x * kRowTasks + k);
        for (int j = 0; j < (search[k] ? count - 1 : count); ++j) list[p0 + j] = t + 2 * j;
        if (search[k]) list[p1] = t + 2 * nr;
    }
    __syncthreads();
    int cb, first, num;
    while (ch.take(&next, cb, first, num)) {
        // the hulls to search, each by the whole warp
        int vi = -1;
        const bool on = ln < num;
        const int e = list[first + (on ? ln : 0)];
        const int t = e / kRowTasks, j = (e % kRowTasks) >> 1, k = e & 1;
        const int c = col[k * BLOCK + t];
        const float4 u = tv[t];
        const int rn = (__float_as_int(u.w) >> 8) & 0xff;
        float4 f = make_float4(-u.x, -u.y, -u.z, __uint_as_float(0xffffffffu));  // the gap row: no vertices known
        if (j < rn) f = hand[tpid[t]].d[j];
        if (cb == kSearchBin) {
            int type, nv, off;
            load_meta(s, c, type, nv, off);
            const f3 d = k ? mk(-f.x, -f.y, -f.z) : mk(f.x, f.y, f.z);
            for (int h = 0; h < num; ++h) {
                const int w = warp_hull_argmax(s.verts32, __shfl_sync(kAll, off, h), max(__shfl_sync(kAll, nv, h), 1),
                                               mk(__shfl_sync(kAll, d.x, h), __shfl_sync(kAll, d.y, h),
                                                  __shfl_sync(kAll, d.z, h)));
                if (ln == h) vi = w;
            }
        } else {
            vi = handoff_vertex(f, k);
        }
        if (on) {
            // the polytope vertices phase A took along this row's direction are read, not searched again
            const f3 df = k ? mk(-f.x, -f.y, -f.z) : mk(f.x, f.y, f.z);
            Col<double> cl;
            load_col(s, c, cl);
            const d3 x = RefineSupportT<MESH>::eval_at(cl, s, mk(widen(df.x), widen(df.y), widen(df.z)), df, vi);
            double* r = rows + t + (6 * j + 3 * k) * BLOCK;
            r[0] = x.x;
            r[BLOCK] = x.y;
            r[2 * BLOCK] = x.z;
        }
        __syncwarp();
    }
    __syncthreads();
    // class of the checks: 0 touching (four rows), 1-3 separated with that many rows, 4 none
    const int cls = touch ? 0 : (sep ? nr : 4);
    if (cls == 4 && in) {
        // a pair R does not check goes to B as it is (rows of a pair of another shape are kept), or
        // is not R's at all
        if (mine) {
            EndRecord& e = lists.records[pid];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                if (j < nr && rows_ok) {
                    e.pq[j][0] = my[(6 * j) * BLOCK];
                    e.pq[j][1] = my[(6 * j + 1) * BLOCK];
                    e.pq[j][2] = my[(6 * j + 2) * BLOCK];
                    e.pq[j][3] = my[(6 * j + 3) * BLOCK];
                    e.pq[j][4] = my[(6 * j + 4) * BLOCK];
                    e.pq[j][5] = my[(6 * j + 5) * BLOCK];
                }
            }
            e.n = rows_ok ? nr : 0;
        }
        lists.run_flag[slot] = (int8_t)mine;
        lists.run_pid[slot] = pid;
    }
    tita[threadIdx.x] = it_a;
    tcls[threadIdx.x] = cls | (nr << 8);
    int rank = 0;
#pragma unroll
    for (int c = 0; c < 4; ++c) {
        const unsigned m = __ballot_sync(kAll, cls == c);
        if (cls == c) rank = __popc(m & ((1u << ln) - 1u));
        if (ln == 0) cnt[c * W + wp] = __popc(m);
    }
    __syncthreads();
    int t = 0, ntask = 0;
#pragma unroll
    for (int c = 0; c < 4; ++c)
#pragma unroll
        for (int w = 0; w < W; ++w) {
            const int k = cnt[c * W + w];
            if (c < cls || (c == cls && w < wp)) t += k;
            ntask += k;
        }
    if (cls < 4) tperm[t + rank] = (unsigned short)threadIdx.x;
    __syncthreads();
    if ((int)threadIdx.x < ntask) {
        const int owner = tperm[threadIdx.x];
        const int x = tcls[owner];
        const int c = x & 0xff, rn = x >> 8;
        r_finish<BLOCK>(rows + owner, rn, c >= 1, c == 0, tv[owner], tita[owner], tpid[owner], slot0 + owner, opt, o,
                        lists);
    }
}

// B over R's run list, in the order of the slots: a pool of S pairs per block
// in shared memory, in rounds as the plain FP64 GJK runs them (gjk_pool.cuh,
// whose pool it uses).  Each round lists the pairs' supports by collider type
// (a hull is searched by the whole warp) and, after the new Minkowski points,
// the simplices by size, and the lanes of a warp take one kind.  A pair's
// first round (the replay) solves the handed-over rows without a support.
// The arithmetic is RefineSupport's and closest_to_origin's as they compile
// for one lane per pair.  With one lane per pair this kernel had 5.4 lanes per
// FP64 instruction: 87,819 scene pairs 385 -> 361 us, 300,032 robot pairs
// 356 -> 299 us, 20,011 pairs of ten types 222 -> 187 us, 3,000 pairs 120 ->
// 107 us, 1M pairs 727 -> 720 us.
// states beside pool::kFree and kLive (the loop has no kEnding)
constexpr int kReplay = pool::kEnding, kSpare = pool::kSpare;

template <int S>
__device__ __forceinline__ void b_finish(const pool::Mem<S, 4>& m, int s, unsigned perm, int n, d3 dir, double vl,
                                         int state, const Handoff* hand, const DistanceOut& o, const Lists& lists) {
    // the closest points and checks (pb_end) run in the end pass
    const int pid = m.pid[s];
    EndRecord& e = lists.records[pid];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        if (k < n) {
            const int r = pool::place_of(perm, k);
            const d3 pk = m.row(m.P, r, s), qk = m.row(m.Q, r, s);
            e.pq[k][0] = pk.x;
            e.pq[k][1] = pk.y;
            e.pq[k][2] = pk.z;
            e.pq[k][3] = qk.x;
            e.pq[k][4] = qk.y;
            e.pq[k][5] = qk.z;
        }
    }
    e.dir[0] = dir.x;
    e.dir[1] = dir.y;
    e.dir[2] = dir.z;
    e.vl = vl;
    e.it = m.it[s] + handoff_iters(hand[pid].v);
    e.state = state;
    e.status = D3D_STATUS_OK;
    e.n = n;
    double* sp = o.simplex + 12 * (int64_t)pid;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const d3 y = m.row(m.Y, pool::place_of(perm, j), s);
        sp[3 * j] = y.x;
        sp[3 * j + 1] = y.y;
        sp[3 * j + 2] = y.z;
    }
    o.n_simplex[pid] = (int8_t)n;
    append_warp(lists.ends, lists.ctr + kNumEnd, true, pid);
}

template <int S, bool MESH>
__global__ void __launch_bounds__(S, 3) k_gjk_mixed_b(d3d_store st, const int32_t* __restrict__ i1,
                                                            const int32_t* __restrict__ i2, d3d_gjk_options opt,
                                                            const Handoff* __restrict__ hand, DistanceOut o,
                                                            Lists lists) {
    constexpr unsigned kAll = 0xffffffffu;
    constexpr int kBins = 2 * kSupportTypes;
    extern __shared__ __align__(16) unsigned char b_smem[];
    pool::Mem<S, 4>& m = *reinterpret_cast<pool::Mem<S, 4>*>(b_smem);
    const int t = threadIdx.x, ln = t & 31;
    const long long n = (long long)lists.ctr[kNumRun];
    const JoltEps<double> E = reference_eps<double>();
    const double tol_sq = opt.tolerance * opt.tolerance;
    const long long share = (n + gridDim.x - 1) / gridDim.x;
    const long long split = share < S ? 0 : n;
    bool exhausted = share == 0;
    WarpChunk chunk;
    m.meta[t] = !exhausted && t >= share ? pool::pack_meta(0, 0, 0, kSpare) : 0;
    if (!exhausted && t >= share) m.it[t] = spare_rounds(t, share);
    if (t < kBins) m.cnt[0][t] = m.cnt[1][t] = 0;
    if (t < 4) m.scnt[0][t] = m.scnt[1][t] = m.next[t >> 1][t & 1] = 0;
    int type[2] = {0, 0};
    __syncthreads();
    for (int par = 0;; par ^= 1) {
        // ---- free slots take new pairs
        int state = pool::meta_state(m.meta[t]);
        const bool want = state == pool::kFree && !exhausted;
        const long long slot = fetch_slot_chunked(lists.ctr + kCurB, want, chunk, kAll, kChunk, split);
        if (want) {
            if (slot >= n) {
                exhausted = true;
            } else {
                const int pid = lists.run[slot];
                const EndRecord& rec = lists.records[pid];
                const int rows = rec.n;
                if (rows < 1 || rows > 4) {
                    lists.fallback[atomicAdd(lists.ctr + kNumFallback, 1ull)] = pid;
                } else {
                    m.pid[t] = pid;
                    m.it[t] = 0;
#pragma unroll
                    for (int k = 0; k < 2; ++k) {
                        const int c = (k ? i2 : i1)[pid];
                        const int4 q = __ldg(reinterpret_cast<const int4*>(st.meta) + c);
                        type[k] = support_bin(q.x, q.w);
                        m.col[k * S + t] = c;
                    }
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        d3 y = mk(0.0, 0.0, 0.0);
                        if (j < rows) {
                            const d3 p = mk(rec.pq[j][0], rec.pq[j][1], rec.pq[j][2]);
                            const d3 q = mk(rec.pq[j][3], rec.pq[j][4], rec.pq[j][5]);
                            m.put(m.P, j, t, p);
                            m.put(m.Q, j, t, q);
                            y = p - q;
                        }
                        m.put(m.Y, j, t, y);
                    }
                    m.meta[t] = pool::pack_meta(0xe4u, rows, 0, kReplay);
                    state = kReplay;
                }
            }
        }
        // ---- list the supports
        int pos[2];
#pragma unroll
        for (int k = 0; k < 2; ++k) {
            const int bin = state == pool::kLive ? type[k] : -1;
            const unsigned same = __match_any_sync(kAll, bin);
            const int leader = __ffs(same) - 1;
            int base = 0;
            if (ln == leader && bin >= 0) base = atomicAdd(&m.cnt[par][bin], __popc(same));
            pos[k] = __shfl_sync(kAll, base, leader) + __popc(same & ((1u << ln) - 1u));
        }
        if (!__syncthreads_or(state == pool::kFree ? !exhausted : state != kSpare)) break;
        const Chunks ch = chunks_of(m.cnt[par], kBins, (ln >> 1) == D3D_HULL ? pool::kHullChunk : 32);
#pragma unroll
        for (int k = 0; k < 2; ++k) {
            const int p = ch.start(type[k]) + pos[k];
            if (state == pool::kLive) m.list[p] = (unsigned short)(2 * t + k);
        }
        __syncthreads();
        int cb, first, count;
        while (ch.take(&m.next[par][0], cb, first, count)) {
            const bool on = ln < count;
            const int e = m.list[first + (on ? ln : 0)];
            const int s = e >> 1, side = e & 1;
            const int c = m.col[side * S + s];
            d3 d = m.direction(s);
            if (side) d = -d;
            const f3 df = RefineSupportT<MESH>::rounded(d);
            int vi = -1;
            if ((cb >> 1) == D3D_HULL) {
                int ty, nv, off;
                load_meta(st, c, ty, nv, off);
                for (int h = 0; h < count; ++h) {
                    const int w = warp_hull_argmax(
                        st.verts32, __shfl_sync(kAll, off, h), max(__shfl_sync(kAll, nv, h), 1),
                        mk(__shfl_sync(kAll, df.x, h), __shfl_sync(kAll, df.y, h), __shfl_sync(kAll, df.z, h)));
                    if (ln == h) vi = w;
                }
            }
            if (on) {
                Col<double> cl;
                load_col(st, c, cl);
                m.put_support(s, side, RefineSupportT<MESH>::eval_at(cl, st, d, df, vi));
            }
            __syncwarp();
        }
        __syncthreads();
        // ---- advance
        int cls = -1;
        if (state == kReplay) {
            cls = 4 - pool::meta_n(m.meta[t]);
        } else if (state == pool::kLive) {
            const unsigned mt = m.meta[t];
            const unsigned perm = mt & 0xffu;
            const int f = pool::meta_fresh(mt), rows = pool::meta_n(mt);
            const int it = m.it[t];
            bool fallback = it >= opt.max_iterations;
            if (!fallback) {
                m.it[t] = it + 1;
                const d3 w = m.row(m.P, f, t) - m.row(m.Q, f, t);
                const d3 dir = m.direction(t);
                const double vl = m.vl[t];
                const double dd = dot(dir, w);
                // duality gap: |v| - (|v|^2 - v.w) / |v| <= distance <= |v|
                const double gap = vl + dd;
                if (dd < 0.0 && dd * dd > vl * opt.max_distance_squared) {
                    fallback = true;  // clipped: the FP64 kernel reports it
                } else if (rows > 0 &&
                           (gap <= kMixedRelGap * vl || gap * gap <= kMixedAbsGap2 * maxf2(1.0, dot(w, w)) * vl)) {
                    b_finish(m, t, perm, rows, -dir, vl, GJK_NO_INTERSECTION, hand, o, lists);
                    m.meta[t] = 0;
                } else {
                    m.put(m.Y, f, t, w);
                    m.meta[t] = pool::pack_meta((perm & ~(3u << (2 * rows))) | ((unsigned)f << (2 * rows)), rows + 1,
                                                0, pool::kLive);
                    cls = 3 - rows;
                }
            }
            if (fallback) {
                lists.fallback[atomicAdd(lists.ctr + kNumFallback, 1ull)] = m.pid[t];
                m.meta[t] = 0;
            }
        } else if (state == kSpare) {
            exhausted = slots_claimed(lists.ctr + kCurB, n);
            if (exhausted || --m.it[t] == 0) m.meta[t] = 0;
        }
        __syncwarp();
        {
            unsigned mine = 0;
            int base = 0;
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const unsigned b = __ballot_sync(kAll, cls == k);
                if (cls == k) mine = b;
                if (ln == k) base = b ? atomicAdd(&m.scnt[par][k], __popc(b)) : 0;
            }
            const int p = __shfl_sync(kAll, base, cls >= 0 ? cls : 0) + __popc(mine & ((1u << ln) - 1u));
            if (cls >= 0) m.solve[cls * S + p] = (unsigned short)t;
        }
        if (t < kBins) m.cnt[par ^ 1][t] = 0;
        if (t < 4) m.scnt[par ^ 1][t] = 0;
        if (t < 2) m.next[par ^ 1][t] = 0;
        __syncthreads();
        // ---- solve, 16 simplices of one size to a chunk
        const Chunks ph = chunks_of(m.scnt[par], 4, 16);
        while (ph.take(&m.next[par][1], cb, first, count)) {
            const int k0 = first - ph.start(cb);
            if (ln < count) {
                const int s = m.solve[cb * S + k0 + ln];
                const unsigned mt = m.meta[s];
                const bool replay = pool::meta_state(mt) == kReplay;
                unsigned perm = mt & 0xffu;
                Simplex<double, RegRows<double>> X;
                X.n = pool::meta_n(mt);
#pragma unroll
                for (int k = 0; k < 4; ++k) X.Y[k] = m.y(mt, k, s);
                double prev = replay ? DBL_MAX : m.prev[s];
                d3 nv;
                double nl;
                int set;
                d3 dir;
                double vl;
                bool fallback = false;
                if (closest_to_origin<double, RegRows<double>, true>(X, prev, E, nv, nl, set)) {
                    dir = nv;
                    vl = nl;
                } else if (replay) {
                    fallback = true;
                } else {
                    --X.n;
                    set = (1 << X.n) - 1;
                    dir = m.direction(s);
                    vl = m.vl[s];
                }
                int ended = -1;
                if (fallback) {
                    lists.fallback[atomicAdd(lists.ctr + kNumFallback, 1ull)] = m.pid[s];
                    m.meta[s] = 0;
                } else if (set == 15) {
                    vl = 0.0;
                    ended = GJK_INTERSECTION;
                } else {
                    unsigned np = perm;
                    int k = 0;
                    double y = 0.0;
#pragma unroll
                    for (int r = 0; r < 4; ++r)
                        if (r < X.n && ((set >> r) & 1)) {
                            np = (np & ~(3u << (2 * k))) | (((perm >> (2 * r)) & 3u) << (2 * k));
                            const double l = dot(X.Y[r], X.Y[r]);
                            if (k == 0 || l > y) y = l;
                            ++k;
                        }
                    perm = np;
                    X.n = k;
                    if (vl <= tol_sq || vl <= E.isect * y) {
                        vl = 0.0;
                        ended = GJK_INTERSECTION;
                    } else {
                        dir = -dir;
                        if (prev - vl <= E.conv * prev) ended = GJK_NO_INTERSECTION;
                    }
                }
                if (ended >= 0) {
                    b_finish(m, s, perm, X.n, dir, vl, ended, hand, o, lists);
                    m.meta[s] = 0;
                } else if (!fallback) {
                    m.prev[s] = vl;
                    m.vl[s] = vl;
                    m.dir[s] = dir.x;
                    m.dir[S + s] = dir.y;
                    m.dir[2 * S + s] = dir.z;
                    m.meta[s] = pool::pack_meta(perm, X.n, pool::free_place(perm, X.n), pool::kLive);
                }
            }
            __syncwarp();
        }
        __syncthreads();
    }
}

// The end pass over B's finished pairs: closest points, sanity and
// consistency checks (pb_end) and the outputs; pairs failing a check go to
// the fallback list.
__global__ void __launch_bounds__(128) k_gjk_mixed_end(d3d_gjk_options opt, DistanceOut o, Lists lists) {
    const int64_t n = (int64_t)lists.ctr[kNumEnd];
    const JoltEps<double> E = reference_eps<double>();
    const int64_t lanes = spread_lanes(n, 128), warps = (int64_t)gridDim.x * 4;  // few pairs: spread
    const int ln = threadIdx.x & 31;
    if (ln >= lanes) return;
    for (int64_t k = ((int64_t)blockIdx.x * 4 + (threadIdx.x >> 5)) * lanes + ln; k < n; k += warps * lanes) {
        const int32_t pid = lists.ends[k];
        const EndRecord& e = lists.records[pid];
        GjkLoop<double, RegRows<double>> g;
        g.S.n = e.n;
        const double* sp = o.simplex + 12 * (int64_t)pid;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            g.S.Y[j] = mk(sp[3 * j], sp[3 * j + 1], sp[3 * j + 2]);
            if (j < e.n)
                g.S.R.put(j, mk(e.pq[j][0], e.pq[j][1], e.pq[j][2]), mk(e.pq[j][3], e.pq[j][4], e.pq[j][5]));
        }
        g.dir = mk(e.dir[0], e.dir[1], e.dir[2]);
        g.vl = e.vl;
        g.prev = 0.0;
        g.it = e.it;
        g.state = e.state;
        g.status = e.status;
        GjkResult<double> r;
        if (pb_end(g, opt, E, r) == PB_DONE) {
            o.dist[pid] = r.dist;
            o.cp1[3 * (int64_t)pid] = r.a.x;
            o.cp1[3 * (int64_t)pid + 1] = r.a.y;
            o.cp1[3 * (int64_t)pid + 2] = r.a.z;
            o.cp2[3 * (int64_t)pid] = r.b.x;
            o.cp2[3 * (int64_t)pid + 1] = r.b.y;
            o.cp2[3 * (int64_t)pid + 2] = r.b.z;
            o.status[pid] = (int8_t)r.status;
            if (o.iterations) o.iterations[pid] = r.iters;
        } else {
            lists.fallback[atomicAdd(lists.ctr + kNumFallback, 1ull)] = pid;
        }
    }
}

inline size_t up(size_t x) { return (x + 255) & ~size_t(255); }

}  // namespace

namespace d3d {

// temporary storage of the run list's stable compaction (CUB) over n slots
size_t select_temp_bytes(int64_t n) {
    size_t b = 0;
    cub::DeviceSelect::Flagged(nullptr, b, static_cast<const int32_t*>(nullptr), static_cast<const int8_t*>(nullptr),
                               static_cast<int32_t*>(nullptr), static_cast<unsigned long long*>(nullptr), (int)n);
    return up(b);
}

size_t gjk_mixed_scratch_bytes(int64_t capacity) {
    const size_t c = (size_t)capacity;
    return 256 + up(sizeof(int32_t) * c) + pair_order_temp_bytes(capacity) + up(sizeof(Handoff) * c) +
           2 * up(sizeof(int32_t) * c) + up(sizeof(EndRecord) * c) + up(c) + 2 * up(sizeof(int32_t) * c) +
           select_temp_bytes(capacity);
}

// B's pairs (and threads) per block
constexpr int kLoopPool = 128;

// R's block: 30 doubles of shared memory per lane
constexpr int kRefineBlock = 128;

template <int BLOCK, bool MESH>
int phase_a_blocks(int64_t n, int per_sm) {
    // alone: down to a pair per warp
    return persistent_blocks((const void*)k_gjk_mixed_a<BLOCK, MESH>, BLOCK, launch_items(32 * n, n), per_sm);
}

template <int BLOCK, bool MESH>
int launch_mixed(const d3d_store& store, const int32_t* i1, const int32_t* i2, const int32_t* order, int64_t n,
                 const int64_t* n_dev, const d3d_gjk_options& opt, Handoff* hand, const DistanceOut& o,
                 const Lists& lists, void* select_temp, size_t select_bytes, int per_sm, cudaStream_t stream) {
    const float tol_sq = (float)(opt.tolerance * opt.tolerance);
    const int full = phase_a_blocks<BLOCK, MESH>(n, per_sm);
    if (shared_gpu() || n >= (int64_t)full * BLOCK)
        k_gjk_mixed_a<BLOCK, MESH><<<full, BLOCK, 0, stream>>>(store, i1, i2, order, n, n_dev, tol_sq,
                                                               (float)opt.max_distance_squared, opt.max_iterations,
                                                               hand, o, lists);
    else
        k_gjk_mixed_a_spread<BLOCK, MESH><<<full, BLOCK, 0, stream>>>(
            store, i1, i2, order, n, n_dev, tol_sq, (float)opt.max_distance_squared, opt.max_iterations, hand, o,
            lists);
    int rc = check_launch("d3d_gjk_distance (mixed, FP32 phase)");
    if (rc) return rc;
    // fewer slots per block where full blocks would leave SMs idle
    int sms = 1, dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    int64_t per = (n + 2 * sms - 1) / (2 * sms);
    per = per < 16 ? 16 : (per > kRefineBlock || shared_gpu() ? kRefineBlock : per);
    k_gjk_mixed_r<kRefineBlock, MESH><<<grid_for(n, (int)per), kRefineBlock, 0, stream>>>(
        store, i1, i2, order, n, (int)per, n_dev, opt, hand, o, lists);
    rc = check_launch("d3d_gjk_distance (mixed, refinement pass)");
    if (rc) return rc;
    // the flagged pairs, in the order of the slots
    cudaError_t e = cub::DeviceSelect::Flagged(select_temp, select_bytes, lists.run_pid, lists.run_flag, lists.run,
                                               lists.ctr + kNumRun, (int)n, stream);
    if (e != cudaSuccess) {
        set_error("d3d_gjk_distance (mixed, run list): %s", cudaGetErrorString(e));
        return D3D_ERR_CUDA;
    }
    const void* kb = (const void*)k_gjk_mixed_b<kLoopPool, MESH>;
    const int smem = (int)sizeof(pool::Mem<kLoopPool, 4>);
    e = cudaFuncSetAttribute(kb, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(kb, cudaFuncAttributePreferredSharedMemoryCarveout,
                                 (int)cudaSharedmemCarveoutMaxShared);
    if (e != cudaSuccess) {
        set_error("d3d_gjk_distance (mixed, FP64 loop): %s", cudaGetErrorString(e));
        return D3D_ERR_CUDA;
    }
    // beside other batches: blocks for a quarter of the pairs, R leaves 10-20 %
    k_gjk_mixed_b<kLoopPool, MESH><<<persistent_blocks(kb, kLoopPool, launch_items(n * kLoopPool, n / 4), 0, smem), kLoopPool, smem, stream>>>(
        store, i1, i2, opt, hand, o, lists);
    rc = check_launch("d3d_gjk_distance (mixed, FP64 loop)");
    if (rc) return rc;
    k_gjk_mixed_end<<<persistent_blocks((const void*)k_gjk_mixed_end, 128, launch_items(32 * n, n)), 128, 0, stream>>>(opt, o, lists);
    return check_launch("d3d_gjk_distance (mixed, end pass)");
}

// The kernels without the MeshGraph branch serve stores without meshes.
template <int BLOCK>
int launch_mixed(const d3d_store& store, const int32_t* i1, const int32_t* i2, const int32_t* order, int64_t n,
                 const int64_t* n_dev, const d3d_gjk_options& opt, Handoff* hand, const DistanceOut& o,
                 const Lists& lists, void* select_temp, size_t select_bytes, int per_sm, cudaStream_t stream) {
    if (store.n_links > 0)
        return launch_mixed<BLOCK, true>(store, i1, i2, order, n, n_dev, opt, hand, o, lists, select_temp,
                                         select_bytes, per_sm, stream);
    return launch_mixed<BLOCK, false>(store, i1, i2, order, n, n_dev, opt, hand, o, lists, select_temp, select_bytes,
                                      per_sm, stream);
}

// Sorted by type only where phase A fills the GPU (or runs beside other
// batches): in a spread grid R, B and the EPA list their work by type
// anyway, phase A's warps hold few lanes, and sorting puts the long pairs
// into the same warps.  Sorted -> unsorted, us: six types 10,000 pairs 487
// -> 413, 65,536 925 -> 726, 77,000 963 -> 793, 262,144 1,522 -> 1,605; ten
// types 20,011 569 -> 538, 77,000 895 -> 818, 90,000 958 -> 1,047.
static bool mixed_sorted(const d3d_tuning& t, int64_t n) {
    if (shared_gpu()) return n >= t.sort_min;
    int dev = 0, sms = 1;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    return n >= sort_from(t, 512 * (int64_t)sms);  // lanes of the full grid (phase_a_min_blocks)
}

template <bool MESH>
static int phase_a_blocks(const d3d_tuning& t, int64_t n) {
    if (t.gjk_block == 64) return phase_a_blocks<64, MESH>(n, blocks_per_sm(t, 64));
    if (t.gjk_block == 256) return phase_a_blocks<256, MESH>(n, blocks_per_sm(t, 256));
    return phase_a_blocks<128, MESH>(n, blocks_per_sm(t, 128));
}

GjkLaunch gjk_mixed_launch(const d3d_store& store, const d3d_tuning& t, int64_t n) {
    const int blocks = store.n_links > 0 ? phase_a_blocks<true>(t, n) : phase_a_blocks<false>(t, n);
    return {t.gjk_block, blocks, gjk_f64_launch(t, n).pool_blocks, mixed_sorted(t, n)};
}

int gjk_mixed_run(const d3d_store& store, const int32_t* i1, const int32_t* i2, int64_t n, const int64_t* n_dev,
                  const d3d_gjk_options& opt, const DistanceOut& o, void* scratch, cudaStream_t stream,
                  const int32_t** sorted) {
    const d3d_tuning t = tuning();
    const bool sched = mixed_sorted(t, n);
    const size_t c = (size_t)n;
    const size_t order_bytes = up(sizeof(int32_t) * c);
    const size_t temp_bytes = pair_order_temp_bytes(n);
    char* p = static_cast<char*>(scratch);
    Lists lists;
    lists.ctr = reinterpret_cast<unsigned long long*>(p);
    p += 256;
    int32_t* order = sched ? reinterpret_cast<int32_t*>(p) : nullptr;
    if (sorted) *sorted = order;
    p += order_bytes;
    void* temp = p;
    p += temp_bytes;
    Handoff* hand = reinterpret_cast<Handoff*>(p);
    p += up(sizeof(Handoff) * c);
    lists.fallback = reinterpret_cast<int32_t*>(p);
    p += up(sizeof(int32_t) * c);
    lists.ends = reinterpret_cast<int32_t*>(p);
    p += up(sizeof(int32_t) * c);
    lists.records = reinterpret_cast<EndRecord*>(p);
    p += up(sizeof(EndRecord) * c);
    lists.run_flag = reinterpret_cast<int8_t*>(p);
    p += up(c);
    lists.run_pid = reinterpret_cast<int32_t*>(p);
    p += up(sizeof(int32_t) * c);
    lists.run = reinterpret_cast<int32_t*>(p);
    p += up(sizeof(int32_t) * c);
    void* select_temp = p;
    const size_t select_bytes = select_temp_bytes(n);
    cudaError_t e = cudaMemsetAsync(lists.ctr, 0, kCounters * sizeof(unsigned long long), stream);
    if (e != cudaSuccess) {
        set_error("d3d_gjk_distance (mixed): %s", cudaGetErrorString(e));
        return D3D_ERR_CUDA;
    }
    int rc = sched ? pair_order(store, i1, i2, n, order, temp, temp_bytes, stream, n_dev) : D3D_SUCCESS;
    if (!rc) {
        if (t.gjk_block == 64)
            rc = launch_mixed<64>(store, i1, i2, order, n, n_dev, opt, hand, o, lists, select_temp, select_bytes,
                                  blocks_per_sm(t, 64), stream);
        else if (t.gjk_block == 256)
            rc = launch_mixed<256>(store, i1, i2, order, n, n_dev, opt, hand, o, lists, select_temp, select_bytes,
                                   blocks_per_sm(t, 256), stream);
        else
            rc = launch_mixed<128>(store, i1, i2, order, n, n_dev, opt, hand, o, lists, select_temp, select_bytes,
                                   blocks_per_sm(t, 128), stream);
    }
    if (!rc)
        rc = launch_gjk_f64(store, i1, i2, lists.fallback, n, lists.ctr + kNumFallback, lists.ctr + kCurC, opt, o,
                            stream);
    return rc;
}

int gjk_distance_mixed(const d3d_store& store, const int32_t* i1, const int32_t* i2, int64_t n,
                       const d3d_gjk_options& opt, double* dist, double* cp1, double* cp2, double* simplex,
                       int8_t* n_simplex, int8_t* status, int32_t* iterations, cudaStream_t stream) {
    void* block = nullptr;
    int rc = scratch_alloc(&block, gjk_mixed_scratch_bytes(n), stream);
    if (rc) return rc;
    DistanceOut o{dist, cp1, cp2, simplex, n_simplex, status, iterations};
    rc = gjk_mixed_run(store, i1, i2, n, nullptr, opt, o, block, stream);
    scratch_free(block, stream);
    return rc;
}

}  // namespace d3d
