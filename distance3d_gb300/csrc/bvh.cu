// bvh.cu -- broad phase: a linear BVH over FP64 axis-aligned boxes.
//
// Build (all on the device):
//   1. bounds of the box centers (warp reductions on order-preserving keys,
//      one atomic per block and bound);
//   2. 63-bit Morton codes of the centers (21 bits per axis), radix-sorted
//      with the leaf index as payload (CUB);
//   3. Karras' (2012) parallel hierarchy: one thread per internal node finds
//      its key range and split from common-prefix lengths, equal codes tied
//      by index;
//   4. bottom-up refit with one atomic visit counter per internal node (no
//      waiting: the second child to arrive merges and climbs on).
// A node is one 64-byte record: the boxes of its two children, their ids and
// the ends of their ranges, so that a traversal step waits for one load.
// (With child ids, ranges and boxes in arrays of their own a step took three
// dependent loads: self pairs of a 131,072-collider scene 109 -> 61 us, the
// 30,011 queries of a 200,003-leaf tree 146 -> 73 us.)
// Internal node boxes are FP32 rounded outward (lower bounds down, upper
// bounds up), so a box that overlaps in FP64 also overlaps in FP32: pruning
// never loses a pair.  Leaves are tested with the caller's exact FP64 boxes
// and the reference's closed-interval rule (aabb_tree.py:504-527), so the
// pair sets equal the reference's AabbTree / brute-force sets bit for bit.
//
// Queries walk the tree with a per-thread stack and compact hits with a warp
// ballot (one atomic per warp and round).  Hits are 64-bit keys sorted on the
// device, so the output order is fixed: self pairs (i, j), i < j ascending;
// box queries (leaf, query) ascending.
#include <cub/cub.cuh>

#include "capi_util.h"
#include "d3d_device.cuh"
#include "scratch.h"

namespace {

constexpr int kBlock = 256;
constexpr int kStack = 128;
constexpr uint32_t kRoot = 0xffffffffu;

inline size_t up(size_t x) { return (x + 255) & ~size_t(255); }

// ----------------------------------------------------------- tree layout
// All arrays live in one caller-provided buffer; offsets depend on n only.
struct Node {
    // children 0 and 1: box lower corner (xyz) and id (w, int bits: >= 0 an internal node, ~index of a
    // leaf), box upper corner (xyz) and last sorted position under the child (w, int bits)
    float4 child[4];
};
struct Tree {
    int64_t n;
    // one block cleared before a build: error flags (4 int32), then the bounds of the centers as
    // keys (uint64: largest ~key per axis, largest key per axis)
    int32_t* flags;
    unsigned long long* bounds;
    int32_t* sorted;    // [n]   sorted position -> original index
    Node* node;         // [n-1]
    uint32_t* parent;   // [n-1 + n] parent << 1 | side of internal nodes, then of leaves (kRoot: the root)
    int32_t* visits;    // [n-1] refit counters, zero between refits
    uint64_t* keys;     // [n]
    uint64_t* keys_out; // [n]
    int32_t* vals;      // [n]
    void* cub_temp;
    size_t cub_bytes;
};

size_t cub_sort_bytes(int64_t n) {
    size_t b = 0;
    cub::DeviceRadixSort::SortPairs(nullptr, b, (const uint64_t*)nullptr, (uint64_t*)nullptr,
                                    (const int32_t*)nullptr, (int32_t*)nullptr, (int)n, 0, 63);
    return b;
}

size_t layout(void* base, int64_t n, Tree* t) {
    const int64_t ni = n > 1 ? n - 1 : 1;
    const size_t cub_bytes = cub_sort_bytes(n > 0 ? n : 1);
    size_t off = 256;
    auto take = [&](size_t bytes) {
        size_t o = off;
        off += up(bytes);
        return o;
    };
    size_t o_flags = take(256);
    size_t o_sorted = take(sizeof(int32_t) * n);
    size_t o_node = take(sizeof(Node) * ni);
    size_t o_parent = take(sizeof(uint32_t) * (ni + n));
    size_t o_visits = take(sizeof(int32_t) * ni);
    size_t o_keys = take(sizeof(uint64_t) * n);
    size_t o_keys_out = take(sizeof(uint64_t) * n);
    size_t o_vals = take(sizeof(int32_t) * n);
    size_t o_cub = take(cub_bytes);
    if (t) {
        char* b = static_cast<char*>(base);
        t->n = n;
        t->flags = reinterpret_cast<int32_t*>(b + o_flags);
        t->bounds = reinterpret_cast<unsigned long long*>(b + o_flags + 16);
        t->sorted = reinterpret_cast<int32_t*>(b + o_sorted);
        t->node = reinterpret_cast<Node*>(b + o_node);
        t->parent = reinterpret_cast<uint32_t*>(b + o_parent);
        t->visits = reinterpret_cast<int32_t*>(b + o_visits);
        t->keys = reinterpret_cast<uint64_t*>(b + o_keys);
        t->keys_out = reinterpret_cast<uint64_t*>(b + o_keys_out);
        t->vals = reinterpret_cast<int32_t*>(b + o_vals);
        t->cub_temp = b + o_cub;
        t->cub_bytes = cub_bytes;
    }
    return off;
}

// ----------------------------------------------------------- build kernels
__device__ __forceinline__ void load_box(const double* aabbs, int64_t i, double* lo, double* hi) {
    const double* a = aabbs + 6 * i;  // [axis][min,max]
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        lo[k] = a[2 * k];
        hi[k] = a[2 * k + 1];
    }
}

// Unsigned order equals the order of the doubles (not NaN); 0 is below every key.
__device__ __forceinline__ unsigned long long order_key(double x) {
    const unsigned long long u = (unsigned long long)__double_as_longlong(x);
    return (u >> 63) ? ~u : (u | 0x8000000000000000ull);
}
__device__ __forceinline__ double from_key(unsigned long long k) {
    return __longlong_as_double((long long)((k >> 63) ? (k & 0x7fffffffffffffffull) : ~k));
}

// The warp's largest 64-bit value, by REDUX on the halves.
__device__ __forceinline__ unsigned long long warp_max64(unsigned long long k) {
    const unsigned hi = __reduce_max_sync(0xffffffffu, (unsigned)(k >> 32));
    const unsigned lo = __reduce_max_sync(0xffffffffu, (unsigned)(k >> 32) == hi ? (unsigned)k : 0u);
    return ((unsigned long long)hi << 32) | lo;
}

// bounds[k]: largest ~key of the centers on axis k (their minimum), bounds[3 + k]: largest key; NaN
// centers are left out.  (Partial bounds per block, reduced by one thread, took 178 us at any size: FP64
// compares one after the other on one lane.)
__global__ void k_center_bounds(const double* __restrict__ aabbs, int64_t n, unsigned long long* __restrict__ bounds) {
    unsigned long long m[6] = {};
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        double lo[3], hi[3];
        load_box(aabbs, i, lo, hi);
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            const double c = 0.5 * (lo[k] + hi[k]);
            const unsigned long long key = order_key(c);
            if (c != c) continue;
            if (~key > m[k]) m[k] = ~key;
            if (key > m[3 + k]) m[3 + k] = key;
        }
    }
    __shared__ unsigned long long best[6];
    if (threadIdx.x < 6) best[threadIdx.x] = 0ull;
    __syncthreads();
#pragma unroll
    for (int k = 0; k < 6; ++k) {
        const unsigned long long w = warp_max64(m[k]);
        if ((threadIdx.x & 31) == 0) atomicMax(best + k, w);
    }
    __syncthreads();
    if (threadIdx.x < 6) atomicMax(bounds + threadIdx.x, best[threadIdx.x]);
}

__device__ __forceinline__ uint64_t spread21(uint64_t v) {
    v &= 0x1fffff;
    v = (v | (v << 32)) & 0x1f00000000ffffull;
    v = (v | (v << 16)) & 0x1f0000ff0000ffull;
    v = (v | (v << 8)) & 0x100f00f00f00f00full;
    v = (v | (v << 4)) & 0x10c30c30c30c30c3ull;
    v = (v | (v << 2)) & 0x1249249249249249ull;
    return v;
}

// 21 bits of the center c on an axis of `least` and extent `ext`, in FP64.
__device__ __noinline__ uint64_t axis_code(double c, double least, double ext) {
    const double x = ext > 0.0 ? (c - least) / ext * 2097152.0 : 0.0;
    return (x != x || x <= 0.0) ? 0ull : (x >= 2097151.0 ? 2097151ull : (uint64_t)x);
}

// axis_code's value without its division, bound by the FP64 pipe: 2^52 + (c -
// least) * (2^52 / ext) holds the code in the upper 21 bits of its mantissa and
// its fraction in the lower 31, a few units off axis_code's at most.  Where those
// could carry into the code, and where the sum is not in [2^52, 2^53) (a NaN, an
// extent out of range, the last center), axis_code decides.  Build of 200,003
// boxes with the division 240 us, without 230 (scaled in FP32 it was 232).
__global__ void k_morton(const double* __restrict__ aabbs, int64_t n, const unsigned long long* __restrict__ bounds,
                         uint64_t* __restrict__ keys, int32_t* __restrict__ vals) {
    __shared__ double least[3], ext[3], scale[3];
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    double lo[3] = {}, hi[3] = {};
    if (i < n) load_box(aabbs, i, lo, hi);
    if (threadIdx.x < 3) {
        const int k = threadIdx.x;
        least[k] = from_key(~bounds[k]);
        ext[k] = from_key(bounds[3 + k]) - least[k];
        scale[k] = 0x1p52 / ext[k];
    }
    __syncthreads();
    if (i >= n) return;
    uint64_t q[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const double c = 0.5 * (lo[k] + hi[k]);
        const uint64_t b = (uint64_t)__double_as_longlong(fma(c - least[k], scale[k], 0x1p52));
        const uint32_t rest = (uint32_t)b & 0x7fffffffu;
        const bool sure = (b >> 52) == 0x433u && rest - 8u < 0x7fffffffu - 16u;
        q[k] = sure ? (b >> 31) & 0x1fffffu : axis_code(c, least[k], ext[k]);
    }
    keys[i] = (spread21(q[0]) << 2) | (spread21(q[1]) << 1) | spread21(q[2]);
    vals[i] = (int32_t)i;
}

// common-prefix length of sorted keys i and j, ties broken by index
__device__ __forceinline__ int delta(const uint64_t* __restrict__ k, int64_t n, int64_t i, int64_t j) {
    if (j < 0 || j >= n) return -1;
    uint64_t a = k[i], b = k[j];
    if (a == b) return 64 + __clz((int)((uint32_t)i ^ (uint32_t)j));
    return __clzll((long long)(a ^ b));
}

__global__ void k_karras(const uint64_t* __restrict__ k, int64_t n, uint32_t* __restrict__ parent,
                         int32_t* __restrict__ visits) {
    int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n - 1) return;
    const int d = (delta(k, n, i, i + 1) - delta(k, n, i, i - 1)) > 0 ? 1 : -1;
    const int dmin = delta(k, n, i, i - d);
    int64_t lmax = 2;
    while (delta(k, n, i, i + lmax * d) > dmin) lmax *= 2;
    int64_t l = 0;
    for (int64_t t = lmax / 2; t >= 1; t /= 2)
        if (delta(k, n, i, i + (l + t) * d) > dmin) l += t;
    const int64_t j = i + l * d;
    const int dnode = delta(k, n, i, j);
    int64_t s = 0, t = l;
    do {
        t = (t + 1) / 2;
        if (delta(k, n, i, i + (s + t) * d) > dnode) s += t;
    } while (t > 1);
    const int64_t gamma = i + s * d + (d < 0 ? -1 : 0);
    const int64_t lo = i < j ? i : j, hi = i < j ? j : i;
    const int left = lo == gamma ? ~(int)gamma : (int)gamma;
    const int right = hi == gamma + 1 ? ~(int)(gamma + 1) : (int)(gamma + 1);
    const int64_t ni = n - 1;
    parent[left >= 0 ? left : ni + ~left] = (uint32_t)(2 * i);
    parent[right >= 0 ? right : ni + ~right] = (uint32_t)(2 * i + 1);
    visits[i] = 0;
    if (i == 0) parent[0] = kRoot;
}

// The nodes' records, from the leaves up: every child writes its half of its
// parent's record (box, id, last position), and the second one to arrive goes
// on with the parent.
__global__ void k_refit(const double* __restrict__ aabbs, Tree t) {
    int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= t.n) return;
    const int leaf = t.sorted[p];
    double dlo[3], dhi[3];
    load_box(aabbs, leaf, dlo, dhi);
    float4 lo = make_float4(__double2float_rd(dlo[0]), __double2float_rd(dlo[1]), __double2float_rd(dlo[2]),
                            __int_as_float(~leaf));
    float4 hi = make_float4(__double2float_ru(dhi[0]), __double2float_ru(dhi[1]), __double2float_ru(dhi[2]),
                            __int_as_float((int)p));
    uint32_t up = t.parent[t.n - 1 + p];
    int guard = 0;
    while (up != kRoot && guard++ < 4 * kStack) {
        const uint32_t side = up & 1, node = up >> 1;
        float4* const rec = t.node[node].child;
        __stcg(rec + 2 * side, lo);
        __stcg(rec + 2 * side + 1, hi);
        __threadfence();
        if (atomicAdd(t.visits + node, 1) == 0) return;  // the sibling subtree is not done yet
        __threadfence();
        t.visits[node] = 0;  // for the next refit
        const float4 olo = __ldcg(rec + 2 * (1 - side)), ohi = __ldcg(rec + 2 * (1 - side) + 1);
        lo = make_float4(fminf(lo.x, olo.x), fminf(lo.y, olo.y), fminf(lo.z, olo.z), __int_as_float((int)node));
        hi = make_float4(fmaxf(hi.x, ohi.x), fmaxf(hi.y, ohi.y), fmaxf(hi.z, ohi.z),
                         __int_as_float(max(__float_as_int(hi.w), __float_as_int(ohi.w))));
        up = t.parent[node];
    }
    if (up != kRoot) atomicExch(t.flags, 1);
}

// ----------------------------------------------------------- queries
__device__ __forceinline__ bool overlap32(const float4& alo, const float4& ahi, const float4& blo, const float4& bhi) {
    return alo.x <= bhi.x && ahi.x >= blo.x && alo.y <= bhi.y && ahi.y >= blo.y && alo.z <= bhi.z && ahi.z >= blo.z;
}

// aabb_tree.py:504-527, closed intervals; the compares on integers (d3d_device.cuh)
__device__ __forceinline__ bool overlap64(const double* a, const double* b) {
    return d3d::le(a[0], b[1]) && d3d::le(b[0], a[1]) && d3d::le(a[2], b[3]) && d3d::le(b[2], a[3]) &&
           d3d::le(a[4], b[5]) && d3d::le(b[4], a[5]);
}

// One hit each of the lanes that call it together: one atomic for all of them.
__device__ __forceinline__ void emit(uint64_t key, unsigned long long* count, uint64_t* out, int64_t cap) {
    const unsigned active = __activemask();
    const int lane = threadIdx.x & 31;
    const int leader = __ffs(active) - 1;
    unsigned long long base = 0;
    if (lane == leader) base = atomicAdd(count, (unsigned long long)__popc(active));
    base = __shfl_sync(active, base, leader);
    const unsigned long long idx = base + __popc(active & ((1u << lane) - 1u));
    if ((int64_t)idx < cap) out[idx] = key;
}

// One thread's walk of the tree for query box `box` (FP64) / qlo, qhi (FP32
// outward): key_of(leaf) gives the key of each leaf whose exact box
// overlaps it, subtrees that end at or before position `after` are skipped.
// The FP32 boxes of the leaves are tested first: they hold the exact ones.
template <typename Key>
__device__ __forceinline__ void walk(const double* __restrict__ aabbs, const Tree& t, const double* box, float4 qlo,
                                     float4 qhi, int after, Key key_of, unsigned long long* count, uint64_t* out,
                                     int64_t cap) {
    int stack[kStack];
    int sp = 0;
    int node = 0;
    while (node >= 0) {
        const float4* r = t.node[node].child;
        const float4 rec[4] = {__ldg(r), __ldg(r + 1), __ldg(r + 2), __ldg(r + 3)};
        int next = -1;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const float4 lo = rec[2 * h], hi = rec[2 * h + 1];
            if (__float_as_int(hi.w) <= after || !overlap32(qlo, qhi, lo, hi)) continue;
            const int x = __float_as_int(lo.w);
            if (x < 0) {
                if (overlap64(box, aabbs + 6 * (int64_t)~x)) emit(key_of(~x), count, out, cap);
            } else if (next < 0) {
                next = x;  // walked next; the other child waits on the stack
            } else if (sp < kStack) {
                stack[sp++] = x;
            } else {
                atomicExch(reinterpret_cast<int*>(count + 1), 1);
            }
        }
        node = next >= 0 ? next : (sp > 0 ? stack[--sp] : -1);
    }
}

// the refit's flag beside the count, so that one copy reads both
__device__ __forceinline__ void pass_flags(const Tree& t, unsigned long long* count) {
    if (blockIdx.x == 0 && threadIdx.x == 0 && t.flags[0]) atomicExch(reinterpret_cast<int*>(count + 1), 1);
}

__device__ __forceinline__ void outward(const double* box, float4& lo, float4& hi) {
    lo = make_float4(__double2float_rd(box[0]), __double2float_rd(box[2]), __double2float_rd(box[4]), 0.f);
    hi = make_float4(__double2float_ru(box[1]), __double2float_ru(box[3]), __double2float_ru(box[5]), 0.f);
}

// Pair keys: the first index above the `bits` of the second.
// Self pairs: thread p (sorted position) reports every leaf after p whose
// exact box overlaps its own, so each unordered pair is found once.
__global__ void k_self_pairs(const double* __restrict__ aabbs, Tree t, int bits, unsigned long long* count,
                             uint64_t* out, int64_t cap) {
    pass_flags(t, count);
    int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= t.n - 1) return;  // the last leaf has no later leaves
    const int op = t.sorted[p];
    double box[6];
#pragma unroll
    for (int k = 0; k < 6; ++k) box[k] = aabbs[6 * (int64_t)op + k];
    float4 qlo, qhi;
    outward(box, qlo, qhi);
    walk(aabbs, t, box, qlo, qhi, (int)p,
         [=](int leaf) { return ((uint64_t)(uint32_t)min(op, leaf) << bits) | (uint32_t)max(op, leaf); }, count, out,
         cap);
}

// Box queries: thread q reports every leaf whose exact box overlaps query q.
__global__ void k_query_boxes(const double* __restrict__ aabbs, Tree t, const double* __restrict__ boxes, int64_t m,
                              int bits, unsigned long long* count, uint64_t* out, int64_t cap) {
    pass_flags(t, count);
    int64_t qi = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (qi >= m) return;
    double box[6];
#pragma unroll
    for (int k = 0; k < 6; ++k) box[k] = boxes[6 * qi + k];
    auto key_of = [=](int leaf) { return ((uint64_t)(uint32_t)leaf << bits) | (uint32_t)qi; };
    if (t.n == 1) {
        const int leaf = t.sorted[0];
        if (overlap64(box, aabbs + 6 * (int64_t)leaf)) emit(key_of(leaf), count, out, cap);
        return;
    }
    float4 qlo, qhi;
    outward(box, qlo, qhi);
    walk(aabbs, t, box, qlo, qhi, -1, key_of, count, out, cap);
}

__global__ void k_decode(const uint64_t* __restrict__ keys, int64_t n, int bits, int32_t* __restrict__ pairs) {
    int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n) return;
    const uint64_t v = keys[k];
    pairs[2 * k] = (int32_t)(v >> bits);
    pairs[2 * k + 1] = (int32_t)(v & ((1ull << bits) - 1));
}

// bits that hold 0 .. n-1
int index_bits(int64_t n) {
    int b = 1;
    while ((int64_t(1) << b) < n) ++b;
    return b;
}

// Sort the hit keys and write int32 pairs; synchronises to read the count.
int finish_pairs(unsigned long long* d_count, uint64_t* keys, uint64_t* keys_alt, void* cub_temp, size_t cub_bytes,
                 int32_t* pairs, int64_t capacity, int64_t* n_pairs, int bits_first, int bits_second, cudaStream_t st) {
    // the pair count and the error flag
    unsigned long long read[2] = {0, 0};
    cudaMemcpyAsync(read, d_count, sizeof(read), cudaMemcpyDeviceToHost, st);
    cudaError_t e = cudaStreamSynchronize(st);
    if (e != cudaSuccess) {
        d3d::set_error("bvh query: %s", cudaGetErrorString(e));
        return D3D_ERR_CUDA;
    }
    const unsigned long long count = read[0];
    if (n_pairs) *n_pairs = (int64_t)count;
    if (read[1]) {
        d3d::set_error("bvh: traversal stack or refit bound exceeded (tree deeper than %d)", kStack);
        return D3D_ERR_CAPACITY;
    }
    if ((int64_t)count > capacity) {
        d3d::set_error("bvh query: %llu pairs exceed the capacity of %lld", count, (long long)capacity);
        return D3D_ERR_CAPACITY;
    }
    if (count == 0) return D3D_SUCCESS;
    // the keys' used bits only: a pass per 8 bits (5 instead of 8 below 2^20 boxes)
    const int bits = bits_first + bits_second;
    size_t need = 0;
    cub::DeviceRadixSort::SortKeys(nullptr, need, keys, keys_alt, (int)count, 0, bits, st);
    if (need > cub_bytes) {
        d3d::set_error("bvh query: sort temporary storage too small");
        return D3D_ERR_CAPACITY;
    }
    e = cub::DeviceRadixSort::SortKeys(cub_temp, need, keys, keys_alt, (int)count, 0, bits, st);
    if (e != cudaSuccess) {
        d3d::set_error("bvh query: sort failed: %s", cudaGetErrorString(e));
        return D3D_ERR_CUDA;
    }
    k_decode<<<d3d::grid_for((int64_t)count, kBlock), kBlock, 0, st>>>(keys_alt, (int64_t)count, bits_second, pairs);
    return d3d::check_launch("bvh query");
}

size_t query_cub_bytes(int64_t capacity) {
    size_t b = 0;
    cub::DeviceRadixSort::SortKeys(nullptr, b, (const uint64_t*)nullptr, (uint64_t*)nullptr,
                                   (int)(capacity > 0 ? capacity : 1), 0, 64);
    return b;
}

}  // namespace

extern "C" size_t d3d_bvh_bytes(int64_t n_leaves) {
    if (n_leaves < 0 || n_leaves >= (int64_t(1) << 31)) return 0;
    return layout(nullptr, n_leaves, nullptr);
}

extern "C" int d3d_bvh_build(const double* aabbs, int64_t n, void* tree, size_t tree_bytes, void* stream) {
    D3D_REQUIRE(n >= 0 && n < (int64_t(1) << 31), "d3d_bvh_build: n out of range");
    D3D_REQUIRE(tree, "d3d_bvh_build: null tree buffer");
    size_t need = layout(nullptr, n, nullptr);
    if (tree_bytes < need) {
        d3d::set_error("d3d_bvh_build: tree buffer of %zu bytes < %zu", tree_bytes, need);
        return D3D_ERR_CAPACITY;
    }
    Tree t;
    layout(tree, n, &t);
    cudaStream_t st = d3d::as_stream(stream);
    cudaMemsetAsync(t.flags, 0, 256, st);  // the bounds' keys with them
    if (n == 0) return d3d::check_launch("d3d_bvh_build");
    D3D_REQUIRE(aabbs, "d3d_bvh_build: null aabbs");
    const unsigned blocks = d3d::grid_for(n, kBlock);
    k_center_bounds<<<blocks < 304 ? blocks : 304, kBlock, 0, st>>>(aabbs, n, t.bounds);
    k_morton<<<blocks, kBlock, 0, st>>>(aabbs, n, t.bounds, t.keys, t.vals);
    size_t cub_bytes = t.cub_bytes;
    cudaError_t e = cub::DeviceRadixSort::SortPairs(t.cub_temp, cub_bytes, t.keys, t.keys_out, t.vals, t.sorted, (int)n,
                                                    0, 63, st);
    if (e != cudaSuccess) {
        d3d::set_error("d3d_bvh_build: sort failed: %s", cudaGetErrorString(e));
        return D3D_ERR_CUDA;
    }
    if (n > 1) {
        k_karras<<<d3d::grid_for(n - 1, kBlock), kBlock, 0, st>>>(t.keys_out, n, t.parent, t.visits);
        k_refit<<<blocks, kBlock, 0, st>>>(aabbs, t);
    }
    return d3d::check_launch("d3d_bvh_build");
}

extern "C" int d3d_bvh_refit(const double* aabbs, int64_t n, void* tree, size_t tree_bytes, void* stream) {
    D3D_REQUIRE(n >= 0 && n < (int64_t(1) << 31), "d3d_bvh_refit: n out of range");
    D3D_REQUIRE(tree, "d3d_bvh_refit: null tree buffer");
    size_t need = layout(nullptr, n, nullptr);
    if (tree_bytes < need) {
        d3d::set_error("d3d_bvh_refit: tree buffer of %zu bytes < %zu", tree_bytes, need);
        return D3D_ERR_CAPACITY;
    }
    if (n == 0) return D3D_SUCCESS;
    D3D_REQUIRE(aabbs, "d3d_bvh_refit: null aabbs");
    Tree t;
    layout(tree, n, &t);
    cudaStream_t st = d3d::as_stream(stream);
    // same leaf order and topology; the boxes of leaves and nodes are redone
    if (n > 1) k_refit<<<d3d::grid_for(n, kBlock), kBlock, 0, st>>>(aabbs, t);
    return d3d::check_launch("d3d_bvh_refit");
}

extern "C" size_t d3d_bvh_query_bytes(int64_t capacity) {
    if (capacity < 0) return 0;
    return 256 + 2 * up(sizeof(uint64_t) * (size_t)(capacity > 0 ? capacity : 1)) + up(query_cub_bytes(capacity));
}

static int query_common(const void* tree, int64_t n, int64_t capacity, void* scratch, size_t scratch_bytes,
                        Tree* t, unsigned long long** count, uint64_t** keys, uint64_t** alt, void** cub_temp,
                        size_t* cub_bytes) {
    D3D_REQUIRE(tree, "bvh query: null tree");
    D3D_REQUIRE(n >= 0 && capacity >= 0, "bvh query: negative size");
    size_t need = d3d_bvh_query_bytes(capacity);
    if (!scratch || scratch_bytes < need) {
        d3d::set_error("bvh query: scratch of %zu bytes < %zu", scratch_bytes, need);
        return D3D_ERR_CAPACITY;
    }
    layout(const_cast<void*>(tree), n, t);
    char* s = static_cast<char*>(scratch);
    *count = reinterpret_cast<unsigned long long*>(s);
    size_t kb = up(sizeof(uint64_t) * (size_t)(capacity > 0 ? capacity : 1));
    *keys = reinterpret_cast<uint64_t*>(s + 256);
    *alt = reinterpret_cast<uint64_t*>(s + 256 + kb);
    *cub_temp = s + 256 + 2 * kb;
    *cub_bytes = up(query_cub_bytes(capacity));
    return D3D_SUCCESS;
}

extern "C" int d3d_bvh_self_pairs(const double* aabbs, int64_t n, const void* tree, int32_t* pairs, int64_t capacity,
                                  int64_t* n_pairs, void* scratch, size_t scratch_bytes, void* stream) {
    Tree t;
    unsigned long long* count;
    uint64_t *keys, *alt;
    void* cub_temp;
    size_t cub_bytes;
    int rc = query_common(tree, n, capacity, scratch, scratch_bytes, &t, &count, &keys, &alt, &cub_temp, &cub_bytes);
    if (rc) return rc;
    cudaStream_t st = d3d::as_stream(stream);
    cudaMemsetAsync(count, 0, 2 * sizeof(unsigned long long), st);
    const int bits = index_bits(n);
    if (n > 1) {
        D3D_REQUIRE(aabbs && (pairs || capacity == 0), "d3d_bvh_self_pairs: null pointer");
        k_self_pairs<<<d3d::grid_for(n - 1, 128), 128, 0, st>>>(aabbs, t, bits, count, keys, capacity);
        rc = d3d::check_launch("d3d_bvh_self_pairs");
        if (rc) return rc;
    }
    return finish_pairs(count, keys, alt, cub_temp, cub_bytes, pairs, capacity, n_pairs, bits, bits, st);
}

extern "C" int d3d_bvh_query(const double* aabbs, int64_t n, const void* tree, const double* boxes, int64_t m,
                             int32_t* pairs, int64_t capacity, int64_t* n_pairs, void* scratch, size_t scratch_bytes,
                             void* stream) {
    Tree t;
    unsigned long long* count;
    uint64_t *keys, *alt;
    void* cub_temp;
    size_t cub_bytes;
    int rc = query_common(tree, n, capacity, scratch, scratch_bytes, &t, &count, &keys, &alt, &cub_temp, &cub_bytes);
    if (rc) return rc;
    D3D_REQUIRE(m >= 0 && m < (int64_t(1) << 31), "d3d_bvh_query: m out of range");
    cudaStream_t st = d3d::as_stream(stream);
    cudaMemsetAsync(count, 0, 2 * sizeof(unsigned long long), st);
    const int bits = index_bits(m);
    if (n > 0 && m > 0) {
        D3D_REQUIRE(aabbs && boxes && (pairs || capacity == 0), "d3d_bvh_query: null pointer");
        k_query_boxes<<<d3d::grid_for(m, 128), 128, 0, st>>>(aabbs, t, boxes, m, bits, count, keys, capacity);
        rc = d3d::check_launch("d3d_bvh_query");
        if (rc) return rc;
    }
    return finish_pairs(count, keys, alt, cub_temp, cub_bytes, pairs, capacity, n_pairs, index_bits(n), bits, st);
}
